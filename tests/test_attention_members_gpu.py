"""32-bit attention whose tiles are shared by the blocks of a cluster: more tiles of keys than blocks, fewer, ends within a tile,
several requests in a tile, every mask and size of head; held to the same restatement as the other forms."""
import pytest
import torch

import test_simt_gpu as simt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,firsts", [([200], [0]), ([65], [130]), ([130], [701]), ([30, 100, 1, 40], [300, 0, 500, 150])])
@pytest.mark.parametrize("d,dv,heads,kv_heads", [(64, 64, 7, 1), (128, 96, 4, 2), (80, 256, 4, 1), (30, 18, 2, 2)])
@pytest.mark.parametrize("mask", ["all", "wide window", "wide chunk"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_members(counts, firsts, d, dv, heads, kv_heads, mask, dtype):
    simt.test_attention_forms(counts, firsts, d, dv, heads, kv_heads, mask, dtype)
