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


@pytest.mark.parametrize("counts,firsts", [([60] * 4, [0] * 4), ([100, 3, 90], [0, 0, 30]), ([1] * 70, [90] * 70), ([300], [20])])
@pytest.mark.parametrize("longest", [0, 1, 2])
def test_short_requests_in_wide_tables(counts, firsts, longest):
    """Tables with room for far more keys than there are: known to be short or not, by one block a tile or shared."""
    from vipera_rs_b200.kernels import ops

    heads, kv_heads, d, page, width = 6, 2, 64, 16, 64
    torch.manual_seed(len(counts))
    tokens = sum(counts)
    entry = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    positions = torch.cat([torch.arange(f, f + c) for c, f in zip(counts, firsts)])
    table = torch.full((len(counts), width), -1, dtype=torch.int32)
    needed = [-(-(c + f) // page) for c, f in zip(counts, firsts)]
    for e, pages in enumerate(needed):
        table[e, :pages] = sum(needed[:e]) + torch.arange(pages)
    q = torch.randn(tokens, heads * d, device="cuda")
    k, v = (torch.randn(sum(needed), page, kv_heads, d, device="cuda") for _ in range(2))
    out = torch.full((tokens, heads * d), float("nan"), device="cuda")
    known = max(c + f for c, f in zip(counts, firsts)) if longest == 1 else 1024 if longest == 2 else 0
    ops.attention(q, out, k, v, token_seq=entry.to(torch.int32).cuda(), positions=positions.to(torch.int32).cuda(), block_table=table.cuda(),
                  num_heads=heads, num_kv_heads=kv_heads, head_dim=d, scale=d ** -0.5, longest=known)
    for e, (count, first) in enumerate(zip(counts, firsts)):
        pages = table[e, :needed[e]].long().cuda()
        keys, values = (z[pages].reshape(-1, kv_heads, d)[:first + count].double().repeat_interleave(heads // kv_heads, dim=1) for z in (k, v))
        own = entry == e
        score = torch.einsum("thd,shd->hts", q[own.cuda()].view(count, heads, d).double(), keys) * d ** -0.5
        hidden = torch.arange(first + count)[None] > torch.arange(first, first + count)[:, None]
        want = torch.einsum("hts,shd->thd", torch.softmax(score.masked_fill(hidden.cuda(), -float("inf")), -1), values).reshape(count, -1)
        # a few roundings of 32-bit sums of up to 320 products and weights
        assert float((out[own.cuda()].double() - want).norm() / want.norm()) < 2e-6


def test_longest_of_a_step():
    """Requests that bring one token do not count, few tokens and kernels that do not ask have no such number."""
    import numpy as np
    from types import SimpleNamespace
    from vipera_rs_b200.parts.attention import GQAttention

    assert GQAttention._longest(np.array([60] * 8), np.array([0] * 8)) == 64
    assert GQAttention._longest(np.array([100, 1, 24]), np.array([0, 4000, 0])) == 128
    assert GQAttention._longest(np.array([700, 1, 323]), np.array([0, 900, 40])) == 1024
    assert GQAttention._longest(np.array([1] * 70), np.array([900] * 70)) == 64
    part = SimpleNamespace(_general=lambda dtype: True, _longest=GQAttention._longest, dtype=torch.float32)
    assert GQAttention.step_forms(part, np.array([60, 5]), np.array([0, 70])) == {"attention.longest": 128}
    assert GQAttention.step_forms(part, np.array([60, 4]), np.array([0, 70])) == {}
    part._general = lambda dtype: False
    assert GQAttention.step_forms(part, np.array([600]), np.array([0])) == {}
