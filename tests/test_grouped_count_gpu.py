"""Grouped products of which only the first tiles of the table are there: those are computed as without a count, rows past
them stay as they were."""
import pytest
import torch

from vipera_rs_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [128, 192, 512])
@pytest.mark.parametrize("ending", [ops.EPI_STORE, ops.EPI_GATED])
@pytest.mark.parametrize("tiles, count", [(1, 0), (1, 1), (7, 6), (7, 1), (40, 33), (40, 40), (40, 90)])
def test_counted_tiles(tiles, count, ending, n):
    torch.manual_seed(0)
    k, groups = 128, 3
    a = torch.randn(tiles * 128, k, device=DEV).bfloat16()
    w = torch.randn(groups, n, k, device=DEV).bfloat16()
    table = torch.randint(0, groups, (tiles,), device=DEV, dtype=torch.int32)
    if ending == ops.EPI_STORE:
        outs = [torch.full((tiles * 128, n), 7.0, device=DEV) for _ in range(2)]
    else:
        outs = [torch.full((tiles * 128, n // 2), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    ops.gemm_tc_grouped(a, w, table, epilogue=ending, out=outs[0])
    ops.gemm_tc_grouped(a, w, table, epilogue=ending, out=outs[1], tile_count=torch.tensor([count], device=DEV, dtype=torch.int32))
    torch.cuda.synchronize()
    ops.check_kernel_status(DEV)
    rows = min(count, tiles) * 128
    assert torch.equal(outs[0][:rows], outs[1][:rows])   # a tile's sums do not depend on which block takes it
    assert bool((outs[1][rows:] == 7.0).all())
    if ending == ops.EPI_STORE and rows:
        want = torch.stack([a[i * 128:(i + 1) * 128].double() @ w[int(table[i])].double().T for i in range(tiles)]).view(-1, n)[:rows]
        # 32-bit sums of 128 exact products, whose absolute values add up to some 82 and at most 200 here
        assert float((outs[1][:rows] - want).abs().max()) < 128 * 2.0 ** -24 * 200
