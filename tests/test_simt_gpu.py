"""The kernels that compute in 32 bits on the CUDA cores, at the sizes where their tiles, slabs and dispatch end,
against 64-bit restatements."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from vipera_rs_b200.kernels import ops

    return ops


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# rows at the borders of the tiles (8, 32, 64, 128), columns that end inside one, inner sizes of a part of a chunk,
# of fewer than eight slabs, of slabs that end early, of rows that do not start on 16 bytes
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 33, 64, 65, 129])
@pytest.mark.parametrize("n,k", [(64, 32), (70, 5), (96, 100), (130, 770), (200, 771), (1536, 808), (9600, 520)])
@pytest.mark.parametrize("types", ["f32", "bf16", "mixed"])
def test_product_tiles_and_slabs(m, n, k, types):
    ops = _ops()
    torch.manual_seed(m * 31 + n + k)
    a = torch.randn(m, k, device=DEV).to(torch.bfloat16 if types == "bf16" else torch.float32)
    w = torch.randn(n, k, device=DEV).to(torch.float32 if types == "f32" else torch.bfloat16)
    if types == "mixed":
        a = a.to(torch.float32)
    bias = torch.randn(n, device=DEV)
    out = torch.full((m, n), float("nan"), device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, bias=bias, out=out)
    # the error of a chain of k roundings of random sign, 2^-24 each, is some sqrt(k) 2^-24 of the sum at most
    assert _rel(out, a.double() @ w.double().T + bias.double()) < 2.0 ** -24 * (k ** 0.5 + 4)
    # a row's result does not depend on the rows beside it, within its class (up to eight rows, or more)
    beside = 1 if m <= 8 else 9
    last = torch.empty(beside, n, device=DEV)
    ops.gemm_simt(a[-beside:].contiguous(), w, epilogue=ops.EPI_STORE, bias=bias, out=last)
    assert torch.equal(last[-1], out[-1])
