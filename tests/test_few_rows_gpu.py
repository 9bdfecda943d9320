"""32-bit products of up to eight rows whose blocks share a run of A: a row's numbers do not depend on how many rows there are,
bit for bit, across the line where the form changes; columns and inner sizes that end inside a block's."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,k", [(32 * 488, 260), (1537, 2700), (4097, 1028), (96, 41700), (14209, 1540)])
@pytest.mark.parametrize("ending", ["store", "residual", "gated"])
def test_rows_alone_and_together(n, k, ending):
    from vipera_rs_b200.kernels import ops

    if ending == "gated":
        n = n // 32 * 32
    torch.manual_seed(n + k)
    a, w, bias = torch.randn(8, k, device=DEV), torch.randn(n, k, device=DEV), torch.randn(n, device=DEV)

    def product(rows):
        if ending == "residual":
            out = torch.ones(len(rows), n, device=DEV)
            ops.gemm_simt(rows, w, epilogue=ops.EPI_RESIDUAL, bias=bias, resid=out)
            return out
        out = torch.full((len(rows), n // 2 if ending == "gated" else n), float("nan"), device=DEV)
        ops.gemm_simt(rows, w, epilogue=ops.EPI_SWIGLU if ending == "gated" else ops.EPI_STORE, bias=bias, out=out)
        return out

    alone = torch.cat([product(a[i:i + 1].contiguous()) for i in range(8)])
    for count in (2, 3, 4, 5, 8):
        assert torch.equal(product(a[:count].contiguous()), alone[:count])
    z = a.double() @ w.double().T + bias.double()
    if ending == "gated":
        z = z.view(8, n // 32, 2, 16)
        want = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(8, n // 2)
    else:
        want = z + (1.0 if ending == "residual" else 0.0)
    # chains of K / 128 products a lane: 2^-24 times the root of their number, and the factors around
    assert float((alone.double() - want).norm() / want.norm()) < 2e-6


@pytest.mark.parametrize("n,k", [(4097, 2100), (9001, 1000), (2049, 3076), (2049, 2052), (14209, 1028)])
@pytest.mark.parametrize("ending", ["store", "gated"])
def test_members_of_enough_runs(n, k, ending):
    """Four, two and eight blocks of a cluster on either side of three runs a block, and four rows on eight."""
    test_rows_alone_and_together(n, k, ending)
