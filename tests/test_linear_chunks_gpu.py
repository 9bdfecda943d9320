"""Linear attention's chunked products (csrc/kernels/linear_chunks.cuh) at the sizes where they can go wrong, against a
64-bit walk over the tokens: chunks of one token and of one too many, heads that fill a part of a tile, decays that are
gone within a token (the products' factors would leave their range), rows that the products do not take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = [[64, 1, 65], [300], [63, 129, 2]]
SIZES = [(4, 4), (64, 128), (100, 36), (128, 256), (256, 260), (18, 30)]


def _walk(q, k, v, decay, state, counts):
    out, ends, at = torch.empty(len(v), v.shape[1], v.shape[2], dtype=torch.float64), [], 0
    for entry, count in enumerate(counts):
        s = state[entry].double()
        for t in range(at, at + count):
            s = decay[t] * s + k[t][:, :, None] * v[t][:, None, :]
            out[t] = (q[t][:, None, :] @ s)[:, 0]
        ends.append(s)
        at += count
    return out, torch.stack(ends)


def _rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm())


def _step(counts):
    starts = torch.tensor([0] + counts).cumsum(0).to(torch.int32).to(DEV)
    slots = torch.arange(len(counts), dtype=torch.int32, device=DEV)
    fresh = torch.tensor([i % 2 for i in range(len(counts))], dtype=torch.int32, device=DEV)
    return starts, slots, fresh


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("dim,vdim", SIZES)
@pytest.mark.parametrize("far", [False, True, "all", "deep"])
def test_decays_per_channel(counts, dim, vdim, far):
    from vipera_rs_b200.kernels import ops

    torch.manual_seed(dim + vdim + sum(counts))
    heads, tokens, entries = 3, sum(counts), len(counts)
    proj = torch.randn(tokens, heads * (2 * dim + 2 * vdim))
    z = torch.randn(tokens, heads * dim)
    if far:   # single tokens that forget everything, and channels that forget within a few
        z[::17] = -3000.0
        z[:, ::5] -= 40.0
    if far in ("all", "deep"):   # every channel leaves the products' range within a chunk; within sixteen tokens, one in seven
        z = torch.randn(tokens, heads * dim) - 16.0 * 1.25
        if far == "deep":
            z[:, 1::7] -= 70.0
    offsets = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim)
    state = torch.randn(entries + 1, heads * dim * vdim)
    starts, slots, fresh = _step(counts)
    part = lambda at, size: proj[:, at:at + heads * size].double().view(tokens, heads, size)  # noqa: E731
    decay = torch.exp(torch.nn.functional.logsigmoid(z.double()) / 16.0).view(tokens, heads, dim, 1)
    begin = torch.stack([state[e].view(heads, dim, vdim) * (1 - e % 2) for e in range(entries)])
    want, ends = _walk(part(0, dim) * dim ** -0.5, part(offsets[1], dim), part(offsets[2], vdim), decay, begin, counts)
    gain, gate = torch.rand(vdim) + 0.5, part(offsets[3], vdim)
    want = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * gain.double() * gate * torch.sigmoid(gate)
    jobs = ops.scan_jobs(tokens, entries)
    kept, out = state.to(DEV), torch.full((tokens, heads * vdim), float("nan"), device=DEV)
    ops.gla(proj.to(DEV), z.to(DEV), offsets=offsets, heads=heads, dim=dim, vdim=vdim, q_scale=dim ** -0.5, tau=16.0,
            norm_weight=gain.to(DEV), norm_eps=1e-6, out_scale=1.0, state=kept, entry_starts=starts, state_slots=slots, fresh=fresh,
            num_entries=entries, partial=torch.empty(ops.gla_shares(dim), tokens, heads * vdim, device=DEV), out=out,
            log_decay=torch.empty(tokens, heads * dim, device=DEV),
            chunk_scratch=(torch.empty(jobs, heads * dim * vdim, device=DEV), torch.empty(jobs, heads * dim, device=DEV)))
    # exponents of up to 60 carry 60 * 2^-24 of relative error each, sums of some hundred terms a few 2^-24 more
    assert _rel(out.view(tokens, heads, vdim), want) < 2e-5
    assert _rel(kept[:entries].view(entries, heads, dim, vdim), ends) < 2e-5
    assert torch.equal(kept[entries].cpu(), state[entries])


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("dim,vdim", SIZES)
def test_decays_per_head(counts, dim, vdim):
    from vipera_rs_b200.kernels import ops

    torch.manual_seed(dim + vdim + sum(counts))
    decays = [0.999, 0.0, -0.7, 1.0]
    heads, tokens, entries = len(decays), sum(counts), len(counts)
    proj = torch.randn(tokens, heads * (2 * dim + 2 * vdim))
    offsets = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim)
    state = torch.randn(entries + 1, heads * dim * vdim)
    starts, slots, fresh = _step(counts)
    part = lambda at, size: proj[:, at:at + heads * size].double().view(tokens, heads, size)  # noqa: E731
    silu = torch.nn.functional.silu
    decay = torch.tensor(decays).double().view(1, heads, 1, 1).expand(tokens, -1, -1, -1)
    begin = torch.stack([state[e].view(heads, dim, vdim) * (1 - e % 2) for e in range(entries)])
    want, ends = _walk(silu(part(0, dim)), silu(part(offsets[1], dim)), silu(part(offsets[2], vdim)), decay, begin, counts)
    gain = torch.rand(heads * vdim) + 0.5
    want = want.view(tokens, -1)
    want = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * gain.double() * torch.sigmoid(part(offsets[3], vdim).reshape(tokens, -1))
    kept, out = state.to(DEV), torch.full((tokens, heads * vdim), float("nan"), device=DEV)
    ops.lightning(proj.to(DEV), offsets=offsets, heads=heads, dim=dim, vdim=vdim, decay=torch.tensor(decays, device=DEV),
                  norm_weight=gain.to(DEV), norm_eps=1e-6, state=kept, entry_starts=starts, state_slots=slots, fresh=fresh,
                  num_entries=entries, raw=torch.empty(tokens, heads * vdim, device=DEV), out=out,
                  chunk_state=torch.empty(ops.scan_jobs(tokens, entries), heads * dim * vdim, device=DEV))
    # sums of some hundred terms: a few 2^-24 each
    assert _rel(out, want) < 1e-5
    assert _rel(kept[:entries].view(entries, heads, dim, vdim), ends) < 1e-5
    assert torch.equal(kept[entries].cpu(), state[entries])


# a value that is not finite shows in its own token's output and in later ones', not in the ones before it in its chunk
@pytest.mark.parametrize("kind", ["channel", "head"])
@pytest.mark.parametrize("dim,vdim", [(128, 256), (128, 96)])
@pytest.mark.parametrize("token", [0, 7, 8, 45, 63, 77])
def test_values_that_are_not_finite(kind, dim, vdim, token):
    from vipera_rs_b200.kernels import ops

    torch.manual_seed(dim + vdim)
    heads, tokens = 2, 100
    proj = torch.randn(tokens, heads * (2 * dim + 2 * vdim), device=DEV)
    offsets = (0, heads * dim, 2 * heads * dim, 2 * heads * dim + heads * vdim)
    starts, slots, fresh = _step([tokens])
    jobs, outs = ops.scan_jobs(tokens, 1), []
    for value in (1.0, float("inf"), float("nan")):
        proj[token, offsets[2]:offsets[2] + heads * vdim] = value
        state, out = torch.zeros(2, heads * dim * vdim, device=DEV), torch.full((tokens, heads * vdim), -7.0, device=DEV)
        common = dict(offsets=offsets, heads=heads, dim=dim, vdim=vdim, norm_eps=1e-6, state=state, entry_starts=starts, state_slots=slots,
                      fresh=fresh, num_entries=1, out=out)
        scratch = torch.empty(jobs, heads * dim * vdim, device=DEV)
        if kind == "channel":
            ops.gla(proj, torch.ones(tokens, heads * dim, device=DEV), q_scale=dim ** -0.5, tau=16.0, norm_weight=torch.ones(vdim, device=DEV), out_scale=1.0,
                    partial=torch.empty(ops.gla_shares(dim), tokens, heads * vdim, device=DEV), log_decay=torch.empty(tokens, heads * dim, device=DEV),
                    chunk_scratch=(scratch, torch.empty(jobs, heads * dim, device=DEV)), **common)
        else:
            ops.lightning(proj, decay=torch.tensor([0.99, 0.5], device=DEV), norm_weight=torch.ones(heads * vdim, device=DEV),
                          raw=torch.empty(tokens, heads * vdim, device=DEV), chunk_state=scratch, **common)
        outs.append(out)
    for out in outs[1:]:
        assert torch.equal(out[:token], outs[0][:token]) and not torch.isfinite(out[token:]).any()


@pytest.mark.parametrize("dim,vdim", [(4, 4), (18, 30), (70, 36), (30, 7)])
def test_requests_of_many_chunks(dim, vdim):
    """The carry's forms for requests of many chunks (rows of whole pairs and not), beside one that ends within its first."""
    test_decays_per_head([850, 3], dim, vdim)
    test_decays_per_head([1700, 1], dim, vdim)
