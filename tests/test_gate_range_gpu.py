"""Output gates of the mixers' endings over the whole range in which a sigmoid is a number: as exact as their results' type, where
the exponential is near the largest 32-bit number too."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOKENS, HEADS = 3, 2


def _gates(width):
    gates = torch.linspace(-88.7, 20.0, TOKENS * width, device=DEV).view(width, TOKENS).T.contiguous()
    gates[:, :4] = torch.tensor([-88.72, -88.5, -88.03, -87.4], device=DEV)
    return gates


def _int(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _ending(kind, gates, vdim, dtype):
    """The kind's output [TOKENS, HEADS * vdim] of one token each of TOKENS requests, all but the gates the same."""
    from vipera_rs_b200.kernels import ops

    dim, generator = 64, torch.Generator(device=DEV).manual_seed(vdim)
    width = HEADS * vdim
    rest = torch.randn(TOKENS, 2 * HEADS * dim + width, device=DEV, generator=generator)
    offsets = (0, HEADS * dim, 2 * HEADS * dim, 2 * HEADS * dim + width)
    out = torch.zeros(TOKENS, width, dtype=dtype, device=DEV)
    gain = 2.0 ** 20
    common = dict(heads=HEADS, dim=dim, vdim=vdim, norm_eps=1e-6, entry_starts=_int(range(TOKENS + 1)), state_slots=_int(range(TOKENS)),
                  fresh=_int([1] * TOKENS), num_entries=TOKENS, out=out)
    if kind == "mlstm":
        proj = torch.cat([rest, gates, torch.ones(TOKENS, 2 * HEADS, device=DEV)], dim=1)
        ops.mlstm(proj, offsets=offsets + (offsets[3] + width, offsets[3] + width + HEADS), q_scale=dim ** -0.5, gate_cap=15.0, denom_eps=1e-6,
                  token_entry=_int(range(TOKENS)), single=True, state=torch.zeros(TOKENS, ops.mlstm_state_floats(HEADS, dim, vdim), device=DEV),
                  o_raw=torch.zeros(TOKENS, width, device=DEV), nm_scratch=torch.zeros(TOKENS, HEADS * (dim + 1), device=DEV),
                  norm_weight=torch.full((width,), gain, device=DEV), **common)
        return out
    proj, state = torch.cat([rest, gates], dim=1), torch.zeros(TOKENS, HEADS * dim * vdim, device=DEV)
    if kind == "lightning":
        ops.lightning(proj, offsets=offsets, decay=torch.tensor([0.9, 0.99], device=DEV), norm_weight=torch.full((width,), gain, device=DEV),
                      state=state, raw=torch.zeros(TOKENS, width, device=DEV), **common)
    else:
        ops.gla(proj, torch.ones(TOKENS, HEADS * dim, device=DEV), offsets=offsets, q_scale=dim ** -0.5, tau=16.0,
                norm_weight=torch.full((vdim,), gain, device=DEV), out_scale=1.0, state=state,
                partial=torch.zeros(ops.gla_shares(dim), TOKENS, width, device=DEV), log_decay=torch.zeros(TOKENS, HEADS * dim, device=DEV), **common)
    return out


@pytest.mark.parametrize("kind", ["mlstm", "lightning", "gla"])
@pytest.mark.parametrize("vdim", [36, 64, 130, 256, 640, 2048, 2100])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gates(kind, vdim, dtype):
    gates = _gates(HEADS * vdim)
    got = _ending(kind, gates, vdim, dtype).double()
    wide = _ending(kind, torch.zeros_like(gates) + 64.0, vdim, torch.float32).double()   # a sigmoid of one
    want = wide * torch.sigmoid(gates.double()) * (gates.double() / 64.0 if kind == "gla" else 1.0)
    # a rounding to the type, and the 32-bit steps: the exponential's two units in the last place, 2^-23 of the smallest normal number
    # times the gain for a sigmoid below that, and a few roundings
    limit = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * want.abs() + wide.abs() * 2.0 ** -148 * (89.0 / 64.0 if kind == "gla" else 1.0)
    assert bool(((got - want).abs() <= limit).all())


def test_gate_of_expanded_latents(monkeypatch):
    from test_latent_heads_gpu import HIDDEN, VDIM, _part, _step

    heads, tokens, outs = 2, 130, []
    part, _ = _part((heads, 256, 0, 16, "interleaved", True), 3, DEV)
    h = torch.randn(tokens, HIDDEN, device=DEV).bfloat16()
    gates = torch.linspace(-88.7, 20.0, tokens * heads * VDIM, device=DEV).view(tokens, -1)
    real, part.up_kv = part.proj, part.up_kv.clone()
    part.up_kv[heads * 128:] *= 2.0 ** 20
    for gate in (torch.full_like(gates, 64.0), gates):
        def proj(ctx, rows, *, epilogue, out, gate=gate):
            real(ctx, rows, epilogue=epilogue, out=out)
            out[:, part.g_off:part.g_off + heads * VDIM] = gate
        proj.out_features = real.out_features
        part.proj = proj
        context, view, _ = _step(part, [tokens], [0], 16, 256)
        assert part.expanded_rows(context) > 0
        part.forward(context, h, torch.zeros(tokens, HIDDEN, device=DEV), view, True)
        outs.append(context.workspace.get("latent.out", (tokens, heads * VDIM), torch.bfloat16).double().clone())
    want = outs[0] * torch.sigmoid(gates.double())
    # two roundings to bfloat16, and 2^-23 of the smallest normal number for a sigmoid below that
    assert bool(((outs[1] - want).abs() <= 2.0 ** -7 * want.abs() + outs[0].abs() * 2.0 ** -148).all())
