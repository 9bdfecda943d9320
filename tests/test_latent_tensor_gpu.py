"""The tcgen05 fold over latents (csrc/kernels/latent_tc.cuh) through the mixer that runs it, against a 64-bit
restatement: every count of column parts, rows that end inside a tile, several requests in one tile, windows that begin
inside a tile of keys, pages of odd sizes, pages that hold no number."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _plain(w, h, kept, counts, firsts, heads, dim, rot, rank, vdim, window, sink):
    frequency = 10000.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
    angle = torch.cat([torch.arange(f, f + c) for c, f in zip(counts, firsts)]).double()[:, None] * frequency
    cos, sin = torch.cos(angle).to(DEV), torch.sin(angle).to(DEV)

    def turn(z, c, s):
        a, b = z[..., 0::2], z[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)

    q = (h @ w["p.q.weight"].T).view(-1, heads, dim + rot)
    turned = turn(q[..., dim:], cos[:, None], sin[:, None])
    down = h @ w["p.dkv.weight"].T
    latent = down[:, :rank] / torch.sqrt((down[:, :rank] ** 2).mean(-1, keepdim=True) + 1e-6) * w["p.dkv.norm.weight"]
    key_part = turn(down[:, rank:], cos, sin)
    up_k, up_v = w["p.uk.weight"].view(heads, dim, rank), w["p.uv.weight"].view(heads, vdim, rank)
    out, at = torch.empty(len(h), heads, vdim, dtype=torch.float64, device=DEV), 0
    for (c0, r0), count, first in zip(kept, counts, firsts):
        c, r = torch.cat([c0.double(), latent[at:at + count]]), torch.cat([r0.double(), key_part[at:at + count]])
        key, query = torch.arange(len(c), device=DEV)[None], torch.arange(first, first + count, device=DEV)[:, None]
        hidden = (key > query) | ((key <= query - window) if window else (key < 0))
        for head in range(heads):
            score = q[at:at + count, head, :dim] @ (c @ up_k[head].T).T + turned[at:at + count, head] @ r.T
            score = (score * (dim + rot) ** -0.5).masked_fill(hidden, -float("inf"))
            if sink:
                score = torch.cat([score, w["p.sink.weight"][head].expand(count, 1)], dim=1)
            out[at:at + count, head] = torch.softmax(score, -1)[:, :len(c)] @ (c @ up_v[head].T)
        at += count
    return out.reshape(len(h), -1) @ w["p.o.weight"].T


# few heads want many tokens: the rule sends shorter steps to the other form
LONG = [([1100], [0]), ([2000, 1, 2100], [3, 60, 0]), ([1500, 1501], [0, 70]), ([700], [333])]
SHORT = [([520], [0]), ([300, 1, 129, 130], [70, 200, 0, 63]), ([64, 65, 63, 400], [0, 1, 300, 0]), ([700, 1, 900], [0, 60, 10])]
SOME = [([520], [0]), ([700, 1, 900], [0, 60, 10]), ([1000, 63, 1100], [5, 300, 0]), ([2000, 1, 2100], [3, 60, 0])]
CASES = [(case, sizes) for cases, sizes in [(LONG, (3, 512, 64, 0, 16)), (SOME, (12, 512, 64, 100, 16)), (LONG[:3] + SOME[2:3], (5, 256, 32, 0, 7)),
                                             (SOME, (7, 64, 8, 50, 64)), (SHORT, (32, 384, 24, 0, 1)), (SHORT, (128, 320, 64, 333, 16))] for case in cases]


@pytest.mark.parametrize("case,sizes", CASES)
def test_fold(case, sizes, monkeypatch):
    (counts, firsts), (heads, rank, rot, window, page) = case, sizes
    from vipera_rs_b200.config.registry import MIXERS
    from vipera_rs_b200.config.spec import PartSpec
    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.parts.base import PagedKVView, StepContext, Workspace

    real, took = ops._function, []

    def asked(family, name, arguments):
        function = real(family, name, arguments)
        return (lambda params: took.append(function(params)) or took[-1]) if name == "vipera_latent_fold_tensor" else function

    monkeypatch.setattr(ops, "_function", asked)
    torch.manual_seed(sum(counts) + heads + rank)
    hidden, dim, vdim, sink, tokens, entries = 256, 32, 64, bool(window), sum(counts), len(counts)
    position = PartSpec("rope_interleaved", {"head_dim": rot, "rotary_dims": rot, "theta": 10000.0, "scaling": None,
                                             "exact_angles": True, "max_positions": 4096})
    params = {"hidden_size": hidden, "num_heads": heads, "head_dim": dim, "rot_dim": rot, "value_dim": vdim, "kv_rank": rank,
              "softmax_scale": (dim + rot) ** -0.5, "norm_eps": 1e-6, "position": position}
    if window:
        params.update(window=window, sink="learned")
    cls = MIXERS.find("latent_attention")
    w = {}
    for name, spec in cls.schema(params, "p").items():
        std = {"p.q.weight": 0.1, "p.uk.weight": 0.08, "p.uv.weight": 0.08, "p.sink.weight": 1.5}.get(name, 0.06)
        tensor = torch.randn(*spec.shape, device=DEV) * std + (1.0 if "norm" in name else 0.0)
        w[name] = tensor if "norm" in name or "sink" in name else tensor.bfloat16()
    part = cls(params, "p", w, torch.bfloat16, DEV)
    part.prepare(4096)
    h = torch.randn(tokens, hidden, device=DEV).bfloat16()
    kept = [(torch.randn(f, rank, device=DEV).bfloat16(), torch.randn(f, rot, device=DEV).bfloat16()) for f in firsts]
    longest = max(c + f for c, f in zip(counts, firsts))
    width = -(-longest // page)
    table = torch.randperm(entries * width).view(entries, width).to(torch.int32)
    k = torch.full((entries * width, page, 1, rank), float("nan"), device=DEV, dtype=torch.bfloat16)
    v = torch.full((entries * width, page, 1, rot), float("nan"), device=DEV, dtype=torch.bfloat16)
    for e, (c, r) in enumerate(kept):
        at = torch.arange(firsts[e])
        where = (table[e].long()[at // page].to(DEV), (at % page).to(DEV))
        k[where[0], where[1], 0], v[where[0], where[1], 0] = c, r
    if window:   # pages that no query's window reaches any more are given back
        for e, f in enumerate(firsts):
            gone = max(0, f - window + 1) // page
            k[table[e, :gone].long().to(DEV)], v[table[e, :gone].long().to(DEV)] = float("nan"), float("nan")
            table[e, :gone] = -1
    device = lambda values: torch.from_numpy(np.ascontiguousarray(values, dtype=np.int32)).to(DEV)  # noqa: E731
    context = StepContext(
        num_tokens=tokens, num_entries=entries, tokens=device(np.zeros(tokens)),
        positions=device(np.concatenate([np.arange(f, f + c) for c, f in zip(counts, firsts)])),
        token_entry=device(np.repeat(np.arange(entries), counts)), entry_starts=device(np.cumsum([0] + counts)), entry_pos0=device(firsts),
        state_slots=device(np.arange(entries)), fresh=device(np.zeros(entries)), block_tables=[table.to(DEV)], logit_rows=None,
        num_logit_rows=0, host_counts=counts, host_pos0=firsts, max_count=max(counts), max_kv_len=longest, all_single=False,
        any_single=1 in counts, dtype=torch.bfloat16, workspace=Workspace(DEV))
    out = torch.zeros(tokens, hidden, device=DEV)
    part.forward(context, h, out, PagedKVView(0, k, v, page, window or None), True)
    torch.cuda.synchronize()
    ops.check_kernel_status(DEV)
    assert took == [1]   # the tcgen05 form ran
    want = _plain({n: t.double() for n, t in w.items()}, h.double(), kept, counts, firsts, heads, dim, rot, rank, vdim, window, sink)
    # bfloat16 operands of five products in a row (queries, latents, weights, mixed latents, heads): 2^-9 each and a little
    assert float((out.double() - want).norm() / want.norm()) < 1e-2
    worst = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(worst.max()) < 4e-2
