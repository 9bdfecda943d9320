"""The mLSTM cell as a walk over prepared chunks (csrc/kernels/mlstm_walk.cuh): chunks that end early, several requests of
unequal length, a state carried into a second step, every size of head it takes, against 64 bits; and where it is chosen."""
import numpy as np
import pytest
import torch

DEV = "cuda:0"


def _plain(proj, offsets, heads, dim, vdim, cap, states, starts):
    q, k, v, g, i, f = (proj.double()[:, o:] for o in offsets)
    out = torch.zeros(len(proj), heads, vdim, dtype=torch.float64, device=DEV)
    for e, (S, n, m) in enumerate(states):
        for t in range(starts[e], starts[e + 1]):
            li, lf = cap * torch.tanh(i[t, :heads] / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(f[t, :heads] / cap))
            qt = q[t, :heads * dim].view(heads, dim) * dim ** -0.5
            kt, vt = k[t, :heads * dim].view(heads, dim), v[t, :heads * vdim].view(heads, vdim)
            new = torch.maximum(lf + m, li)
            keep, take = torch.exp(lf + m - new), torch.exp(li - new)
            S.mul_(keep[:, None, None]).add_(take[:, None, None] * kt[:, :, None] * vt[:, None, :])
            n.mul_(keep[:, None]).add_(take[:, None] * kt)
            m.copy_(new)
            out[t] = torch.einsum("hdv,hd->hv", S, qt) / (torch.maximum((n * qt).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
    normed = out / torch.sqrt((out * out).mean(-1, keepdim=True) + 1e-6)
    return normed.reshape(len(proj), -1) * torch.sigmoid(g[:, :heads * vdim])


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [[[1]], [[63], [2]], [[64], [65]], [[130, 1, 64], [3, 200, 1]], [[17, 70], [65, 1]]])
@pytest.mark.parametrize("sizes", [(2, 64, 32), (1, 128, 96), (3, 256, 64)])
def test_walk(steps, sizes):
    from vipera_rs_b200.kernels import ops

    heads, dim, vdim = sizes
    torch.manual_seed(heads * 100 + len(steps[0]))
    widths = (heads * dim, heads * dim, heads * vdim, heads * vdim, heads, heads)
    offsets = tuple(int(o) for o in np.concatenate([[0], np.cumsum(widths)[:-1]]))
    width, entries = (sum(widths) + 7) // 8 * 8, len(steps[0])
    state = torch.full((entries + 1, ops.mlstm_state_floats(heads, dim, vdim)), float("nan"), device=DEV)
    slots = torch.arange(entries, 0, -1, dtype=torch.int32, device=DEV)
    kept = [(torch.zeros(heads, dim, vdim, dtype=torch.float64, device=DEV), torch.zeros(heads, dim, dtype=torch.float64, device=DEV),
             torch.zeros(heads, dtype=torch.float64, device=DEV)) for _ in range(entries)]
    device = lambda values: torch.from_numpy(np.ascontiguousarray(values, dtype=np.int32)).to(DEV)  # noqa: E731
    for number, counts in enumerate(steps):
        tokens, starts = sum(counts), np.concatenate([[0], np.cumsum(counts)])
        proj = torch.randn(tokens, width, device=DEV)
        proj[:, offsets[5]:offsets[5] + heads] += 3.0
        assert ops.mlstm_walk_takes(proj, offsets, dim, vdim)
        jobs = tokens // ops.MLSTM_CHUNK + entries
        scratch = {name: torch.full((jobs, size), float("nan"), dtype=dtype, device=DEV)
                   for name, (size, dtype) in ops.mlstm_walk_scratch(heads, dim, vdim).items()}
        out = torch.zeros(tokens, heads * vdim, dtype=torch.bfloat16, device=DEV)
        ops.mlstm(proj, offsets=offsets, heads=heads, dim=dim, vdim=vdim, q_scale=dim ** -0.5, gate_cap=15.0, denom_eps=1e-6,
                  entry_starts=device(starts), state_slots=slots, fresh=device([number == 0] * entries),
                  token_entry=device(np.repeat(np.arange(entries), counts)), num_entries=entries, single=False, state=state,
                  o_raw=torch.full((tokens, heads * vdim), float("nan"), device=DEV),
                  nm_scratch=torch.zeros(entries, heads * (dim + 1), device=DEV), norm_weight=torch.ones(heads * vdim, device=DEV),
                  norm_eps=1e-6, out=out, walk_scratch=scratch)
        torch.cuda.synchronize()
        ops.check_kernel_status(DEV)
        want = _plain(proj, offsets, heads, dim, vdim, 15.0, kept, starts)
        # q, k, v, the weights and the state enter products in bfloat16: 2^-9 each, and the output is rounded to it
        assert float((out.double() - want).norm() / want.norm()) < 1e-2
        for e in range(entries):
            row, (S, n, m) = state[int(slots[e])].double(), kept[e]
            for got, exact, bound in ((row[:S.numel()], S, 1e-2), (row[S.numel():S.numel() + n.numel()], n, 1e-2),
                                      (row[S.numel() + n.numel():S.numel() + n.numel() + heads], m, 1e-4)):
                assert float((got - exact.reshape(-1)).norm()) <= bound * float(exact.norm()) + 1e-4


def test_rule():
    """Long steps with large states walk, long steps with small states compute their chunks at once, short ones of large heads walk."""
    from types import SimpleNamespace

    from vipera_rs_b200.parts.mlstm import MLSTM

    def walks(heads, dim, vdim, counts, known=True, width=64):
        part = SimpleNamespace(heads=heads, dim=dim, vdim=vdim, offsets=(0, 8, 16), AT_ONCE_FROM=256)
        ctx = SimpleNamespace(num_tokens=sum(counts), num_entries=len(counts), host_counts=counts if known else [], max_count=sum(counts))
        return MLSTM.walks(part, ctx, torch.zeros(1, width))

    assert walks(8, 256, 512, [2048]) and walks(8, 256, 512, [2048], known=False)
    assert not walks(4, 64, 128, [2048]) and not walks(4, 128, 256, [1024])
    assert walks(4, 128, 256, [65]) and not walks(4, 64, 128, [65])
    assert not walks(8, 256, 500, [2048]) and not walks(8, 256, 512, [2048], width=62) and not walks(8, 96, 512, [2048])
    assert not walks(8, 256, 512, [65] + [1] * 40)


def test_the_plan_holds_the_scratch():
    """Whatever step walks, its scratch fits what the memory plan counts for it: many short portions among them."""
    from types import SimpleNamespace

    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.parts.mlstm import MLSTM

    walked = 0
    for heads, dim, vdim in ((8, 256, 512), (4, 128, 256), (4, 64, 128)):
        part = SimpleNamespace(heads=heads, dim=dim, vdim=vdim, offsets=(0, 8, 16), AT_ONCE_FROM=256)
        params = {"num_heads": heads, "head_dim": dim, "value_dim": vdim}
        for entries in (1, 2, 3, 8, 9, 31, 32, 33, 40, 64, 255, 256, 341):
            for tokens in (48, 96, 130, 200, 255, 300, 512, 1030, 2048):
                ctx = SimpleNamespace(num_tokens=tokens, num_entries=entries, host_counts=[], max_count=tokens)
                if entries > tokens or not MLSTM.walks(part, ctx, torch.zeros(1, 64)):
                    continue
                walked += 1
                scratch = sum(size * dtype.itemsize for size, dtype in ops.mlstm_walk_scratch(heads, dim, vdim).values())
                others = tokens * ((2 * heads * (dim + vdim) + 2 * heads) * 4 + heads * vdim * 6 + heads * (dim + 1) * 4)
                assert (tokens // ops.MLSTM_CHUNK + entries) * scratch <= MLSTM.workspace_bytes(params, tokens, 2) - others
    assert walked > 50


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [[[65, 1, 64, 3, 130, 1, 20], [2, 64, 1, 1, 66, 128, 9]], [[5] * 40]])
def test_walk_of_many_requests(steps):
    """More requests than a handful, lone tokens among them: their chunks lie one request after another."""
    test_walk(steps, (2, 128, 64))
