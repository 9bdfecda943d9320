"""Latent attention that expands every head's keys and values once a step (csrc/kernels/latent_heads.cuh), through the mixer,
against a 64-bit restatement: tiles of 128 queries and keys that end inside one, several requests, windows that begin inside
a tile, both rotations, pages of odd sizes, pages that hold no number; and the rule that chooses the form."""
import numpy as np
import pytest
import torch

from test_latent_tensor_gpu import _plain

DEV = "cuda:0"
DIM, ROT, VDIM, HIDDEN = 128, 64, 128, 256


def _part(sizes, seed, device):
    from vipera_rs_b200.config.registry import MIXERS
    from vipera_rs_b200.config.spec import PartSpec

    heads, rank, window, page, style, gated = sizes
    position = PartSpec("rope_" + style, {"head_dim": ROT, "rotary_dims": ROT, "theta": 10000.0, "scaling": None,
                                          "exact_angles": True, "max_positions": 4096})
    params = {"hidden_size": HIDDEN, "num_heads": heads, "head_dim": DIM, "rot_dim": ROT, "value_dim": VDIM, "kv_rank": rank,
              "softmax_scale": (DIM + ROT) ** -0.5, "norm_eps": 1e-6, "position": position, "output_gate": gated}
    if window:
        params.update(window=window, sink="learned")
    cls, w = MIXERS.find("latent_attention"), {}
    torch.manual_seed(seed)
    for name, spec in cls.schema(params, "p").items():
        std = {"p.q.weight": 0.06, "p.uk.weight": 0.06, "p.uv.weight": 0.06, "p.sink.weight": 1.5}.get(name, 0.06)
        tensor = torch.randn(*spec.shape, device=device) * std + (1.0 if "norm" in name else 0.0)
        w[name] = tensor if "norm" in name or "sink" in name else tensor.bfloat16()
    part = cls(params, "p", w, torch.bfloat16, device)
    return part, w


STEPS = [([64], [0]), ([128], [128]), ([129, 1, 127], [0, 300, 5]), ([1, 257], [700, 1]), ([500, 3], [333, 0]), ([1030], [0])]
SIZES = [(3, 512, 0, 16, "interleaved", False), (5, 256, 100, 7, "interleaved", True), (2, 64, 333, 1, "neox", True), (33, 320, 0, 64, "neox", False)]


@pytest.mark.gpu
@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("sizes", SIZES)
def test_expanded(step, sizes, monkeypatch):
    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.parts import latent
    from vipera_rs_b200.parts.base import PagedKVView, StepContext, Workspace

    monkeypatch.setattr(latent, "EXPANDED_SHARE", 0)
    (counts, firsts), (heads, rank, window, page, style, gated) = step, sizes
    tokens, entries = sum(counts), len(counts)
    part, w = _part(sizes, tokens + heads + rank, DEV)
    part.prepare(4096)
    h = torch.randn(tokens, HIDDEN, device=DEV).bfloat16()
    kept = [(torch.randn(f, rank, device=DEV).bfloat16(), torch.randn(f, ROT, device=DEV).bfloat16()) for f in firsts]
    longest = max(c + f for c, f in zip(counts, firsts))
    width = -(-longest // page)
    table = torch.randperm(entries * width).view(entries, width).to(torch.int32)
    k = torch.full((entries * width, page, 1, rank), float("nan"), device=DEV, dtype=torch.bfloat16)
    v = torch.full((entries * width, page, 1, ROT), float("nan"), device=DEV, dtype=torch.bfloat16)
    for e, (c, r) in enumerate(kept):
        at = torch.arange(firsts[e])
        where = (table[e].long()[at // page].to(DEV), (at % page).to(DEV))
        k[where[0], where[1], 0], v[where[0], where[1], 0] = c, r
        gone = max(0, firsts[e] - window + 1) // page if window else 0   # pages no window reaches any more are given back
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
    for known in (True, False):   # as a step whose requests the host knows, and as a captured one
        context.host_counts = counts if known else []
        assert part.expanded_rows(context) > 0
        out = torch.zeros(tokens, HIDDEN, device=DEV)
        part.forward(context, h, out, PagedKVView(0, k, v, page, window or None), True)
        torch.cuda.synchronize()
        ops.check_kernel_status(DEV)
        wide = {n: t.double() for n, t in w.items()}
        if style == "neox":   # the restatement turns neighbours: put the values that turn together side by side
            order = torch.arange(ROT, device=DEV).view(2, ROT // 2).T.reshape(-1)
            rows = torch.cat([torch.arange(DIM, device=DEV), DIM + order])
            wide["p.q.weight"] = wide["p.q.weight"].view(heads, DIM + ROT, HIDDEN)[:, rows].reshape(heads * (DIM + ROT), HIDDEN)
            wide["p.dkv.weight"] = torch.cat([wide["p.dkv.weight"][:rank], wide["p.dkv.weight"][rank:][order]])
        past = [(c, r[:, order] if style == "neox" else r) for c, r in kept]
        eye = dict(wide, **{"p.o.weight": torch.eye(heads * VDIM, dtype=torch.float64, device=DEV)})
        mixed = _plain(eye, h.double(), past, counts, firsts, heads, DIM, ROT, rank, VDIM, window, bool(window))
        if gated:
            mixed = mixed * torch.sigmoid(h.double() @ wide["p.g.weight"].T)
        want = mixed @ wide["p.o.weight"].T
        # bfloat16 operands of five products in a row (queries, latents, keys or values, weights, heads): 2^-9 each and a little
        assert float((out.double() - want).norm() / want.norm()) < 1e-2
        assert float(((out.double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 4e-2


def test_rule():
    """Rows are each request's visible keys rounded up to 128; lone tokens, few tokens, rows that outweigh their queries and
    other shapes of head stay with the latents, and what a captured step counts on holds for every step of its class."""
    from types import SimpleNamespace

    part, _ = _part((3, 512, 1024, 16, "interleaved", True), 0, "cpu")

    def step(counts, firsts, **changes):
        fields = dict(host_counts=counts, host_pos0=firsts, num_tokens=sum(counts), num_entries=len(counts), dtype=torch.bfloat16,
                      all_single=max(counts) == 1, max_kv_len=max(c + f for c, f in zip(counts, firsts)))
        return SimpleNamespace(**dict(fields, **changes))

    assert part.expanded_rows(step([2048], [0])) == 2048
    assert part.expanded_rows(step([300, 1], [3000, 5000])) == 1408 + 1024     # no further back than the window
    assert part.expanded_rows(step([1] * 64, [2000] * 64)) == 0
    assert part.expanded_rows(step([63], [0])) == 0
    assert part.expanded_rows(step([64] + [1] * 10, [0] + [2000] * 10)) == 0
    assert part.expanded_rows(step([2048], [0], dtype=torch.float32)) == 0
    for counts, firsts in (([900, 100, 24], [0, 70, 3000]), ([1024], [7000]), ([1023, 1], [0, 4000])):
        known, captured = step(counts, firsts), step(counts, firsts, host_counts=[])
        if part.expanded_rows(captured):
            assert 0 < part.expanded_rows(known) <= part.expanded_rows(captured)


def _step(part, counts, firsts, page, rank, window=0, kept=None):
    """The step's context and pages that hold `kept` (random latents where none are given)."""
    from vipera_rs_b200.parts.base import PagedKVView, StepContext, Workspace

    tokens, entries, longest = sum(counts), len(counts), max(c + f for c, f in zip(counts, firsts))
    width = -(-longest // page)
    table = torch.arange(entries * width).view(entries, width).to(torch.int32)
    kept = kept or [(torch.randn(f, rank, device=DEV).bfloat16(), torch.randn(f, ROT, device=DEV).bfloat16()) for f in firsts]
    k = torch.zeros(entries * width, page, 1, rank, device=DEV, dtype=torch.bfloat16)
    v = torch.zeros(entries * width, page, 1, ROT, device=DEV, dtype=torch.bfloat16)
    for e, (c, r) in enumerate(kept):
        k.view(entries, width * page, rank)[e, :len(c)], v.view(entries, width * page, ROT)[e, :len(c)] = c, r
    device = lambda values: torch.from_numpy(np.ascontiguousarray(values, dtype=np.int32)).to(DEV)  # noqa: E731
    context = StepContext(
        num_tokens=tokens, num_entries=entries, tokens=device(np.zeros(tokens)),
        positions=device(np.concatenate([np.arange(f, f + c) for c, f in zip(counts, firsts)])),
        token_entry=device(np.repeat(np.arange(entries), counts)), entry_starts=device(np.cumsum([0] + counts)), entry_pos0=device(firsts),
        state_slots=device(np.arange(entries)), fresh=device(np.zeros(entries)), block_tables=[table.to(DEV)], logit_rows=None,
        num_logit_rows=0, host_counts=counts, host_pos0=firsts, max_count=max(counts), max_kv_len=longest, all_single=False,
        any_single=1 in counts, dtype=torch.bfloat16, workspace=Workspace(DEV))
    part.prepare(4096)
    return context, PagedKVView(0, k, v, page, window or None), kept


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(3, 512, 0, 16, "interleaved", False), (2, 256, 100, 7, "neox", True)])
@pytest.mark.parametrize("token", [0, 1, 63, 64, 100, 127, 128, 200, 299])
def test_tokens_that_are_not_finite(sizes, token):
    """A token whose numbers are not finite shows in its own output and in those of the tokens that see it, nowhere else."""
    heads, rank, window, page, style, gated = sizes
    part, _ = _part(sizes, 5, DEV)
    h = torch.randn(370, HIDDEN, device=DEV).bfloat16()
    outs = []
    for value in (None, float("nan"), float("inf")):
        if value is not None:
            h[token] = value
        context, view, _ = _step(part, [300, 70], [0, 0], page, rank, window)
        assert part.expanded_rows(context) > 0
        out = torch.zeros(370, HIDDEN, device=DEV)
        part.forward(context, h, out, view, True)
        outs.append(out)
    end = min(300, token + window) if window else 300
    for out in outs[1:]:
        assert torch.equal(out[:token], outs[0][:token]) and torch.equal(out[end:], outs[0][end:])
        assert not torch.isfinite(out[token:end]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("window", [0, 100])
def test_values_that_are_not_finite(window):
    """Two values of a head are infinite for every token: they show in those columns of every token's heads, in no other column."""
    sizes = (2, 256, window, 16, "interleaved", False)
    mixed = []
    for value in (None, float("inf")):
        part, _ = _part(sizes, 7, DEV)
        if value is not None:
            part.up_kv[(2 + 1) * 128 + 5, 17], part.up_kv[(2 + 1) * 128 + 100, 30] = value, -value     # head 1, its values 5 and 100
        torch.manual_seed(3)
        h = torch.randn(333, HIDDEN, device=DEV).bfloat16()
        context, view, _ = _step(part, [333], [40], 16, 256, window)
        assert part.expanded_rows(context) > 0
        part.forward(context, h, torch.zeros(333, HIDDEN, device=DEV), view, True)
        mixed.append(context.workspace.get("latent.out", (333, 256), torch.bfloat16).clone())
    columns = (torch.arange(256, device=DEV) != 128 + 5) & (torch.arange(256, device=DEV) != 128 + 100)
    assert torch.equal(mixed[0][:, columns], mixed[1][:, columns])
    assert not torch.isfinite(mixed[1][:, ~columns]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("own_cache", [True, False])
def test_query_latents_and_shared_pages(gated, own_cache):
    """Queries that come through a latent (a buffer of their own, the gate in another), and a layer that reads another's pages."""
    from vipera_rs_b200.kernels import ops

    heads, rank, q_rank, counts, firsts = 3, 256, 96, [150, 1, 200], [70, 40, 0]
    parts, weights = [], []
    for index in range(1 if own_cache else 2):
        writer = index == 0
        part, w = _part((heads, rank, 0, 16, "interleaved", gated), index, DEV)
        params = dict(part.params, q_rank=q_rank, own_cache=writer)
        schema = type(part).schema(params, "p")
        for name, std in (("p.dq.weight", 0.06), ("p.uq.weight", 0.1)):
            w[name] = (torch.randn(*schema[name].shape, device=DEV) * std).bfloat16()
        w["p.dq.norm.weight"] = torch.randn(q_rank, device=DEV) * 0.1 + 1.0
        parts.append(type(part)(params, "p", {name: w[name] for name in schema}, torch.bfloat16, DEV))
        weights.append(w)
    h = torch.randn(sum(counts), HIDDEN, device=DEV).bfloat16()
    context, view, kept = _step(parts[-1], counts, firsts, 16, rank)
    parts[0].prepare(4096)
    for part in parts:
        assert part.expanded_rows(context) > 0
        out = torch.zeros(len(h), HIDDEN, device=DEV)
        part.forward(context, h, out, view, part.own_cache)
    torch.cuda.synchronize()
    ops.check_kernel_status(DEV)
    wide = {name: t.double() for name, t in weights[-1].items()}
    for name in ("p.dkv.weight", "p.dkv.norm.weight"):
        wide[name] = weights[0][name].double()
    # the restatement's queries are a product of its rows: the query latents stand beside them
    low = h.double() @ wide["p.dq.weight"].T
    low = low / torch.sqrt((low * low).mean(-1, keepdim=True) + 1e-6) * wide["p.dq.norm.weight"]
    rows, zeros = torch.cat([h.double(), low], dim=1), lambda n, m: torch.zeros(n, m, dtype=torch.float64, device=DEV)  # noqa: E731
    wide["p.q.weight"] = torch.cat([zeros(heads * (DIM + ROT), HIDDEN), wide["p.uq.weight"]], dim=1)
    wide["p.dkv.weight"] = torch.cat([wide["p.dkv.weight"], zeros(rank + ROT, q_rank)], dim=1)
    eye = dict(wide, **{"p.o.weight": torch.eye(heads * VDIM, dtype=torch.float64, device=DEV)})
    want = _plain(eye, rows, kept, counts, firsts, heads, DIM, ROT, rank, VDIM, 0, False)
    if gated:
        want = want * torch.sigmoid(h.double() @ wide["p.g.weight"].T)
    want = want @ wide["p.o.weight"].T
    # bfloat16 operands of six products in a row: 2^-9 each and a little
    assert float((out.double() - want).norm() / want.norm()) < 1e-2
    assert float(((out.double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 4e-2


def _folder(monkeypatch, window):
    """A one-layer model of such heads, its scales such that attention outweighs the tokens' own rows, and sharp enough to show."""
    import nuvezen_cases as cases

    name = f"heads_of_128_{window}"
    layer = cases.latent(heads=3, dim=DIM, rot_dim=ROT, vdim=VDIM, rank=256, q_rank=96, window=window, base=10000.0, scale=192 ** -0.5)
    monkeypatch.setitem(cases.CONFIGS, name, cases.config([layer], width=256, vocab=300, eps=1e-5))
    monkeypatch.setitem(cases.RULES, "attending", {".ls1": (0.0, 4.0), ".mix.uq": 5.0, ".mix.dkv": 4.0, ".mix.uk": 8.0, ".mix.uv": 8.0, ".mix.o": 8.0})
    return cases, cases.folder(name, "bfloat16", 7, "attending")


# (requests, tokens each brings) step by step: paddings of 81, 62 and 54 tokens; the second and third behind histories, a lone token among them
STEPS_OF_A_RUN = [([0, 1], [200, 103]), ([0, 1, 2], [100, 1, 221]), ([2, 3, 4, 0], [64, 64, 64, 10])]


@pytest.mark.gpu
@pytest.mark.parametrize("window", [0, 150])
def test_captured_steps(window, monkeypatch):
    """Steps through the runner, padded to their size class and replayed from a graph, whose rows follow from the step's own requests."""
    from vipera_rs_b200.cache import CachePools
    from vipera_rs_b200.engine import ModelRunner, StepInput
    from vipera_rs_b200.engine.loader import load_model
    from vipera_rs_b200.kernels import ops

    cases, path = _folder(monkeypatch, window)
    model = load_model(path, "bfloat16", DEV)
    pools = CachePools(model.cache_requests, page_size=16, num_pages=100, num_state_slots=8, dtype=torch.bfloat16, device=torch.device(DEV))
    runner, taken, real = ModelRunner(model, pools, max_model_len=1024), [], ops.latent_heads
    monkeypatch.setattr(ops, "latent_heads", lambda *args, **named: taken.append(named["rows"].shape[0]) or real(*args, **named))
    rng = np.random.RandomState(11)
    tokens = {request: rng.randint(0, 300, 400).astype(np.int32) for request in range(5)}
    done = dict.fromkeys(tokens, 0)
    for requests, counts in STEPS_OF_A_RUN:
        for request, count in zip(requests, counts):
            if done[request] == 0:
                pools.manager.open(request)
            pools.manager.reserve(request, done[request] + count)
            pools.manager.commit(request, done[request])
        step = StepInput(requests=requests, counts=counts, pos0=[done[r] for r in requests], fresh=[int(done[r] == 0) for r in requests],
                         tokens=np.concatenate([tokens[r][done[r]:done[r] + c] for r, c in zip(requests, counts)]),
                         logit_rows=np.arange(sum(counts), dtype=np.int32))
        before = len(taken)
        got = [runner.run(step).double().cpu() for _ in range(2)]
        assert len(taken) == before + 2 and taken[-1] in (512, 1024, 2048)     # a warm-up and a capture; the second run replays
        assert torch.equal(got[0], got[1])
        ops.check_kernel_status(DEV)
        at = 0
        for request, count in zip(requests, counts):
            want = torch.from_numpy(np.asarray(cases.plain_logits(path, tokens[request][:done[request] + count].tolist())))[done[request]:]
            # bfloat16 operands of seven products in a row, the rows' norms between them
            assert float((got[0][at:at + count] - want).norm() / want.norm()) < 4e-2, (requests, counts, request)
            at += count
            done[request] += count
    assert runner.eager_steps == 0 and len(runner._step_graphs) == len(STEPS_OF_A_RUN)


def test_rows_of_captured_steps():
    """A captured step's rows hold every request's, its padding's too; they are not what a size class leaves room for."""
    from types import SimpleNamespace

    part, _ = _part((3, 512, 0, 16, "interleaved", True), 0, "cpu")
    windowed, _ = _part((3, 512, 1024, 16, "interleaved", True), 0, "cpu")

    def rows(counts, firsts, own=part):
        return own.step_forms(np.array(counts), np.array(firsts)).get(own._form_name(), 0)

    assert rows([64] * 15 + [64], [0] * 16) == 2048             # fifteen prompts of 64 and their padding
    assert rows([500] * 4 + [48], [0] * 5) == 4096
    assert rows([1200, 1, 437, 110, 300], [0, 700, 64, 3000, 0]) == 8192
    assert rows([2048], [0]) == 2048 and rows([1030, 506], [0, 0]) == 2048
    assert rows([512], [7000]) == 8192 and rows([512], [7000], windowed) == 2048
    assert rows([512, 8, 1], [0, 0, 20000]) == 0                # more rows than are planned for
    assert rows([64] + [1] * 10, [0] + [2000] * 10) == 0 and rows([63], [0]) == 0
    # a captured step whose requests nobody named expands all its bound allows: no more rows than it brings tokens
    step = dict(host_counts=[], host_pos0=[], dtype=torch.bfloat16, all_single=False, extras={"graph": True})
    assert part.expanded_rows(SimpleNamespace(num_tokens=1024, num_entries=16, max_kv_len=1024, **step)) == 0
    assert part.expanded_rows(SimpleNamespace(num_tokens=2048, num_entries=1, max_kv_len=2048, **step)) == 2048
    step["extras"] = {"graph": True, "forms": part.step_forms(np.array([1030, 506]), np.array([0, 0]))}
    assert part.expanded_rows(SimpleNamespace(num_tokens=1536, num_entries=2, max_kv_len=4096, **step)) == 2048


def test_plan():
    """The memory plan counts the rows of expanded keys and values for runs that expand them."""
    from vipera_rs_b200.parts.latent import EXPANDED_ROWS, LatentAttention

    sizes = {"num_heads": 32, "kv_rank": 512, "rot_dim": 64, "head_dim": 128, "value_dim": 128}
    bytes_of = lambda element, **other: LatentAttention.workspace_bytes(dict(sizes, **other), 2048, element)  # noqa: E731
    mixed = 2048 * 32 * 128                     # the heads' outputs are in the run's type; the rest is alike
    assert bytes_of(4) - bytes_of(2) == mixed * 2 - EXPANDED_ROWS * (32 * 256 + 512 + 64) * 2
    assert bytes_of(4, rot_dim=32) - bytes_of(2, rot_dim=32) == mixed * 2
