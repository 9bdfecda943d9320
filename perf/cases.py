"""What this engine is measured on: whole steps of the decoder, its single mixers and feed-forwards, the device sampler.

A case is a dict of plain values whose ``kind`` says which entry point runs:

``step``       one step of a small Qwen2 decoder through ``ModelRunner.run``, as ``Engine`` runs it (a replayed graph of the
               step's size class): single tokens behind a history, portions of prompts, both; bfloat16 and the 32-bit path
``latent``     attention over a cached low-rank latent, one layer's mixer (``MIXERS`` "latent_attention")
``lightning``  linear attention with one decay per head ("lightning")
``gla``        gated linear attention ("gla")
``mlstm``      the matrix-memory cell ("mlstm")
``moe``        a mixture of gated units beside a shared one (``FEED_FORWARDS`` "moe_mlp")
``sample``     temperature sampling with top-k, top-p and min-p over a step's logits (``ops.sample``)

``counts`` lists the tokens each request of the step brings and ``history`` how many it has in the cache, as
"700,13" or "64x1" (sixty-four requests of one token).
"""
import math

import numpy as np
import torch

from vipera_rs_b200.cache import CachePools
from vipera_rs_b200.config import architecture_of
from vipera_rs_b200.config.registry import FEED_FORWARDS, MIXERS
from vipera_rs_b200.config.spec import PartSpec
from vipera_rs_b200.engine import ModelRunner, StepInput
from vipera_rs_b200.kernels import ops
from vipera_rs_b200.parts.base import PagedKVView, StateView, StepContext, Workspace
from vipera_rs_b200.parts.model import DecoderModel
from vipera_rs_b200.weights import WeightSource

DEVICE = "cuda"
PAGE = 16            # the engine's default page size
EPS = 1e-6
THETA = 10000.0
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    qwen_1_5b = dict(kind="step", dtype="bfloat16", width=1536, heads=12, kv_heads=2, dim=128, inner=8960, vocab=32000)
    latent = dict(kind="latent", width=1536, heads=12, dim=128, rot=64, vdim=128, rank=512, q_rank=768, window=1024, sink=True,
                  gate=False)
    return [
        # one user's chat: a single token through layers of the 1.5B shape, the smallest call there is
        dict(qwen_1_5b, name="decode_1", layers=2, counts="1", history="500"),
        # a full serving batch on layers of the 7B shape
        dict(qwen_1_5b, name="decode_64_7b", layers=2, width=3584, heads=28, kv_heads=4, inner=18944, counts="64x1", history="64x2048"),
        # a prompt of the benchmark's length
        dict(qwen_1_5b, name="prefill_2048", layers=4, counts="2048", history="0"),
        # the 32-bit path: a small batch, and portions of prompts of odd lengths beside a decoding request (0.5B shape, heads of 64)
        dict(qwen_1_5b, name="fp32_decode_8", dtype="float32", layers=2, counts="8x1", history="8x1000"),
        dict(qwen_1_5b, name="fp32_portions", dtype="float32", layers=2, width=896, heads=14, dim=64, inner=4864,
             counts="700,1,323", history="0,900,40"),
        # attention over latents: a prompt with a window, sinks and a query latent; portions behind histories, many heads, a gate
        dict(latent, name="latent_2048", counts="2048", history="0"),
        dict(latent, name="latent_portions", width=4096, heads=32, q_rank=0, window=0, sink=False, gate=True,
             counts="1200,1,437,110", history="0,700,64,3000"),
        # the recurrences over a prompt and over several requests' portions
        dict(kind="lightning", name="lightning_2048", width=1536, heads=6, dim=128, vdim=256, counts="2048", history="0"),
        dict(kind="gla", name="gla_portions", width=4096, heads=8, dim=128, vdim=256, counts="1024,901,77", history="0,33,0"),
        dict(kind="mlstm", name="mlstm_2048", width=4096, heads=8, dim=256, vdim=512, counts="2048", history="0"),
        # a mixture of experts over a prompt
        dict(kind="moe", name="moe_2048", width=1536, inner=1792, experts=16, top=4, shared=1792, counts="2048", history="0"),
        # the draw behind a decode step of 64 requests over the vocabulary of the 1.5B shape
        dict(kind="sample", name="sample_64", rows=64, vocab=151936),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _ragged(rng, most_tokens):
    """Counts and histories of a step with portions: one to five requests, some of a single token."""
    left, counts, history = most_tokens, [], []
    for index in range(rng.choice([1, 1, 2, 3, 5])):
        count = 1 if index and rng.random() < 0.3 else min(left, _log_int(rng, 17, most_tokens))
        if count <= 0:
            break
        counts.append(count)
        history.append(_log_int(rng, 1, 3000) if count == 1 or rng.random() < 0.4 else 0)
        left -= count
    return ",".join(map(str, counts)), ",".join(map(str, history))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "fp32", "fp32", "latent", "latent", "lightning", "gla", "mlstm", "moe", "sample"])
    if kind in ("decode", "prefill", "fp32"):
        width, heads, kv_heads, dim, inner = rng.choice([(896, 14, 2, 64, 4864), (1536, 12, 2, 128, 8960), (2048, 16, 2, 128, 5632)])
        case = dict(kind="step", dtype="float32" if kind == "fp32" else "bfloat16", layers=rng.choice([1, 2]), width=width,
                    heads=heads, kv_heads=kv_heads, dim=dim, inner=inner, vocab=rng.choice([8000, 32000]))
        if kind == "decode" or (kind == "fp32" and rng.random() < 0.5):
            batch = _log_int(rng, 1, 64 if kind == "decode" else 32)
            case.update(counts="%dx1" % batch, history="%dx%d" % (batch, _log_int(rng, 5, 3000)))
        else:
            counts, history = _ragged(rng, 2048 if kind == "prefill" else 800)
            case.update(counts=counts, history=history)
        return case
    if kind == "sample":
        return dict(kind="sample", rows=_log_int(rng, 1, 64), vocab=rng.choice([32000, 50257, 128256, 151936]))
    counts, history = _ragged(rng, 2048)
    if kind == "latent":
        own = rng.random() < 0.5
        return dict(kind="latent", width=rng.choice([1024, 1536, 2048]), heads=rng.choice([8, 12, 16, 20]), dim=128, rot=64,
                    vdim=128, rank=rng.choice([256, 512, 512]), q_rank=768 if own else 0, window=rng.choice([0, 0, 512, 1024]),
                    sink=own, gate=not own, counts=counts, history=history)
    if kind == "moe":
        return dict(kind="moe", width=rng.choice([1024, 1536, 2048]), inner=rng.choice([704, 1792, 2240]), experts=16,
                    top=rng.choice([2, 4]), shared=rng.choice([0, 1792]), counts=counts, history=history)
    dim, vdim = rng.choice([(128, 256), (64, 128), (256, 256)] if kind != "mlstm" else [(128, 256), (256, 512), (64, 128)])
    return dict(kind=kind, width=rng.choice([1024, 1536, 2048]), heads=rng.choice([4, 6, 8]), dim=dim, vdim=vdim, counts=counts,
                history=history if kind != "mlstm" else ",".join("0" for _ in counts.split(",")))


def _list(text):
    out = []
    for item in text.split(","):
        times, _, value = item.rpartition("x")
        out.extend([int(value)] * (int(times) if times else 1))
    return out


# ---------------------------------------------------------------------------------------
# weights and inputs, from the seed alone
# ---------------------------------------------------------------------------------------
class _Numbers:
    """Named random tensors: the same for prepare() and exact()."""

    def __init__(self, seed):
        self.seed = int(seed)

    def normal(self, name, shape, std=1.0, mean=0.0, dtype=torch.float32):
        number = self.seed * 1000003
        for letter in name:
            number = (number * 131 + ord(letter)) % (1 << 62)
        generator = torch.Generator(device=DEVICE)
        generator.manual_seed(number)
        return torch.randn(shape, generator=generator, device=DEVICE).mul_(std).add_(mean).to(dtype)


def _weights(case, seed):
    """The tensors of a case's model or part by name, in the types a model folder stores them in."""
    numbers, kind = _Numbers(seed), case["kind"]
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    w, width = {}, case["width"]

    def matrix(name, *shape, std=0.02):
        w[name] = numbers.normal(name, shape, std, dtype=dtype)

    def gain(name, size):
        w[name] = numbers.normal(name, (size,), 0.01, 1.0)

    heads, dim = case.get("heads"), case.get("dim")
    if kind == "step":
        matrix("model.embed_tokens.weight", case["vocab"], width, std=0.05)
        for layer in range(case["layers"]):
            at = "model.layers.%d." % layer
            gain(at + "input_layernorm.weight", width)
            gain(at + "post_attention_layernorm.weight", width)
            for name, rows in (("q", heads * dim), ("k", case["kv_heads"] * dim), ("v", case["kv_heads"] * dim)):
                matrix(at + "self_attn.%s_proj.weight" % name, rows, width)
                matrix(at + "self_attn.%s_proj.bias" % name, rows)
            matrix(at + "self_attn.o_proj.weight", width, heads * dim)
            matrix(at + "mlp.gate_proj.weight", case["inner"], width)
            matrix(at + "mlp.up_proj.weight", case["inner"], width)
            matrix(at + "mlp.down_proj.weight", width, case["inner"])
        gain("model.norm.weight", width)
        return w
    if kind == "moe":
        w["p.router.weight"] = numbers.normal("router", (case["experts"], width), 0.02)
        units = [("e%d" % k, case["inner"]) for k in range(case["experts"])]
        for unit, size in units + ([("shared", case["shared"])] if case["shared"] else []):
            matrix("p.%s.gate.weight" % unit, size, width)
            matrix("p.%s.up.weight" % unit, size, width)
            matrix("p.%s.down.weight" % unit, width, size)
        return w
    vdim = case["vdim"]
    if kind == "latent":
        rank, rot = case["rank"], case["rot"]
        if case["q_rank"]:
            matrix("p.dq.weight", case["q_rank"], width)
            gain("p.dq.norm.weight", case["q_rank"])
        matrix("p.uq.weight" if case["q_rank"] else "p.q.weight", heads * (dim + rot), case["q_rank"] or width, std=0.03)
        if case["sink"]:
            w["p.sink.weight"] = numbers.normal("sink", (heads,), 1.5)
        matrix("p.uk.weight", heads * dim, rank, std=0.04)
        matrix("p.uv.weight", heads * vdim, rank, std=0.04)
        matrix("p.o.weight", width, heads * vdim)
        matrix("p.dkv.weight", rank + rot, width)
        gain("p.dkv.norm.weight", rank)
        if case["gate"]:
            matrix("p.g.weight", heads * vdim, width)
        return w
    for name, rows in (("q", heads * dim), ("k", heads * dim), ("v", heads * vdim), ("g", heads * vdim)):
        matrix("p.%s.weight" % name, rows, width)
    matrix("p.o.weight", width, heads * vdim)
    gain("p.norm.weight", vdim if kind == "gla" else heads * vdim)
    if kind == "gla":
        matrix("p.a1.weight", 16, width)
        matrix("p.a2.weight", heads * dim, 16, std=0.3)
        matrix("p.a2.bias", heads * dim)
    if kind == "mlstm":
        for name in ("i", "f"):
            matrix("p.%s.weight" % name, heads, width)
            w["p.%s.bias" % name] = numbers.normal(name + "bias", (heads,), 0.5, 3.0 if name == "f" else 0.0, dtype=dtype)
    return w


def _decays(case):
    """The linear attention's decays: from 1 - 2^-5 for the first head to 1 - 2^-10 for the last."""
    return [1.0 - 2.0 ** (-5.0 - 5.0 * index / max(case["heads"] - 1, 1)) for index in range(case["heads"])]


def _inputs(case, seed):
    """(normed rows [tokens, width] in bfloat16, per request what its cache holds)."""
    numbers = _Numbers(seed)
    counts, history = _list(case["counts"]), _list(case["history"])
    rows = numbers.normal("rows", (sum(counts), case["width"]), dtype=torch.bfloat16)
    kept = None
    if case["kind"] == "latent":
        kept = [(numbers.normal("c%d" % e, (n, case["rank"]), dtype=torch.bfloat16),
                 numbers.normal("r%d" % e, (n, case["rot"]), dtype=torch.bfloat16)) for e, n in enumerate(history)]
    elif case["kind"] in ("lightning", "gla"):
        kept = [numbers.normal("s%d" % e, (case["heads"], case["dim"], case["vdim"]), 0.5 if n else 0.0) for e, n in enumerate(history)]
    return rows, kept


def _tokens(case, seed):
    return np.random.RandomState(seed % (1 << 31)).randint(0, case["vocab"], sum(_list(case["counts"]))).astype(np.int32)


def _past(case, seed, layer, entry, length):
    """Keys and values of a request's earlier tokens in one layer, [length, kv_heads, dim] each."""
    shape = (length, case["kv_heads"], case["dim"])
    numbers, dtype = _Numbers(seed), DTYPES[case["dtype"]]
    return (numbers.normal("k%d.%d" % (layer, entry), shape, 0.5, dtype=dtype),
            numbers.normal("v%d.%d" % (layer, entry), shape, 0.5, dtype=dtype))


# ---------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------
class _Given(WeightSource):
    def __init__(self, tensors):
        self.tensors = tensors

    def names(self):
        return list(self.tensors)

    def shape(self, name):
        return tuple(self.tensors[name].shape)

    def get(self, name):
        return self.tensors[name]


def _prepare_step(case, seed):
    counts, history = _list(case["counts"]), _list(case["history"])
    dtype = DTYPES[case["dtype"]]
    config = {"architectures": ["Qwen2ForCausalLM"], "num_hidden_layers": case["layers"], "hidden_size": case["width"],
              "num_attention_heads": case["heads"], "num_key_value_heads": case["kv_heads"], "head_dim": case["dim"],
              "intermediate_size": case["inner"], "vocab_size": case["vocab"], "rope_theta": THETA, "rms_norm_eps": EPS,
              "tie_word_embeddings": True, "max_position_embeddings": 8192}
    arch = architecture_of(config)
    model = DecoderModel(arch.model_spec(arch.config_from_dict(config)), _Given(_weights(case, seed)), dtype, DEVICE)
    pages = sum(-(-(c + h) // PAGE) for c, h in zip(counts, history)) + 1
    pools = CachePools(model.cache_requests, page_size=PAGE, num_pages=pages, num_state_slots=len(counts), dtype=dtype, device=DEVICE)
    runner = ModelRunner(model, pools, max_model_len=8192)
    manager = pools.manager
    for entry, (count, length) in enumerate(zip(counts, history)):
        manager.open(entry)
        manager.reserve(entry, count + length)
        manager.commit(entry, length)
    for entry, length in enumerate(history):
        if length:
            table = torch.from_numpy(manager.tables([entry], 0, -(-(length + counts[entry]) // PAGE))[0].astype(np.int64)).to(DEVICE)
            position = torch.arange(length, device=DEVICE)
            place = table[position // PAGE] * PAGE + position % PAGE
            for layer in range(case["layers"]):
                k, v = _past(case, seed, layer, entry, length)
                view = pools.views[layer]
                view.k.view(-1, case["kv_heads"], case["dim"])[place] = k
                view.v.view(-1, case["kv_heads"], case["dim"])[place] = v
    step = StepInput(requests=list(range(len(counts))), tokens=_tokens(case, seed), counts=counts, pos0=history,
                     fresh=[int(h == 0) for h in history], logit_rows=np.cumsum(counts).astype(np.int32) - 1)
    # what a step leaves: the logits and the keys and values in the pages (the spare page behind them is nobody's)
    kept = [half[:-1] for layer in range(case["layers"]) for half in (pools.views[layer].k, pools.views[layer].v)]
    return {"runner": runner, "step": step, "kept": kept}


def _rotation(case):
    return PartSpec("rope_interleaved", {"head_dim": case["rot"], "rotary_dims": case["rot"], "theta": THETA, "scaling": None,
                                         "exact_angles": True, "max_positions": 8192})


def _prepare_part(case, seed):
    kind, width = case["kind"], case["width"]
    counts, history = _list(case["counts"]), _list(case["history"])
    rows, kept = _inputs(case, seed)
    if kind == "moe":
        params = {"hidden_size": width, "intermediate_size": case["inner"], "experts": case["experts"], "top": case["top"],
                  "score": "softmax", "renormalize": True, "activation": "silu"}
        if case["shared"]:
            params["shared_size"] = case["shared"]
    else:
        params = {"hidden_size": width, "num_heads": case["heads"], "head_dim": case["dim"], "value_dim": case["vdim"], "norm_eps": EPS}
    if kind == "latent":
        params.update(rot_dim=case["rot"], kv_rank=case["rank"], softmax_scale=(case["dim"] + case["rot"]) ** -0.5,
                      position=_rotation(case), output_gate=case["gate"])
        if case["q_rank"]:
            params["q_rank"] = case["q_rank"]
        if case["window"]:
            params["window"] = case["window"]
        if case["sink"]:
            params["sink"] = "learned"
    elif kind == "lightning":
        params["decay"] = _decays(case)
    elif kind == "gla":
        params.update(tau=16.0, decay_rank=16)
    elif kind == "mlstm":
        params["gate_cap"] = 15.0
    registry, name = (FEED_FORWARDS, "moe_mlp") if kind == "moe" else (MIXERS, "latent_attention" if kind == "latent" else kind)
    part = registry.find(name)(params, "p", _weights(case, seed), torch.bfloat16, DEVICE)
    getattr(part, "prepare", lambda reach: None)(8192)

    entries, total = len(counts), sum(counts)
    starts = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    positions = np.concatenate([np.arange(h, h + c) for c, h in zip(counts, history)]).astype(np.int32)
    longest = max(c + h for c, h in zip(counts, history))
    pages = [-(-(c + h) // PAGE) for c, h in zip(counts, history)]
    table = np.full((entries, -(-longest // PAGE)), -1, dtype=np.int32)
    for entry, own in enumerate(pages):
        table[entry, :own] = sum(pages[:entry]) + np.arange(own)

    def device(values):
        return torch.from_numpy(np.ascontiguousarray(values, dtype=np.int32)).to(DEVICE)

    cache, outputs = None, []
    if kind == "latent":
        k = torch.zeros(sum(pages), PAGE, 1, case["rank"], dtype=torch.bfloat16, device=DEVICE)
        v = torch.zeros(sum(pages), PAGE, 1, case["rot"], dtype=torch.bfloat16, device=DEVICE)
        for entry, (c, r) in enumerate(kept):
            at = sum(pages[:entry]) * PAGE
            k.view(-1, case["rank"])[at:at + len(c)] = c
            v.view(-1, case["rot"])[at:at + len(r)] = r
        cache, outputs = PagedKVView(0, k, v, PAGE, case["window"] or None), [k, v]
    elif kind != "moe":
        request = part.cache_request()
        data = torch.zeros(entries + 1, *request.shape, dtype=request.dtype, device=DEVICE)
        if kept is not None:
            for entry, state in enumerate(kept):
                data[entry] = state.reshape(-1)
        cache, outputs = StateView(data), [data[:entries]]
    tokens = device(np.zeros(total))
    context = StepContext(
        num_tokens=total, num_entries=entries, tokens=tokens, positions=device(positions),
        token_entry=device(np.repeat(np.arange(entries), counts)), entry_starts=device(starts), entry_pos0=device(history),
        state_slots=device(np.arange(entries)), fresh=device([int(h == 0) for h in history]), block_tables=[device(table)],
        logit_rows=None, num_logit_rows=0, host_counts=counts, host_pos0=history, max_count=max(counts), max_kv_len=longest,
        all_single=max(counts) == 1, any_single=1 in counts, dtype=torch.bfloat16, workspace=Workspace(DEVICE))
    stream = torch.zeros(total, width, device=DEVICE)
    return {"part": part, "context": context, "rows": rows, "stream": stream, "cache": cache, "outputs": outputs}


def _sample_settings(case, seed):
    rows = case["rows"]
    turn = np.arange(rows) % 4
    # by turns: top-k 50 and top-p 0.95; top-p 0.9 alone; a cooler draw with top-p and min-p; greedy
    return {"temperature": np.choose(turn, [0.8, 1.0, 0.7, 0.0]).astype(np.float32),
            "top_k": np.choose(turn, [50, 0, 0, 0]).astype(np.int32),
            "top_p": np.choose(turn, [0.95, 0.9, 0.9, 1.0]).astype(np.float32),
            "min_p": np.choose(turn, [0.0, 0.0, 0.05, 0.0]).astype(np.float32),
            "uniform": np.random.RandomState(seed % (1 << 31)).random_sample(rows)}


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    if case["kind"] != "sample":
        return _prepare_part(case, seed)
    state = {name: torch.from_numpy(values).to(DEVICE) for name, values in _sample_settings(case, seed).items()}
    # logits as peaked as a trained model's: the likeliest ten hold about half of the mass
    state["logits"] = _Numbers(seed).normal("logits", (case["rows"], case["vocab"]), 4.0)
    state["tokens"] = torch.zeros(case["rows"], dtype=torch.int32, device=DEVICE)
    state["status"] = torch.zeros(case["rows"], dtype=torch.int32, device=DEVICE)
    return state


def run(state):
    if "runner" in state:
        return {"logits": state["runner"].run(state["step"]), "kept": state["kept"]}
    if "logits" in state:
        ops.sample(**state)
        return {"tokens": state["tokens"], "status": state["status"]}
    part, context, stream = state["part"], state["context"], state["stream"]
    if state["cache"] is None:
        part.forward(context, state["rows"], stream)
    else:
        part.forward(context, state["rows"], stream, state["cache"], True)
    return {"stream": stream, "kept": state["outputs"]}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _pairs(counts, history, window=0):
    """(query, key) pairs a causal mask leaves, all requests together."""
    total = 0
    for count, length in zip(counts, history):
        seen = np.arange(length + 1, length + count + 1)
        total += int(np.minimum(seen, window).sum() if window else seen.sum())
    return total


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 2.0 * case["rows"] * case["vocab"]}
    counts, history = _list(case["counts"]), _list(case["history"])
    tokens, width = sum(counts), case["width"]
    size = 4 if case.get("dtype") == "float32" else 2
    if kind == "step":
        q, kv, inner = case["heads"] * case["dim"], case["kv_heads"] * case["dim"], case["inner"]
        layer = width * (2 * q + 2 * kv) + 3 * width * inner
        seen = sum(c + h for c, h in zip(counts, history))
        flops = case["layers"] * (2.0 * tokens * layer + 4.0 * _pairs(counts, history) * q) + 2.0 * len(counts) * width * case["vocab"]
        held = case["layers"] * (layer * size + 2 * seen * kv * size) + case["vocab"] * width * size
        return {"bytes": float(held + tokens * width * size + len(counts) * case["vocab"] * 4), "flops": flops}
    stream = tokens * width * (2 + 8)          # the normed rows in, the stream in and out
    if kind == "moe":
        matrices = 3.0 * width * (case["experts"] * case["inner"] + case["shared"])
        if tokens * case["top"] < case["experts"]:
            matrices = 3.0 * width * (tokens * case["top"] * case["inner"] + case["shared"])
        return {"bytes": matrices * 2 + stream, "flops": 2.0 * tokens * (3.0 * width * (case["top"] * case["inner"] + case["shared"]))}
    heads, dim, vdim = case["heads"], case["dim"], case["vdim"]
    if kind == "latent":
        rank, rot, q_rank = case["rank"], case["rot"], case["q_rank"]
        window = case["window"]
        projections = (width * q_rank + q_rank * heads * (dim + rot)) if q_rank else width * heads * (dim + rot)
        projections += width * (rank + rot) + width * heads * vdim * (2 if case["gate"] else 1) + heads * (dim + vdim) * rank
        seen = sum(c + (min(h, window) if window else h) for c, h in zip(counts, history))
        # the fewest operations: keys and values of every head expanded once, then plain attention
        pairs = _pairs(counts, history, window)
        expand = heads * (dim + vdim) * rank * (seen - tokens)
        flops = 2.0 * tokens * projections + 2.0 * expand + 2.0 * pairs * heads * (dim + rot + vdim)
        return {"bytes": projections * 2.0 + 2.0 * seen * (rank + rot) + stream, "flops": flops}
    projections = width * heads * (2 * dim + 3 * vdim)
    if kind == "gla":
        projections += 16 * (width + heads * dim)
    if kind == "mlstm":
        projections += 2 * heads * width
    state = 2.0 * 4 * len(counts) * heads * dim * vdim
    return {"bytes": projections * 2.0 + state + stream, "flops": 2.0 * tokens * projections + 4.0 * tokens * heads * dim * vdim}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"      # drawn ids
    if case.get("dtype") == "float32":
        return {"rel": 2e-5}
    return {"rel": 2e-2}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, plainly
# ---------------------------------------------------------------------------------------
def _norm(x, weight):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * weight


def _spans(counts):
    at = 0
    for entry, count in enumerate(counts):
        yield entry, at, at + count
        at += count


def _exact_step(case, seed):
    w = {name: tensor.double() for name, tensor in _weights(case, seed).items()}
    counts, history = _list(case["counts"]), _list(case["history"])
    heads, kv_heads, dim = case["heads"], case["kv_heads"], case["dim"]
    x = w["model.embed_tokens.weight"][torch.from_numpy(_tokens(case, seed).astype(np.int64)).to(DEVICE)]
    position = torch.cat([torch.arange(h, h + c) for c, h in zip(counts, history)])
    # the angles are formed in 32 bits by definition
    inverse = 1.0 / torch.pow(torch.tensor(THETA), 2.0 * torch.arange(dim // 2, dtype=torch.float32) / float(dim))
    angle = position.float()[:, None] * inverse[None, :]
    cos, sin = torch.cos(angle).double().to(DEVICE)[:, None], torch.sin(angle).double().to(DEVICE)[:, None]

    def turn(z):
        a, b = z[..., :dim // 2], z[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

    for layer in range(case["layers"]):
        at = "model.layers.%d." % layer
        h = _norm(x, w[at + "input_layernorm.weight"])
        q, k, v = (h @ w[at + "self_attn.%s_proj.weight" % n].T + w[at + "self_attn.%s_proj.bias" % n] for n in "qkv")
        q, k, v = turn(q.view(-1, heads, dim)), turn(k.view(-1, kv_heads, dim)), v.view(-1, kv_heads, dim)
        mixed = torch.empty_like(q)
        for entry, begin, end in _spans(counts):
            past_k, past_v = _past(case, seed, layer, entry, history[entry])
            keys, values = torch.cat([past_k.double(), k[begin:end]]), torch.cat([past_v.double(), v[begin:end]])
            hidden = torch.arange(len(keys), device=DEVICE)[None, :] > torch.arange(history[entry], len(keys), device=DEVICE)[:, None]
            for head in range(heads):
                group = head // (heads // kv_heads)
                score = (q[begin:end, head] @ keys[:, group].T / math.sqrt(dim)).masked_fill_(hidden, -math.inf)
                mixed[begin:end, head] = torch.softmax(score, -1) @ values[:, group]
        x = x + mixed.reshape(len(x), -1) @ w[at + "self_attn.o_proj.weight"].T
        h = _norm(x, w[at + "post_attention_layernorm.weight"])
        gate = h @ w[at + "mlp.gate_proj.weight"].T
        x = x + (torch.nn.functional.silu(gate) * (h @ w[at + "mlp.up_proj.weight"].T)) @ w[at + "mlp.down_proj.weight"].T
    last = torch.tensor([end - 1 for _, _, end in _spans(counts)], device=DEVICE)
    logits = _norm(x[last], w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T
    return {"logits": logits, "kept": [None] * (2 * case["layers"])}   # the pages follow from the layers before and are not repeated


def _exact_latent(case, w, h, kept):
    counts, history = _list(case["counts"]), _list(case["history"])
    heads, dim, rot, rank, vdim = (case[n] for n in ("heads", "dim", "rot", "rank", "vdim"))
    frequency = THETA ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
    position = torch.cat([torch.arange(a, a + c) for c, a in zip(counts, history)])
    angle = position.double()[:, None] * frequency[None, :]
    # cosines and sines are rounded to 32 bits by definition
    cos, sin = torch.cos(angle).float().double().to(DEVICE), torch.sin(angle).float().double().to(DEVICE)

    def turn(z, c, s):
        a, b = z[..., 0::2], z[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)

    if case["q_rank"]:
        q = _norm(h @ w["p.dq.weight"].T, w["p.dq.norm.weight"]) @ w["p.uq.weight"].T
    else:
        q = h @ w["p.q.weight"].T
    q = q.view(-1, heads, dim + rot)
    q_turned = turn(q[..., dim:], cos[:, None], sin[:, None])
    down = h @ w["p.dkv.weight"].T
    latent, key_part = _norm(down[:, :rank], w["p.dkv.norm.weight"]), turn(down[:, rank:], cos, sin)
    up_k, up_v = w["p.uk.weight"].view(heads, dim, rank), w["p.uv.weight"].view(heads, vdim, rank)
    out = torch.empty(len(h), heads, vdim, dtype=torch.float64, device=DEVICE)
    for entry, begin, end in _spans(counts):
        c = torch.cat([kept[entry][0].double(), latent[begin:end]])
        r = torch.cat([kept[entry][1].double(), key_part[begin:end]])
        key, query = torch.arange(len(c), device=DEVICE)[None, :], torch.arange(history[entry], len(c), device=DEVICE)[:, None]
        hidden = key > query
        if case["window"]:
            hidden |= key <= query - case["window"]
        for head in range(heads):
            score = q[begin:end, head, :dim] @ (c @ up_k[head].T).T + q_turned[begin:end, head] @ r.T
            score = (score * (dim + rot) ** -0.5).masked_fill_(hidden, -math.inf)
            if case["sink"]:
                score = torch.cat([score, w["p.sink.weight"][head].expand(end - begin, 1)], dim=1)
            out[begin:end, head] = torch.softmax(score, -1)[:, :len(c)] @ (c @ up_v[head].T)
    out = out.reshape(len(h), -1)
    if case["gate"]:
        out = out * torch.sigmoid(h @ w["p.g.weight"].T)
    return out @ w["p.o.weight"].T, [None, None]


def _exact_recurrence(case, w, h, kept):
    kind, counts = case["kind"], _list(case["counts"])
    heads, dim, vdim = case["heads"], case["dim"], case["vdim"]
    q, k, v, g = (h @ w["p.%s.weight" % n].T for n in "qkvg")
    q, k, v, g = q.view(-1, heads, dim), k.view(-1, heads, dim), v.view(-1, heads, vdim), g.view(-1, heads, vdim)
    states, out = [], torch.empty_like(v)
    if kind == "lightning":
        q, k, v = (torch.nn.functional.silu(z) for z in (q, k, v))
        decay = torch.tensor(_decays(case), dtype=torch.float64, device=DEVICE).float().double().view(1, heads, 1, 1).expand(len(h), -1, -1, -1)
    elif kind == "gla":
        z = (h @ w["p.a1.weight"].T) @ w["p.a2.weight"].T + w["p.a2.bias"]
        decay = torch.exp(torch.nn.functional.logsigmoid(z) / 16.0).view(-1, heads, dim, 1)
        q = q * dim ** -0.5
    else:
        li, lf = (15.0 * torch.tanh((h @ w["p.%s.weight" % n].T + w["p.%s.bias" % n]) / 15.0) for n in "if")
        lf, q = torch.nn.functional.logsigmoid(lf), q * dim ** -0.5
    for entry, begin, end in _spans(counts):
        if kind != "mlstm":
            s = kept[entry].double()
            for t in range(begin, end):
                s = decay[t] * s + k[t][:, :, None] * v[t][:, None, :]
                out[t] = (q[t][:, None, :] @ s)[:, 0]
            states.append(s.reshape(-1))
            continue
        s = torch.zeros(heads, dim, vdim, dtype=torch.float64, device=DEVICE)
        n = torch.zeros(heads, dim, dtype=torch.float64, device=DEVICE)
        m = torch.zeros(heads, dtype=torch.float64, device=DEVICE)
        for t in range(begin, end):
            top = torch.maximum(lf[t] + m, li[t])
            old, new = torch.exp(lf[t] + m - top), torch.exp(li[t] - top)
            s = old[:, None, None] * s + new[:, None, None] * (k[t][:, :, None] * v[t][:, None, :])
            n, m = old[:, None] * n + new[:, None] * k[t], top
            below = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            out[t] = (q[t][:, None, :] @ s)[:, 0] / below[:, None]
    if kind == "lightning":
        mixed = _norm(out.reshape(len(h), -1), w["p.norm.weight"]) * torch.sigmoid(g.reshape(len(h), -1))
    elif kind == "gla":
        mixed = (_norm(out, w["p.norm.weight"]) * torch.nn.functional.silu(g)).reshape(len(h), -1)
    else:
        each = out / torch.sqrt((out * out).mean(-1, keepdim=True) + EPS)
        mixed = each.reshape(len(h), -1) * w["p.norm.weight"] * torch.sigmoid(g.reshape(len(h), -1))
    # (the cell's state is kept in a layout of its own: no 64-bit value beside it)
    return mixed @ w["p.o.weight"].T, [torch.stack(states) if states else None]


def _exact_moe(case, w, h):
    score = torch.softmax(h @ w["p.router.weight"].T, -1)
    weight, chosen = score.topk(case["top"], dim=-1)
    weight = weight / weight.sum(-1, keepdim=True)

    def unit(name, rows):
        inner = torch.nn.functional.silu(rows @ w["p.%s.gate.weight" % name].T) * (rows @ w["p.%s.up.weight" % name].T)
        return inner @ w["p.%s.down.weight" % name].T

    out = unit("shared", h) if case["shared"] else torch.zeros_like(h)
    for expert in range(case["experts"]):
        row, place = torch.nonzero(chosen == expert, as_tuple=True)
        out[row] += weight[row, place, None] * unit("e%d" % expert, h[row])
    return out


def _exact_sample(case, seed):
    settings = _sample_settings(case, seed)
    logits = _Numbers(seed).normal("logits", (case["rows"], case["vocab"]), 4.0).double()
    tokens = []
    for row in range(case["rows"]):
        values, ids = logits[row].sort(descending=True, stable=True)
        if settings["temperature"][row] == 0:
            tokens.append(int(ids[0]))
            continue
        weight = torch.exp((values - values[0]) / float(settings["temperature"][row]))
        kept = weight[:int(settings["top_k"][row]) or None]
        below = torch.nonzero(kept.cumsum(0) >= float(settings["top_p"][row]) * weight.sum())
        kept = kept[:int(below[0]) + 1] if len(below) else kept
        kept = torch.where(kept >= float(settings["min_p"][row]) * weight[0], kept, 0.0)
        running = kept.cumsum(0)
        tokens.append(int(ids[int(torch.searchsorted(running, settings["uniform"][row] * running[-1:], right=True))]))
    return {"tokens": np.asarray(tokens, dtype=np.int32), "status": np.zeros(case["rows"], dtype=np.int32)}


def exact(case, seed):
    if case["kind"] == "sample":
        return _exact_sample(case, seed)
    if case["kind"] == "step":
        return _exact_step(case, seed)
    w = {name: tensor.double() for name, tensor in _weights(case, seed).items()}
    rows, kept = _inputs(case, seed)
    if case["kind"] == "moe":
        return {"stream": _exact_moe(case, w, rows.double()), "kept": []}
    stream, states = (_exact_latent if case["kind"] == "latent" else _exact_recurrence)(case, w, rows.double(), kept)
    return {"stream": stream, "kept": states}
