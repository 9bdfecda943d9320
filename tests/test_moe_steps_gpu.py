"""Steps of many tokens through the mixture of units: four tokens share a block of the router, the assignments are
grouped in batches of a block's threads, and the output may be added to the stream at once.  The oracle is the same
tokens in steps small enough that a block takes one of them; a token's sums run in one order in both."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ops():
    from vipera_rs_b200.kernels import ops

    return ops


def _run(ops, h, router, up, down, top, identity, always, always_gate, dtype, target=None):
    tokens, hidden = h.shape
    matrices, ff = down.shape[0], down.shape[2]
    slots, capacity = top + always, ops.moe_capacity(tokens, top + always, matrices)
    chosen = torch.full((tokens, slots), -7, dtype=torch.int32, device=DEV)
    weight = torch.full((tokens, slots), float("nan"), device=DEV)
    rows = torch.full((tokens, slots * hidden), float("nan"), device=DEV)
    ops.moe(h, router=router, gate_up=up, down=down, gate_group=16, top=top, groups=2, keep=1, group_top=2, softmax_scores=True,
            renormalize=True, activation=ops.ACT_SILU, chosen=chosen, weight=weight,
            scratch=torch.zeros(ops.moe_scratch_words(tokens, slots, matrices), dtype=torch.int32, device=DEV),
            act=torch.full((capacity, ff), float("nan"), dtype=dtype, device=DEV), rows=rows,
            xs=torch.full((capacity, hidden), float("nan"), dtype=dtype, device=DEV),
            ys=torch.full((capacity, hidden), float("nan"), device=DEV), identity=identity, always=always, route_scale=1.5,
            always_gate=always_gate, target=target)
    return chosen, weight, rows.view(tokens, slots, hidden)


# the least tokens that share a block, a last block that is not full, more assignments than one batch of a thread's;
# rows that end within a vector's batch; identity outputs and a gate of the always-used unit
@pytest.mark.parametrize("tokens,hidden,ff,outputs,identity,always,gate,top", [
    (592, 64, 32, 6, 0, 0, False, 2), (595, 136, 48, 8, 2, 1, True, 3), (2050, 264, 32, 12, 0, 1, False, 5), (601, 72, 24, 6, 2, 0, False, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_many_tokens_like_few(tokens, hidden, ff, outputs, identity, always, gate, top, dtype):
    ops = _ops()
    torch.manual_seed(tokens + hidden)
    matrices = outputs - identity + always
    h = torch.randn(tokens, hidden, device=DEV).to(dtype)
    router = torch.randn(outputs + int(gate), hidden, device=DEV) * 0.3
    up = (torch.randn(matrices, 2 * ff, hidden, device=DEV) * 0.2).to(dtype)
    down = (torch.randn(matrices, hidden, ff, device=DEV) * 0.2).to(dtype)
    if ff % 16:
        up = up[:, :2 * (ff // 16 * 16)].contiguous()
        down = down[:, :, :ff // 16 * 16].contiguous()
    arguments = (router, up, down, top, identity, always, gate, dtype)
    chosen, weight, rows = _run(ops, h, *arguments)
    parts = [_run(ops, h[i:i + 500], *arguments) for i in range(0, tokens, 500)]
    for whole, few in zip((chosen, weight, rows), zip(*parts)):
        assert torch.equal(whole, torch.cat(few))
    stream = torch.randn(tokens, hidden, device=DEV)
    want = rows[:, 0].clone()
    for place in range(1, rows.shape[1]):
        want += rows[:, place]
    want = stream + want
    _run(ops, h, *arguments, target=stream)
    assert torch.equal(stream, want)
