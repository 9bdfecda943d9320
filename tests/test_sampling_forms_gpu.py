"""The device sampler's cluster form at the sizes where it can go wrong: rows of one value, rows that end within a run
of 1,024, rows too long to be kept, ties that are cut by id, rows the host has to draw.  Held to the host sampler."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("vocab", [1, 3, 64, 1023, 1025, 5003, 32000, 151936, 420001])
def test_draws_are_the_host_samplers(vocab):
    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.sampling import draw_temperature

    torch.manual_seed(vocab)
    logits = torch.randn(9, vocab) * 4
    logits[1] = 0.25                                   # all equal: the lowest ids are kept
    logits[2] = torch.randint(-3, 3, (vocab,)).float()  # few values, many ties at any bound
    logits[3, ::2], logits[3, 1::2] = 0.0, -1000.0
    logits[4, vocab // 2 + 1:] = float("-inf")
    logits[5] = float("nan")
    configs = [(1.0, 50, 0.95, 0.0), (0.7, 0, 0.9, 0.05), (2.5, 4096, 1.0, 0.0), (1.0, 0, 1.0, 0.0), (0.0, 7, 0.5, 0.1), (1.3, 5000, 0.9, 0.0)]
    uniform = torch.rand(9, dtype=torch.float64)
    for temperature, top_k, top_p, min_p in configs:
        tokens = torch.full((9,), -7, dtype=torch.int32, device=DEV)
        status = torch.full((9,), -7, dtype=torch.int32, device=DEV)
        full = lambda value, dtype=torch.float32: torch.full((9,), value, dtype=dtype, device=DEV)  # noqa: E731
        ops.sample(logits.to(DEV), temperature=full(temperature), top_k=full(top_k, torch.int32), top_p=full(top_p), min_p=full(min_p),
                   uniform=uniform.to(DEV), tokens=tokens, status=status)
        for row in range(9):
            if row == 5:
                assert int(status[row]) == ops.SAMPLE_NO_FINITE
                continue
            if top_k > ops.SAMPLER_MAX_TOP_K and temperature:
                assert int(status[row]) == ops.SAMPLE_NEEDS_HOST
                continue
            if int(status[row]) == ops.SAMPLE_NEEDS_HOST:
                # only where nothing cuts the row to a number and the best 4,096 hold less than top-p asks for
                assert top_k == 0 and temperature and vocab > 4096
                weight = torch.softmax(logits[row].double() / temperature, 0).sort(descending=True).values
                assert float(weight[:4096].sum()) < top_p + 1e-6
                continue
            assert int(status[row]) == ops.SAMPLE_OK
            config = {"temperature": temperature, "top_k": top_k, "top_p": top_p, "min_p": min_p}
            if temperature:
                assert int(tokens[row]) == draw_temperature(logits[row].numpy(), config, [], float(uniform[row])), (row, config)
            else:
                best = logits[row][torch.isfinite(logits[row])].max()
                assert int(tokens[row]) == int(torch.nonzero(logits[row] == best)[0])
