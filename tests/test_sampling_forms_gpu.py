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


@pytest.mark.parametrize("vocab", [70, 4097, 65536, 151937])
@pytest.mark.parametrize("settings", [(1.0, 64, 1.0, 0.0), (1.0, 0, 0.6, 0.0), (0.9, 1000, 0.97, 0.02), (1.0, 4096, 1.0, 1e-4)])
def test_draws_over_the_bins(vocab, settings):
    """Bins of equal steps where they go wrong: what is wanted lies below the bins filled first, more ids in one than are
    ranked within it, steps of a few units in the last place, one value far below all others."""
    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.sampling import draw_temperature

    torch.manual_seed(vocab + settings[1])
    logits = torch.randn(6, vocab)
    logits[0] = logits[0] * 0.01 - 1.0
    logits[0, vocab // 3] = 2.0                       # the others lie in the lowest bins
    logits[1, vocab // 2] = -1e6                      # all but one in the first bin
    logits[2] = 1.0 + torch.randint(0, 5, (vocab,)) * 2.0 ** -23
    logits[3] = (logits[3] * 4).round() / 4           # ties within a bin
    logits[4] = torch.linspace(0.0, 12.0, vocab)[torch.randperm(vocab)]
    logits[5, vocab // 2:] = float("inf")             # counts as no logit
    uniform = torch.rand(6, dtype=torch.float64)
    temperature, top_k, top_p, min_p = settings
    tokens, status = (torch.full((6,), -7, dtype=torch.int32, device=DEV) for _ in range(2))
    full = lambda value, dtype=torch.float32: torch.full((6,), value, dtype=dtype, device=DEV)  # noqa: E731
    ops.sample(logits.to(DEV), temperature=full(temperature), top_k=full(top_k, torch.int32), top_p=full(top_p), min_p=full(min_p),
               uniform=uniform.to(DEV), tokens=tokens, status=status)
    config = {"temperature": temperature, "top_k": top_k, "top_p": top_p, "min_p": min_p}
    for row in range(6):
        if int(status[row]) == ops.SAMPLE_NEEDS_HOST:
            weight = torch.softmax(logits[row].masked_fill(torch.isinf(logits[row]), -float("inf")).double() / temperature, 0)
            assert top_k == 0 and float(weight.sort(descending=True).values[:4096].sum()) < top_p + 1e-6
            continue
        assert int(status[row]) == ops.SAMPLE_OK
        assert int(tokens[row]) == draw_temperature(logits[row].numpy(), config, [], float(uniform[row])), (row, config)
