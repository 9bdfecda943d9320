"""The room of 32-bit products for the parts of their left operand: one for all products and graphs of a runner, and known
to the memory plan."""
import pytest
import torch


def test_the_plan_counts_the_room():
    from vipera_rs_b200.config import architecture_of
    from vipera_rs_b200.engine import planner

    config = {"architectures": ["Qwen2ForCausalLM"], "num_hidden_layers": 2, "hidden_size": 256, "num_attention_heads": 4,
              "num_key_value_heads": 2, "intermediate_size": 704, "vocab_size": 512, "rope_theta": 10000.0, "rms_norm_eps": 1e-6,
              "tie_word_embeddings": True, "max_position_embeddings": 512}
    arch = architecture_of(config)
    spec = arch.model_spec(arch.config_from_dict(config))
    wide, narrow = (planner.workspace_bytes(spec, 1, size, tokens=1) for size in (4, 2))
    assert wide - narrow >= planner.PRODUCT_PARTS_BYTES


@pytest.mark.gpu
def test_no_product_wants_more_than_the_plan_counts():
    from vipera_rs_b200.engine import planner
    from vipera_rs_b200.kernels import ops

    for m, n, k in [(65, 256, 4096), (2048, 4096, 14336), (100000, 1000, 70000), (8192, 9728, 896)]:
        assert 0 < ops.gemm_simt_room(m, n, k) <= planner.PRODUCT_PARTS_BYTES


@pytest.mark.gpu
def test_captured_products_share_the_room():
    from types import SimpleNamespace

    from vipera_rs_b200.kernels import ops
    from vipera_rs_b200.parts.base import Workspace
    from vipera_rs_b200.parts.linear import Linear

    device = "cuda:0"
    torch.manual_seed(1)
    linear = Linear(torch.randn(512, 4096, device=device), torch.float32, device)
    context = SimpleNamespace(workspace=Workspace(device))
    rows = [1024, 512, 640, 768, 896, 960]
    inputs = [torch.randn(m, 4096, device=device) for m in rows]
    outs = [torch.empty(m, 512, device=device) for m in rows]
    room = ops.gemm_simt_room(1024, 512, 4096)
    assert room > 20 << 20
    for a, out in zip(inputs, outs):
        linear(context, a, out=out)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before, graphs = torch.cuda.memory_reserved(), []
    eager = [out.clone() for out in outs]
    for a, out in zip(inputs, outs):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            linear(context, a, out=out)
        graphs.append(graph)
    kept = torch.cuda.memory_reserved() - before
    assert kept < room, kept
    for out, graph in zip(outs, graphs):
        out.zero_()
        graph.replay()
    assert all(torch.equal(out, want) for out, want in zip(outs, eager))
