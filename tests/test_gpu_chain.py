"""The layer's many-token sequence against the same steps called one by one, and replayed from a
CUDA graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth          # noqa: E402
from moonshine_b200.layer import MoELayer, bf16_tensor_to_bits   # noqa: E402
from tests import gpu_util as G                # noqa: E402

SHAPE = dict(hidden=1024, expert_hidden=512, top_k=4, shared_hidden=0)


@pytest.mark.parametrize("tokens,experts,bias", [
    (9, 16, "uniform"),         # packed kernel only
    (16, 16, "hot4"),
    (40, 16, "hot4"),           # four experts with all 40 tokens, the others with few or none
    (65, 64, "hot4"),           # groups of all three kernels
    (300, 64, "zipf"),
])
def test_layer_equals_its_steps(tokens, experts, bias):
    """The layer converts a token once for all its product rows and skips tokens that no packed group
    needs; the step by itself converts every product row.  Same bits."""
    cfg = synth.baseline_config(experts=experts, bias_mode=bias, **SHAPE)
    d, k = cfg["hidden"], cfg["top_k"]
    layer = MoELayer(cfg, synth.make_layer(cfg, 3), seed=3, device=G.DEV, max_tokens=tokens)
    x = G.dev(synth.activations(4, tokens, d)).view(torch.bfloat16)
    want, ids, weights = layer.forward(x, want_routes=True)
    routes = tokens * k
    off, sr, st, inv = [G.empty((experts + 1,), np.uint32)] + [G.empty((routes,), np.uint32) for _ in range(3)]
    need = ops.k3_moe_dispatch_workspace_bytes(tokens, k, experts)
    ws = torch.empty(need, dtype=torch.uint8, device=G.DEV)
    assert ops.k3_moe_dispatch_build(off, sr, st, inv, ids, tokens, k, experts, ws, need)
    need = ops.k3_moe_experts_workspace_bytes(layer.desc, routes, tokens)
    assert need
    ws = torch.empty(need, dtype=torch.uint8, device=G.DEV)
    rows, out = torch.empty((routes, d), dtype=x.dtype, device=G.DEV), torch.empty_like(x)
    assert ops.k3_moe_experts_grouped_ws(layer.desc, rows, None, x, st, tokens, off, routes, ws, need)
    assert ops.k3_moe_combine(out, rows, inv, weights, None, tokens, k, d)
    torch.cuda.synchronize()
    assert ops.k3_moe_device_status() == 0
    assert np.array_equal(bf16_tensor_to_bits(out), bf16_tensor_to_bits(want))


@pytest.mark.parametrize("tokens", [12, 40, 300])
def test_many_token_layer_replays_from_a_cuda_graph(tokens):
    """Including the launches that start before the kernel in front of them has ended."""
    cfg = synth.baseline_config(experts=16, **{**SHAPE, "shared_hidden": 512})
    layer = MoELayer(cfg, synth.make_layer(cfg, 3), seed=3, device=G.DEV, max_tokens=tokens)
    xs = [G.dev(synth.activations(5 + i, tokens, cfg["hidden"])).view(torch.bfloat16) for i in range(3)]
    eager = [bf16_tensor_to_bits(layer.forward(x)) for x in xs]
    static_x, stream, graph = xs[0].clone(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        layer.forward(static_x)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            static_out = layer.forward(layer.forward(static_x))
            first_out = layer.forward(static_x)
    for i in (1, 2, 0, 2):
        static_x.copy_(xs[i])
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(bf16_tensor_to_bits(first_out), eager[i]), i
    again = layer.forward(layer.forward(xs[2]))
    assert np.array_equal(bf16_tensor_to_bits(static_out), bf16_tensor_to_bits(again))
    assert ops.k3_moe_device_status() == 0
