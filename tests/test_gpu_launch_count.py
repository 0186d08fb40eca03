"""The benchmark's counts of launches per layer pass are what a pass launches."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
runtime = pytest.importorskip("cuda.bindings.runtime")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import bench                                            # noqa: E402
from moonshine_b200 import synth                        # noqa: E402
from moonshine_b200.layer import LatentMoELayer, MoELayer   # noqa: E402


def launched(layer, x):
    layer.forward(x)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        layer.forward(x)
    _, _, count = runtime.cudaGraphGetNodes(graph.raw_cuda_graph())
    _, nodes, _ = runtime.cudaGraphGetNodes(graph.raw_cuda_graph(), count)
    return sum(runtime.cudaGraphNodeGetType(n)[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for n in nodes)


@pytest.mark.parametrize("tokens", [1, 2, 8, 9, 16, 17, 31, 32, 64, 65, 256, 257])
def test_launches_per_step(tokens):
    cfg = synth.baseline_config(experts=32)
    layer = MoELayer(cfg, synth.make_layer(cfg, 1, experts=False), seed=1, max_tokens=tokens)
    x = torch.randn((tokens, cfg["hidden"]), device="cuda").to(torch.bfloat16)
    assert launched(layer, x) == bench.launches_per_step(tokens, True)


@pytest.mark.parametrize("tokens", [32, 65, 257])
def test_latent_launches_per_step(tokens):
    cfg = synth.baseline_config(experts=32, expert_hidden=512, activation=synth.ACT_SITU, q8_block=128,
                                q8_scale_type=synth.Q8_F32, route_scale=1.0)
    layer = LatentMoELayer(cfg, 3584, seed=0, device="cuda:0", max_tokens=tokens)
    x = torch.randn((tokens, cfg["hidden"]), device="cuda").to(torch.bfloat16)
    assert launched(layer, x) == bench.latent_launches_per_step(tokens, True)
