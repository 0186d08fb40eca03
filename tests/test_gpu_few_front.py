"""A few tokens: the products that depend on them alone go in one launch (router logits, shared gate and
up, latent projection) and keep the bits of their own kernels; the latent shape's last two
projections and their sum in another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth                            # noqa: E402
from moonshine_b200.layer import MoELayer                        # noqa: E402
from tests import gpu_util as G                                  # noqa: E402
from tests import test_gpu_latent as latent                      # noqa: E402


@pytest.mark.parametrize("tokens,hidden,shared,experts", [
    (9, 1024, 288, 21),         # eight splits; a block of router rows that ends early
    (16, 4096, 512, 16),        # sixteen splits from 4096 columns on
    (17, 1024, 256, 33),
    (24, 4096, 544, 17),
    (31, 4096, 4096, 16),
])
def test_layer_equals_its_steps(tokens, hidden, shared, experts):
    block = 32 if shared % 128 else 128
    cfg = synth.baseline_config(hidden=hidden, expert_hidden=512, experts=experts, top_k=4, shared_hidden=shared,
                                q8_block=block, q8_scale_type=synth.Q8_F16)
    layer = MoELayer(cfg, synth.make_layer(cfg, 3), seed=3, device=G.DEV, max_tokens=tokens)
    x = G.dev(synth.activations(4, tokens, hidden)).view(torch.bfloat16)
    want, ids, weights = layer.forward(x, want_routes=True)
    k, routes = 4, tokens * 4
    ids1, wts1, logits = G.empty((tokens, k), np.uint32), G.empty((tokens, k), np.float32), G.empty((tokens, experts), np.float32)
    assert ops.k3_moe_route(layer.desc, ids1, wts1, logits, x, tokens)
    assert np.array_equal(G.host(ids1).view(np.uint32), ids.cpu().numpy().view(np.uint32))
    assert np.array_equal(G.host(wts1), weights.cpu().numpy())
    off, sr, st, inv = [G.empty((experts + 1,), np.uint32)] + [G.empty((routes,), np.uint32) for _ in range(3)]
    need = ops.k3_moe_dispatch_workspace_bytes(tokens, k, experts)
    ws = torch.empty(need, dtype=torch.uint8, device=G.DEV)
    assert ops.k3_moe_dispatch_build(off, sr, st, inv, ids, tokens, k, experts, ws, need)
    need = ops.k3_moe_experts_workspace_bytes(layer.desc, routes, tokens)
    ws = torch.empty(need, dtype=torch.uint8, device=G.DEV)
    rows, out, sh = (torch.empty((n, hidden), dtype=x.dtype, device=G.DEV) for n in (routes, tokens, tokens))
    g, u, a = (torch.empty((tokens, shared), dtype=x.dtype, device=G.DEV) for _ in range(3))
    assert ops.k3_moe_experts_grouped_ws(layer.desc, rows, None, x, st, tokens, off, routes, ws, need)
    assert ops.k3_moe_shared_expert(layer.desc, sh, g, u, a, x, tokens)
    assert ops.k3_moe_combine(out, rows, inv, weights, sh, tokens, k, hidden)
    torch.cuda.synchronize()
    assert ops.k3_moe_device_status() == 0
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("tokens,hidden,width,shared", [
    (2, 1024, 512, 256),
    (8, 4096, 512, 256),        # sixteen splits in front, eight at the end
    (9, 1024, 544, 256),        # latent rows that end inside a pair of 16-row blocks
    (31, 4096, 512, 4096),      # the last two projections have different splits: one after the other
])
def test_latent_layer_matches_oracle(oracle, monkeypatch, tokens, hidden, width, shared):
    if width % latent.BLOCK:
        monkeypatch.setattr(latent, "BLOCK", 32)
    for name, value in (("H", hidden), ("L", width), ("S", shared)):
        monkeypatch.setattr(latent, name, value)
    latent.test_latent_layer_matches_oracle(oracle, tokens)
