"""A few tokens: the products that depend on them alone go in one launch (router logits, shared gate and
up, latent projection) and keep the bits of their own kernels; the latent shape's last two
projections and their sum in another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import _native, ops, synth                   # noqa: E402
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


@pytest.mark.parametrize("hidden,width,shared,block,f16", [
    (1024, 512, 256, 128, False),       # eight splits in front and at the end
    (4096, 512, 256, 32, True),         # sixteen in front, eight at the end
    (4096, 4096, 4128, 32, False),      # sixteen everywhere
    (7168, 3584, 2048, 128, False),     # the real shape
    (4096, 512, 4096, 64, True),        # the last two projections have different splits: one after the other
    (1056, 544, 96, 32, True),          # rows and columns that end inside a block, a pair of blocks and a step
])
def test_latent_layer_equals_its_separate_launches(hidden, width, shared, block, f16):
    """Without a shared expert every product of the latent layer has a launch of its own: that result, the
    shared expert and the add give the bits of the joined launches, for every number of rows' tiles."""
    g = torch.Generator(device=G.DEV)
    g.manual_seed(hidden + width + shared)
    e, k, inner = 24, 4, 512

    def q8(rows, cols):
        s = torch.rand((rows, cols // block), generator=g, device=G.DEV) * 9e-4 + 1e-4
        return torch.randint(-127, 128, (rows, cols), generator=g, device=G.DEV, dtype=torch.int8), s.half() if f16 else s

    def normal(*shape, sigma=1.0):
        return (torch.randn(shape, generator=g, device=G.DEV) * sigma).to(torch.bfloat16)

    t = {"router_weight": normal(e, hidden, sigma=0.02), "router_bias": torch.rand(e, generator=g, device=G.DEV) * 0.2 - 0.1}
    for n, rows, cols in (("w1", inner, width), ("w3", inner, width), ("w2", width, inner)):
        t[n + "_packed"] = torch.randint(0, 256, (e, rows, cols // 2), generator=g, device=G.DEV, dtype=torch.uint8)
        t[n + "_scales"] = torch.randint(119, 124, (e, rows, cols // 32), generator=g, device=G.DEV, dtype=torch.uint8)
    for n, rows, cols in (("gate", shared, hidden), ("up", shared, hidden), ("down", hidden, shared)):
        t[f"shared_{n}_q"], t[f"shared_{n}_s"] = q8(rows, cols)
    p = {"norm_weight": normal(width, sigma=0.5)}
    p["down_q"], p["down_s"] = q8(width, hidden)
    p["up_q"], p["up_s"] = q8(hidden, width)
    desc = _native.LatentDesc(latent=width, norm_epsilon=1e-5, **{n: v.data_ptr() for n, v in p.items()})
    for n, v in dict(hidden=hidden, expert_hidden=inner, expert_count=e, local_expert_count=e, top_k=k, shared_hidden=shared,
                     q8_block=block, q8_scale_type=int(f16), activation=ops.ACT_SITU, beta=4.0, linear_beta=25.0,
                     route_scale=1.0, **{n: v.data_ptr() for n, v in t.items()}).items():
        setattr(desc.layer, n, v)
    for tokens in (1, 2, 8, 9, 16, 17, 24, 25, 31):
        x = normal(tokens, hidden)
        need = ops.k3_moe_latent_workspace_bytes(desc, tokens)
        ws = torch.empty(need, dtype=torch.uint8, device=G.DEV)
        got, full, sh, want = (torch.empty_like(x) for _ in range(4))
        ids, ids1 = (G.empty((tokens, k), np.uint32) for _ in range(2))
        wts, wts1, logits = G.empty((tokens, k), np.float32), G.empty((tokens, k), np.float32), G.empty((tokens, e), np.float32)
        gate, up, act = (torch.empty((tokens, shared), dtype=x.dtype, device=G.DEV) for _ in range(3))
        assert ops.k3_moe_latent_layer_forward(desc, got, x, tokens, ws, need, ids, wts)
        assert ops.k3_moe_route(desc.layer, ids1, wts1, logits, x, tokens)
        assert ops.k3_moe_shared_expert(desc.layer, sh, gate, up, act, x, tokens)
        desc.layer.shared_hidden = 0
        assert ops.k3_moe_latent_layer_forward(desc, full, x, tokens, ws, need, None, None)
        desc.layer.shared_hidden = shared
        assert ops.k3_rocm_add_bf16(want, full, sh, tokens * hidden)
        torch.cuda.synchronize()
        assert ops.k3_moe_device_status() == 0
        assert torch.equal(ids, ids1) and torch.equal(wts, wts1), tokens
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), tokens
        assert torch.isfinite(got.float()).all() and (got != 0).any()
