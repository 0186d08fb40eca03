"""Shared expert of 1 to 31 token rows (Q8 products on mma.sync): edges of the 8-row tiles and the
16-row blocks, column counts that leave splits without a step, both scale formats."""
import numpy as np
import pytest

from moonshine_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import _native, ops        # noqa: E402
from tests import gpu_util as G                # noqa: E402


@pytest.mark.parametrize("tokens", [1, 2, 7, 8, 9, 16, 17, 24, 25, 31])
@pytest.mark.parametrize("d,s,block,st", [
    (1024, 512, 32, synth.Q8_F16),
    (3584, 384, 128, synth.Q8_F32),
    (160, 96, 32, synth.Q8_F32),            # five and three column steps for eight splits
    (7168, 2048, 32, synth.Q8_F16),
])
def test_shared_expert_of_few_rows(oracle, tokens, d, s, block, st):
    cfg = synth.baseline_config(hidden=d, expert_hidden=512, experts=8, top_k=2, shared_hidden=s,
                                q8_block=block, q8_scale_type=st)
    w = synth.make_layer(cfg, seed=9, experts=False)
    x = synth.activations(tokens, tokens, d)
    desc = _native.LayerDesc(hidden=d, expert_hidden=512, expert_count=8, top_k=2, shared_hidden=s,
                             q8_block=block, q8_scale_type=st, activation=cfg["activation"],
                             route_scale=1.0, local_expert_count=8)
    keep = {k: G.dev(w[k]) for k in w if k.startswith("shared")}
    for k, v in keep.items():
        setattr(desc, k, v.data_ptr())
    out = G.empty((tokens, d), np.uint16)
    g, u, a = (G.empty((tokens, s), np.uint16) for _ in range(3))
    assert ops.k3_moe_shared_expert(desc, out, g, u, a, G.dev(x), tokens)
    want = {n: oracle.q8_gemm(w[f"shared_{n}_q"], w[f"shared_{n}_s"], x, s, d, block, st) for n in ("gate", "up")}
    got_a = G.host(a, np.uint16)
    # fp32 sums in another order: about one result in 2^9 falls on the other side of a bf16
    # rounding line and moves by 2^-8, so rel-L2 is near 2^-8 * 2^-4.5 = 2e-4
    assert G.rel_l2(G.host(g, np.uint16), want["gate"]) <= 1e-3
    assert G.rel_l2(G.host(u, np.uint16), want["up"]) <= 1e-3
    act = oracle.activation(G.host(g, np.uint16), G.host(u, np.uint16), cfg["activation"])
    assert G.rel_l2(got_a, act) <= 1e-3
    down = oracle.q8_gemm(w["shared_down_q"], w["shared_down_s"], got_a, d, s, block, st)
    assert G.rel_l2(G.host(out, np.uint16), down) <= 1e-3
