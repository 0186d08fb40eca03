"""A value that is not finite makes the results of its own row NaN and of no other, whichever
kernel the row's group goes to (up to 16 rows, 17 to 64, more; one token)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import _native, ops, synth  # noqa: E402
from tests import gpu_util as G                # noqa: E402
from tests import test_gpu_tc as tc            # noqa: E402

INF, NEG_INF, NAN, LARGE = 0x7F80, 0xFF80, 0x7FC0, 0x7E00      # bf16; LARGE = 2^125


def experts(counts, d=1024, i=512, seed=31, smaller=0):
    """A description with len(counts) experts; gate and up weights times 2^-smaller."""
    e = len(counts)
    cfg = synth.baseline_config(hidden=d, expert_hidden=i, experts=e, top_k=2, shared_hidden=0)
    w = synth.make_layer(cfg, seed=seed)
    desc = _native.LayerDesc(hidden=d, expert_hidden=i, expert_count=e, top_k=2, shared_hidden=0,
                             activation=ops.ACT_SWIGLU, route_scale=1.0, local_expert_count=e)
    for k in ("w1_scales", "w3_scales"):
        w[k] = w[k] - np.uint8(smaller)
    keep = {k: G.dev(w[k]) for k in w if k.startswith("w")}
    for k, v in keep.items():
        setattr(desc, k, v.data_ptr())
    return desc, keep


@pytest.mark.parametrize("gathered", [False, True])
@pytest.mark.parametrize("counts", [[3, 16, 20, 1], [3, 64, 200, 17]])
@pytest.mark.parametrize("value", [NAN, INF, NEG_INF])
def test_grouped_products(counts, value, gathered):
    d, rows = 1024, sum(counts)
    # weights so small that an infinity taken for the largest finite value would not overflow by itself
    desc, keep = experts(counts, smaller=90)
    x, offsets = synth.activations(31, rows, d), np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    hit = [0, 4, int(offsets[2]) + 6, rows - 1]                # one row of each group
    x[hit, 77] = value
    index, source = None, 0
    if gathered:
        order = np.random.default_rng(3).permutation(rows).astype(np.uint32)
        index, source, x = G.dev(np.argsort(order).astype(np.uint32)), rows, x[order]
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, source)
    ws, out = torch.empty(need, dtype=torch.uint8, device="cuda"), G.empty((rows, d), np.uint16)
    assert ops.k3_moe_experts_grouped_ws(desc, out, None, G.dev(x), index, source, G.dev(offsets), rows, ws, need)
    tc.status_ok()
    nan = np.isnan(G.bf16_f32(G.host(out, np.uint16)))
    assert nan[hit].all()
    assert not np.delete(nan, hit, axis=0).any()


@pytest.mark.parametrize("counts", [[3, 16, 20, 1], [3, 64, 200, 17]])
def test_an_activation_that_overflows(counts):
    """Finite rows so large that gate * up leaves bf16's range: the products of gate and up are
    finite, the activation is infinite in some columns, the row's results are NaN."""
    d, i, rows = 1024, 512, sum(counts)
    desc, keep = experts(counts)
    x, offsets = synth.activations(31, rows, d), np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    hit = [0, 4, int(offsets[2]) + 6, rows - 1]
    x[hit, 77] = LARGE
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, 0)
    ws, out = torch.empty(need, dtype=torch.uint8, device="cuda"), G.empty((rows, d), np.uint16)
    act = G.empty((rows, i), np.uint16)
    assert ops.k3_moe_experts_grouped_ws(desc, out, act, G.dev(x), None, 0, G.dev(offsets), rows, ws, need)
    tc.status_ok()
    a = G.bf16_f32(G.host(act, np.uint16))
    assert np.isinf(a[hit]).any(axis=1).all()
    nan = np.isnan(G.bf16_f32(G.host(out, np.uint16)))
    assert nan[hit].all()
    assert not np.delete(nan, hit, axis=0).any()


@pytest.mark.parametrize("value", [NAN, INF, NEG_INF, LARGE])
def test_one_token(value):
    d = 1024
    desc, keep = experts([1, 1, 1, 1])
    x = synth.activations(31, 1, d)
    need = ops.k3_moe_experts_token_workspace_bytes(desc)
    assert need
    ws, out = torch.empty(need, dtype=torch.uint8, device="cuda"), G.empty((1, d), np.uint16)
    ids, weights = G.dev(np.array([2, 0], np.uint32)), G.dev(np.array([0.5, 0.5], np.float32))
    assert ops.k3_moe_experts_token(desc, out, G.dev(x), ids, weights, ws, need)
    assert np.isfinite(G.bf16_f32(G.host(out, np.uint16))).all()
    x[0, 77] = value
    assert ops.k3_moe_experts_token(desc, out, G.dev(x), ids, weights, ws, need)
    tc.status_ok()
    assert np.isnan(G.bf16_f32(G.host(out, np.uint16))).all()
