"""Q8 products of few rows on values at the edges of their types: int8 -128 and 127, infinities and
NaN in a token row, against 64-bit sums."""
import numpy as np
import pytest

from moonshine_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import _native, ops        # noqa: E402
from tests import gpu_util as G                # noqa: E402


def gate_products(q, scales, x, d, s):
    """The gate product of the shared expert (bf16 [tokens, s]) as float64."""
    tokens = x.shape[0]
    keep = [G.dev(q), G.dev(scales), G.dev(np.zeros((d, s), np.int8)), G.dev(np.zeros((d, s // 32), np.float32))]
    desc = _native.LayerDesc(hidden=d, expert_hidden=512, expert_count=8, top_k=2, shared_hidden=s, q8_block=32,
                             q8_scale_type=synth.Q8_F32, activation=ops.ACT_SWIGLU, route_scale=1.0,
                             local_expert_count=8)
    desc.shared_gate_q = desc.shared_up_q = keep[0].data_ptr()
    desc.shared_gate_s = desc.shared_up_s = keep[1].data_ptr()
    desc.shared_down_q, desc.shared_down_s = keep[2].data_ptr(), keep[3].data_ptr()
    out = G.empty((tokens, d), np.uint16)
    g, u, a = (G.empty((tokens, s), np.uint16) for _ in range(3))
    assert ops.k3_moe_shared_expert(desc, out, g, u, a, G.dev(x), tokens)
    assert np.array_equal(G.host(g), G.host(u))
    return G.bf16_f32(G.host(g, np.uint16)).astype(np.float64)


@pytest.mark.parametrize("tokens", [1, 9, 31])
@pytest.mark.parametrize("d", [1024, 4096])
def test_edges_of_int8(tokens, d):
    s = 64
    rng = np.random.default_rng(tokens)
    q = rng.choice(np.array([-128, -127, -1, 0, 1, 127], np.int8), (s, d))
    q[0], q[1] = -128, 127
    scales = rng.uniform(1e-4, 1e-3, (s, d // 32)).astype(np.float32)
    x = synth.activations(3, tokens, d)
    want = G.bf16_f32(x).astype(np.float64) @ (q.astype(np.float64) * np.repeat(scales.astype(np.float64), 32, 1)).T
    got = gate_products(q, scales, x, d, s)
    # rounding to bf16 is at most 2^-9 of the result; fp32 sums of d terms are off by less than
    # d / 2 * 2^-24 of the sum of magnitudes
    magnitude = np.abs(G.bf16_f32(x)).astype(np.float64) @ (np.abs(q.astype(np.float64))
                                                            * np.repeat(scales.astype(np.float64), 32, 1)).T
    assert (np.abs(got - want) <= np.abs(want) * 2.0 ** -8 + magnitude * d * 2.0 ** -25).all()


@pytest.mark.parametrize("tokens", [1, 9, 31])
@pytest.mark.parametrize("value", [0x7F80, 0xFF80, 0x7FC0])
def test_values_that_are_not_finite(tokens, value):
    """An infinity times a nonzero weight is infinite, times zero NaN; other rows stay as they are."""
    d, s = 1024, 64
    rng = np.random.default_rng(tokens)
    q = rng.integers(-3, 4, (s, d)).astype(np.int8)
    scales = rng.uniform(1e-4, 1e-3, (s, d // 32)).astype(np.float32)
    x = synth.activations(3, tokens, d)
    clean = gate_products(q, scales, x, d, s)
    hit = tokens // 2
    x[hit, 77] = value
    got = gate_products(q, scales, x, d, s)
    assert np.array_equal(np.delete(got, hit, axis=0), np.delete(clean, hit, axis=0))
    with np.errstate(invalid="ignore"):
        want = float(G.bf16_f32(np.array([value], np.uint16))[0]) * q[:, 77].astype(np.float64)
    assert np.array_equal(got[hit], want, equal_nan=True)
