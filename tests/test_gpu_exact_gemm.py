"""BF16 and Q8 products whose summation order is fixed, at the edges of the tiles the
launcher picks by the number of input rows, and router rows at the edges of the block
selection: equal to the oracle bit for bit (the order of every fp32 addition is the
reference's, so there is no tolerance to state)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth          # noqa: E402
from tests import gpu_util as G                # noqa: E402

VECTORS = [1, 2, 3, 5, 8, 9, 17, 33]


def _x(seed, n, cols):
    return synth.bf16_bits(synth.normal_f32(synth.stream_key(seed, n), n * cols, 1.0)).reshape(n, cols)


@pytest.mark.parametrize("vectors", VECTORS)
@pytest.mark.parametrize("rows,cols,block,st", [(1, 8, 8, 0), (19, 2048, 128, 0), (37, 2312, 8, 1), (33, 7168, 32, 1)])
def test_q8_rows(oracle, vectors, rows, cols, block, st):
    q = synth.int8_uniform(synth.stream_key(31, rows), rows * cols).reshape(rows, cols)
    s = synth.uniform_f32(synth.stream_key(32, rows), rows * cols // block, 1e-4, 1e-3)
    s = s.astype(np.float16 if st else np.float32).reshape(rows, cols // block)
    x = _x(33, vectors, cols)
    out = G.empty((vectors, rows), np.uint16)
    assert ops.k3_moe_q8_gemm_bf16(out, G.dev(q), G.dev(s), G.dev(x), vectors, rows, cols, block, st)
    assert np.array_equal(G.host(out, np.uint16), oracle.q8_gemm(q, s, x, rows, cols, block, st).reshape(vectors, rows))


@pytest.mark.parametrize("vectors", VECTORS)
@pytest.mark.parametrize("rows,cols", [(1, 4), (19, 260), (35, 1021), (33, 7168)])
def test_bf16_rows(oracle, vectors, rows, cols):
    w = synth.bf16_bits(synth.normal_f32(synth.stream_key(34, rows), rows * cols, 0.05)).reshape(rows, cols)
    x = _x(35, vectors, cols)
    out = G.empty((vectors, rows), np.float32)
    assert ops.k3_rocm_bf16_gemm_f32(out, G.dev(w), G.dev(x), vectors, rows, cols)
    want = np.asarray(oracle.bf16_gemm(w, x, rows, cols)).reshape(vectors, rows)
    assert np.array_equal(G.host(out).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("experts,top_k", [(1, 1), (33, 32), (127, 5), (256, 16), (1024, 32)])
def test_router_rows_with_ties(oracle, experts, top_k):
    # logits on a coarse grid: most of the selection is decided by ties, many rows pass more
    # than 256 candidates; sigmoid of grid values is far enough apart to be order-safe
    rows = 9
    logits = np.round(synth.normal_f32(synth.stream_key(36, experts), rows * experts, 1.7)).reshape(rows, experts)
    bias = np.zeros(experts, np.float32)
    ids, w = G.empty((rows, top_k), np.uint32), G.empty((rows, top_k), np.float32)
    assert ops.k3_rocm_router_topk_f32_batch(ids, w, G.dev(logits.astype(np.float32)), G.dev(bias), rows, experts,
                                             top_k, 2.5)
    want = [oracle.router_topk(logits[v].astype(np.float32), bias, top_k, 2.5) for v in range(rows)]
    assert np.array_equal(G.host(ids, np.uint32), np.stack([np.asarray(i).reshape(-1) for i, _ in want]))
    # device expf against libm: two ulps of a score, carried through the sum and the quotient
    assert np.abs(G.host(w) - np.stack([np.asarray(x).reshape(-1) for _, x in want])).max() <= 2.5e-6
