"""MXFP4 operator products at the edges of the row kernels: the one-tile kernel and the tile
kernels at the vector counts where the width of a pass changes, scale groups that do not
divide into the eight K splits, rows that do not fill a block, misaligned vectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth          # noqa: E402
from tests import gpu_util as G                # noqa: E402


@pytest.mark.parametrize("vectors", [1, 8, 9, 17, 25, 33, 57, 113])
@pytest.mark.parametrize("rows,cols", [(1, 32), (33, 96), (65, 544), (3072, 608)])
def test_rows_against_oracle_and_single_calls(oracle, vectors, rows, cols):
    p = synth.bytes_uniform(synth.stream_key(41, cols), rows * cols // 2)
    s = synth.bytes_uniform(synth.stream_key(42, cols), rows * cols // 32, 0, 128)
    x = synth.bf16_bits(synth.normal_f32(synth.stream_key(43, vectors), vectors * cols, 1.0)).reshape(vectors, cols)
    dp, ds, dx = G.dev(p), G.dev(s), G.dev(x)
    out = G.empty((vectors, rows), np.uint16)
    assert ops.k3_rocm_mxfp4_gemm_bf16(out, dp, ds, dx, vectors, rows, cols)
    got = G.host(out, np.uint16)
    # the reference's acceptance rule for another summation order (tests/gpu_util.py)
    G.check_mxfp4_envelope(got, oracle.mxfp4_gemm(p, s, x, rows, cols).reshape(vectors, rows),
                           oracle.mxfp4_gemm_f64(p, s, x, rows, cols).reshape(vectors, rows))
    one = G.empty((rows,), np.uint16)
    for v in {0, vectors // 2, vectors - 1}:
        assert ops.k3_rocm_mxfp4_gemv_bf16(one, dp, ds, dx[v], rows, cols)
        assert np.array_equal(G.host(one, np.uint16), got[v])


def test_misaligned_vectors_equal_aligned_ones():
    rows, cols, vectors = 40, 3584, 11
    p, s = (G.dev(synth.bytes_uniform(synth.stream_key(44, i), rows * cols // d, *r))
            for i, d, r in ((1, 2, (0, 256)), (2, 32, (119, 5))))
    x = G.dev(synth.bf16_bits(synth.normal_f32(synth.stream_key(44, 3), vectors * cols, 1.0)))
    odd = torch.empty(vectors * cols + 1, dtype=torch.int16, device="cuda")[1:]
    odd.copy_(x)
    a, b = G.empty((vectors, rows), np.uint16), G.empty((vectors, rows), np.uint16)
    assert ops.k3_rocm_mxfp4_gemm_bf16(a, p, s, x, vectors, rows, cols)
    assert ops.k3_rocm_mxfp4_gemm_bf16(b, p, s, odd.data_ptr(), vectors, rows, cols)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
