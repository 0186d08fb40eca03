"""Rows wider than what a grid's second dimension or a block's registers hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth          # noqa: E402
from tests import gpu_util as G                # noqa: E402


@pytest.mark.parametrize("hidden", [65534 * 512, 65535 * 512 + 8, 65535 * 512 + 3])
def test_weighted_sum(hidden):
    rows = G.dev((np.arange(hidden, dtype=np.uint32) % 16001 + 0x3C00).astype(np.uint16))
    out = G.empty((hidden,), np.uint16)
    assert ops.k3_rocm_weighted_sum_bf16(out, rows, G.dev(np.ones(1, np.float32)), 1, hidden)
    assert torch.equal(out, rows)


@pytest.mark.parametrize("hidden", [8192, 8193, 20000])
def test_rms_norm_of_rows_that_registers_do_not_hold(oracle, hidden):
    """8192 columns are held in a block's registers between the two passes, 8193 are not; in place
    as well."""
    x, w = synth.activations(3, 3, hidden), synth.activations(4, 1, hidden)[0]
    want = oracle.rms_norm(x, w, hidden, 1e-5)
    xd, out = G.dev(x), G.empty((3, hidden), np.uint16)
    assert ops.k3_rocm_rms_norm_bf16(out, xd, G.dev(w), 3, hidden, 1e-5)
    assert np.array_equal(G.host(out, np.uint16), want)
    assert ops.k3_rocm_rms_norm_bf16(xd, xd, G.dev(w), 3, hidden, 1e-5)
    assert np.array_equal(G.host(xd, np.uint16), want)
