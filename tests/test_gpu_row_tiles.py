"""Two-term kernel: groups of more than 64 rows are cut into even tiles of at most 160 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import synth                       # noqa: E402
from tests import gpu_util as G                        # noqa: E402
from tests.test_gpu_nonfinite import experts           # noqa: E402
from tests import test_gpu_tc as tc                    # noqa: E402


@pytest.mark.parametrize("counts", [
    [64, 65, 80, 81, 128, 129, 144, 145],
    [159, 160, 161, 0, 176, 320, 321, 17],             # one, two and three tiles; a multiple of 16 short and over
    [481, 1, 96, 640, 641, 16, 33, 2],
])
def test_products_at_the_tile_edges(oracle, counts):
    tc.test_grouped_expert_products_block_scaled(oracle, counts, True)


@pytest.mark.parametrize("d,i", [(512, 512), (7168, 2048)])       # one pair of scale batches per item, and many
def test_row_bits_do_not_depend_on_the_tile(d, i):
    """The same 65 rows at the start of groups of different sizes, and as the group's last rows."""
    counts = [65, 160, 161, 330]
    desc, keep = experts([1] * len(counts), d, i)
    same = synth.activations(3, 65, d)
    x = synth.activations(7, sum(counts), d)
    ends = np.cumsum(counts)
    for n, end in zip(counts, ends):
        x[end - n:end - n + 65] = same
    for n in ("w1_packed", "w1_scales", "w3_packed", "w3_scales", "w2_packed", "w2_scales"):   # the same expert everywhere
        t = keep[n].view(torch.uint8).view(len(counts), -1)
        t[1:] = t[0]
    from moonshine_b200 import ops
    rows = sum(counts)
    offsets = np.concatenate([[0], ends]).astype(np.uint32)
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, 0)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")

    def run(values):
        out, act = G.empty((rows, d), np.uint16), G.empty((rows, i), np.uint16)
        assert ops.k3_moe_experts_grouped_ws(desc, out, act, G.dev(values), None, 0, G.dev(offsets), rows, ws, need)
        tc.status_ok()
        return G.host(act, np.uint16), G.host(out, np.uint16)

    act, out = run(x)
    for n, end in zip(counts[1:], ends[1:]):
        assert np.array_equal(out[end - n:end - n + 65], out[:65]) and np.array_equal(act[end - n:end - n + 65], act[:65])
    for n, end in zip(counts, ends):
        x[end - 65:end] = same
    act, out = run(x)
    for n, end in zip(counts[1:], ends[1:]):
        assert np.array_equal(out[end - 65:end], out[:65]) and np.array_equal(act[end - 65:end], act[:65])
