"""Q8 products of 1 to 31 rows: a row's results have the same bits in a batch of any size."""
import numpy as np
import pytest

from moonshine_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import _native, ops        # noqa: E402
from tests import gpu_util as G                # noqa: E402


@pytest.mark.parametrize("d,s,block", [(7168, 2048, 32), (4096, 4128, 32), (4128, 4256, 32), (4064, 512, 32),
                                       (8192, 7168, 128)])
def test_shared_expert_rows_do_not_depend_on_the_batch(d, s, block):
    """Both sides of the 4096 columns where the number of splits changes, column counts that leave
    some splits a step short, and every number of 8-row tiles."""
    cfg = synth.baseline_config(hidden=d, expert_hidden=512, experts=8, top_k=2, shared_hidden=s, q8_block=block,
                                q8_scale_type=synth.Q8_F16)
    w = synth.make_layer(cfg, seed=9, experts=False)
    x = G.dev(synth.activations(4, 31, d))
    desc = _native.LayerDesc(hidden=d, expert_hidden=512, expert_count=8, top_k=2, shared_hidden=s, q8_block=block,
                             q8_scale_type=synth.Q8_F16, activation=cfg["activation"], route_scale=1.0,
                             local_expert_count=8)
    keep = {k: G.dev(w[k]) for k in w if k.startswith("shared")}
    for k, v in keep.items():
        setattr(desc, k, v.data_ptr())

    def run(tokens):
        out = G.empty((tokens, d), np.uint16)
        g, u, a = (G.empty((tokens, s), np.uint16) for _ in range(3))
        assert ops.k3_moe_shared_expert(desc, out, g, u, a, x, tokens)
        return [G.host(t, np.uint16) for t in (g, u, a, out)]

    whole = run(31)
    for tokens in (1, 2, 8, 9, 16, 17, 24, 25):
        for got, want in zip(run(tokens), whole):
            assert np.array_equal(got, want[:tokens]), tokens
