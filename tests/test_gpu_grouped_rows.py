"""Grouped expert products where a group's row count decides the kernel and the operand
layout: up to 16 rows packed (8 and 9 rows: the accumulator halves), up to 32 and 64 rows
stacked two-term tiles, more with the terms as the A operand; groups of all kinds in one
call.  Same bars as tests/test_gpu_tc.py."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import numpy as np                             # noqa: E402

from moonshine_b200 import _native, ops, synth  # noqa: E402
from tests import gpu_util as G                # noqa: E402
from tests import test_gpu_tc as tc            # noqa: E402


@pytest.mark.parametrize("gathered", [False, True])
@pytest.mark.parametrize("counts", [
    [1, 2, 7, 8, 9, 15, 16, 17],
    [31, 32, 33, 47, 48, 63, 64, 65],
    [3, 0, 96, 127, 20, 128, 129, 40],
    [5, 5, 5, 5, 5, 5, 5, 5],
])
def test_row_counts_at_the_dispatch_edges(oracle, counts, gathered):
    tc.test_grouped_expert_products_block_scaled(oracle, counts, gathered)


@pytest.mark.parametrize("counts", [[65, 95, 96, 97, 0, 112, 113, 127], [128, 129, 192, 193, 0, 200, 256, 257]])
def test_tiles_of_more_than_64_rows(oracle, counts):
    tc.test_grouped_expert_products_block_scaled(oracle, counts, True)


def test_result_rows_of_any_alignment():
    """A result row is stored in 32-byte pieces where its address allows it: same bytes when the
    caller's buffers start two or sixteen bytes further."""
    d, i, e, rows = 1024, 512, 2, 200
    cfg = synth.baseline_config(hidden=d, expert_hidden=i, experts=e, top_k=2, shared_hidden=0)
    w = synth.make_layer(cfg, seed=29)
    x, offsets = G.dev(synth.activations(29, rows, d)), G.dev(np.array([0, 150, rows], np.uint32))
    desc = _native.LayerDesc(hidden=d, expert_hidden=i, expert_count=e, top_k=2, shared_hidden=0,
                             activation=cfg["activation"], route_scale=1.0, local_expert_count=e)
    keep = {k: G.dev(w[k]) for k in w if k.startswith("w")}
    for k, v in keep.items():
        setattr(desc, k, v.data_ptr())
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, 0)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    results = []
    for shift in (0, 1, 8):
        out, act = G.empty(rows * d + shift, np.uint16)[shift:], G.empty(rows * i + shift, np.uint16)[shift:]
        assert ops.k3_moe_experts_grouped_ws(desc, out, act, x, None, 0, offsets, rows, ws, need)
        tc.status_ok()
        results.append((G.host(out).tobytes(), G.host(act).tobytes()))
    assert results[0] == results[1] == results[2]


@pytest.mark.parametrize("counts", [[3, 16, 20, 1], [3, 16, 200, 1]])
def test_a_nan_reaches_its_own_row_only(counts):
    """One NaN in a row makes this row's results NaN and no other's, in every kernel."""
    d, i, e, rows = 1024, 512, 4, sum(counts)
    cfg = synth.baseline_config(hidden=d, expert_hidden=i, experts=e, top_k=2, shared_hidden=0)
    w = synth.make_layer(cfg, seed=31)
    x, offsets = synth.activations(31, rows, d), np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    hit = [0, 4, 25, rows - 1]
    x[hit, 77] = 0x7FC0
    desc = _native.LayerDesc(hidden=d, expert_hidden=i, expert_count=e, top_k=2, shared_hidden=0,
                             activation=cfg["activation"], route_scale=1.0, local_expert_count=e)
    keep = {k: G.dev(w[k]) for k in w if k.startswith("w")}
    for k, v in keep.items():
        setattr(desc, k, v.data_ptr())
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, 0)
    ws, out = torch.empty(need, dtype=torch.uint8, device="cuda"), G.empty((rows, d), np.uint16)
    assert ops.k3_moe_experts_grouped_ws(desc, out, None, G.dev(x), None, 0, G.dev(offsets), rows, ws, need)
    tc.status_ok()
    nan = np.isnan(G.bf16_f32(G.host(out, np.uint16)))
    assert nan[hit].all()
    assert not np.delete(nan, hit, axis=0).any()
