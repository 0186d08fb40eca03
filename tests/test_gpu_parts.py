"""A part of a pass gets the bits of the whole pass: the grouped expert products with the groups'
rows and places given, and the pipelined form of the expert-parallel pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from moonshine_b200 import ops, synth          # noqa: E402
from tests import gpu_util as G                # noqa: E402
from tests import test_gpu_tc as tc            # noqa: E402
from tests.test_gpu_nonfinite import experts   # noqa: E402

D, I = 7168, 2048          # wide enough for sums whose order shows in bf16


def products(desc, x, counts, group_rows=None, place=None):
    rows = int(sum(counts))
    offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    need = ops.k3_moe_experts_workspace_bytes(desc, rows, 0)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    out, act = G.empty((rows, D), np.uint16), G.empty((rows, I), np.uint16)
    if place is None:
        assert ops.k3_moe_experts_grouped_ws(desc, out, act, G.dev(x), None, 0, G.dev(offsets), rows, ws, need)
    else:
        assert ops.k3_moe_experts_grouped_part(desc, out, act, G.dev(x), None, 0, G.dev(offsets), G.dev(group_rows),
                                               G.dev(place), rows, ws, need)
    tc.status_ok()
    return G.host(act, np.uint16), G.host(out, np.uint16)


@pytest.mark.parametrize("counts", [[16, 17, 64, 65], [130, 33, 200, 3], [127, 192, 193, 40], [128, 257, 129, 0]])
@pytest.mark.parametrize("parts", [2, 3])
def test_products_of_a_part(counts, parts):
    """Rows dealt to the parts in blocks of random length, so that a part's rows lie in all tiles
    of a group, in few of them or in none."""
    desc, keep = experts(counts, D, I)
    rows = sum(counts)
    rng = np.random.default_rng(rows + parts)
    x = synth.activations(7, rows, D)
    group = np.repeat(np.arange(len(counts)), counts)
    place = np.concatenate([np.arange(c) for c in counts]).astype(np.uint32)
    owner = np.repeat(rng.integers(0, parts, rows), rng.integers(1, 12, rows))[:rows]
    act, out = products(desc, x, counts)
    alone = 0
    for p in range(parts):
        mine = np.flatnonzero(owner == p)
        assert mine.size >= 32
        part_counts = np.bincount(group[mine], minlength=len(counts))
        got = products(desc, x[mine], part_counts, np.array(counts, np.uint32), place[mine])
        assert np.array_equal(got[0], act[mine]) and np.array_equal(got[1], out[mine])
        by_itself = products(desc, x[mine], part_counts)
        alone += int((by_itself[1] != out[mine]).any())
    assert alone > 0                             # without the pass's counts the bits do differ


def test_invalid_arguments_of_a_part():
    desc, keep = experts([40, 40], D, I)
    need = ops.k3_moe_experts_workspace_bytes(desc, 80, 0)
    buf = torch.zeros(max(need, 80 * D * 2), dtype=torch.uint8, device="cuda")
    call = lambda **k: ops.k3_moe_experts_grouped_part(
        *(k.get(n, v) for n, v in [("desc", desc), ("out", buf), ("act", None), ("x", buf), ("index", None),
                                   ("source", 0), ("offsets", buf), ("group_rows", buf), ("place", buf), ("rows", 80),
                                   ("ws", buf), ("bytes", need)]))
    for bad in ({"out": None}, {"x": None}, {"offsets": None}, {"group_rows": None}, {"place": None}, {"rows": 0},
                {"rows": 31}, {"ws": None}, {"bytes": need - 1}, {"index": buf}):
        assert not call(**bad), bad


def test_pipelined_pass_equals_the_whole_one():
    """One rank: all of the exchange's steps, with the products in pieces."""
    import torch.distributed as dist
    from moonshine_b200 import ep
    from moonshine_b200.layer import MoELayer, bf16_tensor_to_bits
    import socket
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    device = torch.device("cuda", 0)
    torch.cuda.set_device(0)
    dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1, device_id=device)
    try:
        cfg = synth.baseline_config(hidden=4096, expert_hidden=1024, experts=16, top_k=4, shared_hidden=512)
        layer = MoELayer(cfg, synth.make_layer(cfg, seed=5), seed=5, device=device, max_tokens=1)
        for tokens in (128, 301):
            x = G.dev(synth.activations(6, tokens, cfg["hidden"])).view(torch.bfloat16)
            whole, ids, _ = ep.ep_forward(ep.NativeBackend(layer), x, cfg)
            for pieces in (2, 3):
                backends = [ep.NativeBackend(layer) for _ in range(pieces)]
                streams = [torch.cuda.Stream(device) for _ in range(pieces)]
                got, got_ids, _ = ep.ep_forward_pipelined(backends, x, cfg, streams=streams)
                torch.cuda.synchronize()
                assert torch.equal(got_ids, ids)
                assert np.array_equal(bf16_tensor_to_bits(got), bf16_tensor_to_bits(whole)), (tokens, pieces)
    finally:
        torch.cuda.synchronize()
        dist.destroy_process_group()
