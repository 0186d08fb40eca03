"""Device dispatch on both sides of the one-block form's limits: 4096 routes, and the expert counts
around the default shared memory of a block."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from moonshine_b200 import ops                 # noqa: E402
from tests import gpu_util as G                # noqa: E402


def build(ids, tokens, top_k, experts):
    """Outputs of k3_moe_dispatch_build: offsets, sorted_route, sorted_token, inv_perm."""
    routes = tokens * top_k
    bufs = [G.empty((experts + 1,), np.uint32)] + [G.empty((routes,), np.uint32) for _ in range(3)]
    for b in bufs:
        b.fill_(-1)
    ws_bytes = ops.k3_moe_dispatch_workspace_bytes(tokens, top_k, experts)
    ws = G.empty((ws_bytes,), np.uint8)
    assert ops.k3_moe_dispatch_build(*bufs, G.dev(ids), tokens, top_k, experts, ws, ws_bytes)
    return [G.host(b, np.uint32) for b in bufs]


def check(routes, experts, seed):
    ids = np.random.default_rng(seed).integers(0, experts, routes).astype(np.uint32)
    offsets, sorted_route, sorted_token, inv = build(ids, routes, 1, experts)
    order = np.argsort(ids, kind="stable").astype(np.uint32)           # (expert asc, route asc)
    assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(np.bincount(ids, minlength=experts))]))
    assert np.array_equal(sorted_route, order) and np.array_equal(sorted_token, order)
    assert np.array_equal(inv[order], np.arange(routes))


def test_expert_counts_around_the_default_shared_memory():
    """In a process of its own, smallest first: a call with more experts raises the limit of the
    one-block kernel for all later ones."""
    res = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]


@pytest.mark.parametrize("tokens,top_k,experts", [(64, 4, 32), (512, 8, 32), (513, 8, 32), (700, 8, 896)])
def test_out_of_range_ids_on_both_sides_of_the_route_limit(tokens, top_k, experts):
    """They are left out of the order, the status word says so, and all other routes are placed."""
    assert ops.k3_moe_device_status_clear()
    rng = np.random.default_rng(tokens)
    ids = rng.integers(0, experts, tokens * top_k).astype(np.uint32)
    build(ids, tokens, top_k, experts)
    assert ops.k3_moe_device_status() == 0
    bad = rng.choice(ids.size, 7, replace=False)
    ids[bad] = [experts, experts + 1, 0xFFFFFFFF, 0x80000000, 1 << 20, experts + 31, 0xFFFFFFFE]
    offsets, sorted_route, sorted_token, inv = build(ids, tokens, top_k, experts)
    assert ops.k3_moe_device_status() & 2
    assert ops.k3_moe_device_status_clear() and ops.k3_moe_device_status() == 0
    good = np.flatnonzero(ids < experts)
    order = good[np.argsort(ids[good], kind="stable")].astype(np.uint32)
    assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(np.bincount(ids[good], minlength=experts))]))
    n = good.size
    assert np.array_equal(sorted_route[:n], order) and np.array_equal(sorted_token[:n], order // top_k)
    assert np.array_equal(inv[order], np.arange(n))
    assert (sorted_route[n:] == 0xFFFFFFFF).all() and (inv[bad] == 0xFFFFFFFF).all()       # untouched


def test_the_shared_histograms_of_a_larger_call_do_not_leak():
    """Of the calls without a workspace only those above 4096 routes use the shared array: a large
    one, a smaller one with another expert count, and the large one again."""
    import ctypes as C
    for tokens, top_k, experts in ((8192, 16, 896), (700, 8, 64), (8192, 16, 896)):
        ids = np.random.default_rng(tokens).integers(0, experts, tokens * top_k).astype(np.uint32)
        got = [G.empty((experts + 1,), np.uint32)] + [G.empty((ids.size,), np.uint32) for _ in range(3)]
        err = C.create_string_buffer(256)
        assert ops.k3_moe_dispatch_build_noalloc(*got, G.dev(ids), tokens, top_k, experts, err, 256), err.value
        for a, b in zip(got, build(ids, tokens, top_k, experts)):
            assert np.array_equal(G.host(a, np.uint32), b)


if __name__ == "__main__":
    for e in (1, 765, 766, 767, 768, 1024):
        for n in (1, 4096, 4097):
            check(n, e, seed=e + n)
