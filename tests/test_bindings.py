"""Calls with their arguments converted in C behave as the ctypes form does: results, errors and
what is refused.  Every call ends at the library's own argument checks."""
import ctypes as C
import os
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ops():
    from moonshine_b200 import build
    build.build()
    from moonshine_b200 import ops
    return ops


def outcome(fn, args, kwargs):
    try:
        return "returned", fn(*args, **kwargs)
    except Exception as e:
        return type(e).__name__, str(e)


T = torch.zeros(4, 4)


def forms():
    from moonshine_b200 import _native
    desc, latent = _native.LayerDesc(), _native.LatentDesc()
    add = "k3_rocm_add_bf16"                   # (output, left, right, uint64 count, stream); no output: False
    for a, k in [((None, T, T, 0, 0), {}), ((None, T, T, 0), {"stream": 0}), ((None, T, T, 0), {"stream": T}),
                 ((None, T, T), {"stream": 0}), ((None, T, T, 0, 0, 0), {}), ((None, T, T, 0), {"other": 0}),
                 ((None, T.t(), T, 0), {"stream": 0}), ((None, T, T, 0), {"stream": T.t()}),
                 ((None, torch.nn.Parameter(T), 5, 0), {"stream": 0}), ((None, C.c_void_p(5), T, 0), {"stream": 0}),
                 ((None, np.int64(5), T, np.uint32(3)), {"stream": 0}), ((None, T, T, True), {"stream": 0}),
                 ((None, T, T, 1.0), {"stream": 0}), ((None, T, T, -1), {"stream": 0}),
                 ((None, T, T, 2 ** 70), {"stream": 0}), ((None, 2 ** 64, -1, 0), {"stream": 0}),
                 ((None, "x", T, 0), {"stream": 0}), ((None, 1.5, T, 0), {"stream": 0}), ((), {}),
                 ((None, T, T, 0), {}), ((None, T, T, 0), {"stream": None}), ((None, T, T, 0, None), {})]:
        yield add, a, k
    for d in (desc, C.byref(desc), C.pointer(desc), None, latent, bytes(C.sizeof(desc)), bytearray(C.sizeof(desc)),
              np.zeros(C.sizeof(desc), np.uint8), T, 5):
        yield "k3_moe_route", (d, None, None, None, None, 0), {"stream": 0}
    for d in (latent, C.byref(latent), None, desc, bytes(C.sizeof(latent))):
        yield "k3_moe_latent_layer_forward", (d, None, None, 0, None, 0, None, None), {"stream": 0}
    for epsilon in (1e-5, 1, 1e300, float("nan"), np.float32(1), "x"):
        yield "k3_rocm_rms_norm_bf16", (None, None, None, 0, 0, epsilon), {"stream": 0}


def test_bound_and_ctypes_forms_agree(ops):
    from moonshine_b200 import _native
    for name, args, kwargs in forms():
        got = outcome(getattr(ops, name), args, kwargs)
        want = outcome(ops._make(name, *_native.SIGNATURES[name]), args, kwargs)
        assert got == want, (name, args, kwargs)


def test_bound_forms_are_in_use_where_they_are_built(ops):
    from moonshine_b200 import build
    bound = os.path.exists(build.BINDINGS)
    assert (type(ops.k3_rocm_add_bf16).__name__ == "builtin_function_or_method") == bound
    assert type(ops.k3_moe_ep_plan).__name__ == "function"             # not an inner-loop call: stays ctypes


def test_a_broken_binding_file_is_an_error(tmp_path):
    """Of the package's files only a copy is touched."""
    import shutil
    import subprocess
    pkg = tmp_path / "moonshine_b200"
    pkg.mkdir()
    for f in ("__init__.py", "_native.py", "ops.py"):
        shutil.copy(os.path.join(ROOT, "moonshine_b200", f), pkg / f)
    run = lambda: subprocess.run([sys.executable, "-c", "from moonshine_b200 import ops; print(ops.k3_rocm_add_bf16)"],
                                 cwd=tmp_path, capture_output=True, text=True, env={**os.environ, "PYTHONPATH": ""})
    res = run()
    assert res.returncode == 0 and "function" in res.stdout, res.stderr         # no file: ctypes
    (pkg / "_k3ops.so").write_bytes(b"not a library")
    res = run()
    assert res.returncode != 0 and "ImportError" in res.stderr


def test_a_build_without_a_cpp_compiler_leaves_ctypes(tmp_path, monkeypatch, capsys):
    from moonshine_b200 import build
    build.build()
    before = os.stat(build.LIB).st_mtime_ns
    target = tmp_path / "_k3ops.so"
    target.write_bytes(b"stale")
    os.utime(target, (0, 0))
    monkeypatch.setattr(build, "BINDINGS", str(target))
    monkeypatch.setenv("CXX", str(tmp_path / "missing-compiler"))
    assert build.build() == build.LIB
    assert "ctypes" in capsys.readouterr().err
    assert not target.exists() and os.stat(build.LIB).st_mtime_ns == before
