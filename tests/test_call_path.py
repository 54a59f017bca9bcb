"""The Python call path: the compiled extension of this interpreter, its build, and the same calls through ctypes where it cannot be
compiled."""
import os
import subprocess
import sys
import sysconfig

import numpy as np
import pytest

import cann_hccl_b200 as H
from cann_hccl_b200 import _calls, build
from cann_hccl_b200 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_extension_carries_the_interpreters_tag():
    L.lib()
    assert build.fastcall_path().endswith(sysconfig.get_config_var("EXT_SUFFIX")) and os.path.exists(build.fastcall_path())
    assert L.fast.__name__ == "_fastcall"


PROG = """
import sys, warnings
sys.path.insert(0, {root!r})
from cann_hccl_b200 import build
build.LIB = {lib!r}
def everything(*a, **k):
    raise AssertionError("the whole library was to be built")
build.build = everything
if {broken!r}:
    build.sysconfig = type("S", (), {{"get_config_var": staticmethod(lambda n: ".none.so"), "get_paths": staticmethod(lambda: {{"include": "/nonexistent"}})}})
import numpy as np
import cann_hccl_b200 as H
from cann_hccl_b200 import _lib as L
with warnings.catch_warnings(record=True) as w:
    warnings.simplefilter("always")
    c = H.Communicator.init_local(2, device=False)
x, y = [np.ones(5, np.float32) for _ in range(2)], [np.zeros(5, np.float32) for _ in range(2)]
c.all_reduce(x, y)
assert (y[1] == 2).all()
print(type(L.fast).__name__, len([m for m in w if "ctypes" in str(m.message)]))
"""


@pytest.mark.parametrize("broken,want", [(False, "module 0"), (True, "Calls 1")])
def test_missing_extension_is_compiled_alone_or_done_without(tmp_path, broken, want):
    """The library is there, the extension is not: only the extension is compiled; without Python's headers calls go through ctypes."""
    r = subprocess.run([sys.executable, "-c", PROG.format(root=ROOT, lib=str(tmp_path), broken=broken)], capture_output=True, text=True,
                       env=dict(os.environ, HCCL_B200_LIB=build.lib_path()), timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == want, r.stdout + r.stderr
    assert len(os.listdir(tmp_path)) == (0 if broken else 1)


@pytest.fixture(params=["extension", "ctypes"])
def path(request, monkeypatch):
    L.lib()
    if request.param == "ctypes":
        calls = _calls.Calls(L.lib())
        from cann_hccl_b200.utils.dtypes import dtype_table
        calls.setup(dtype_table(False), None, None)
        monkeypatch.setattr(L, "fast", calls)
    return L.fast


def test_both_forms_make_the_same_calls(path):
    p, n = 3, 7
    c = H.Communicator.init_local(p, device=False)
    x = [np.arange(p * n, dtype=np.float32) + 100 * r for r in range(p)]
    total = sum(x)
    out = [np.zeros(p * n, np.float32) for _ in range(p)]
    c.all_reduce(x, out)
    assert all(np.array_equal(o, total) for o in out)
    part = [np.zeros(n, np.float32) for _ in range(p)]
    c.reduce_scatter(tuple(x), part)
    assert np.array_equal(np.concatenate(part), total)
    c.all_gather(part, out)
    assert all(np.array_equal(o, total) for o in out)
    c.all_to_all(x, out)
    assert np.array_equal(out[1], np.concatenate([y[n:2 * n] for y in x]))
    c.barrier()
    counts, displs = [n, 0, 2], [0, n, n + 3]
    c.all_gather_v([y[:k] if k else None for y, k in zip(x, counts)], out, counts, displs)
    assert all(np.array_equal(o[:n], x[0][:n]) and np.array_equal(o[n + 3:n + 5], x[2][:2]) for o in out)
    sc = np.full((p, p), n, np.uint64)
    sd = np.tile(np.arange(p, dtype=np.uint64) * np.uint64(n), (p, 1))
    c.all_to_all_v(x, sc, sd, out, sc, sd)
    assert np.array_equal(out[2], np.concatenate([y[2 * n:] for y in x]))
    one = H.Communicator.init_local(1, device=False)
    got = np.zeros(n, np.float32)
    one.all_reduce(x[0][:n].copy(), got)
    assert np.array_equal(got, x[0][:n])
    for bad, error in (([x[0]], AssertionError), ([x[0], x[1], object()], AttributeError)):
        with pytest.raises(error):
            c.collective(L.ALLREDUCE, bad, out, n, L.FP32)
    with pytest.raises(KeyError):
        c.all_reduce([y.astype(np.complex64) for y in x], out)
    for good, bad in (([x[0]], [None]), ([x[0]], None)):
        with pytest.raises(TypeError):
            path.moe_dispatch(0, 1, 0, good, bad, 0)
        with pytest.raises(TypeError):
            path.moe_combine(0, 1, 0, 0, good, good, bad, 0)
    assert path.moe_dispatch(0, 1, 0, [x[0]], [x[0]], 0) == path.moe_combine(0, 1, 0, 0, [x[0]], [x[0]], [x[0]], 0) == L.E_PTR
    assert c.destroy() == one.destroy() == L.SUCCESS
