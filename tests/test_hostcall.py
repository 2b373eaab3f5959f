"""Entry points called without ctypes: argument conversion, and what only ctypes converts."""
import ctypes as C
import os
import subprocess
import warnings

import numpy as np
import pytest

from dfccl_b200 import _build
from dfccl_b200 import native as nv


def test_arguments():
    if nv._hostcall() is None:
        pytest.skip("no compiler or no interpreter headers: the entry points go through ctypes")
    f = nv.entry("dfcclGetBackend")
    v = C.c_int(-1)
    assert f(C.addressof(v)) == nv.SUCCESS and v.value in (nv.BACKEND_CUDA, nv.BACKEND_HOST)
    assert f(None) != nv.SUCCESS and nv.entry("dfcclGetBackend") is f
    g = nv.entry("dfcclGemmReserveSms")
    assert g(-1) == nv.INVALID_ARGUMENT and g(np.int64(129)) == nv.INVALID_ARGUMENT        # negative; anything with an index
    for bad in (1.5, "x", C.c_void_p(0)):
        with pytest.raises(TypeError):
            g(bad)
    with pytest.raises(TypeError):
        f(*range(15))


def test_submissions_take_what_ctypes_takes():
    old = nv.get_backend()
    nv.set_backend("host")
    try:
        (comm,) = nv.Comm.init_loopback(1)
        ctx = nv.RankCtx(0)
        ctx.prepare(0, comm, nv.ALLREDUCE, 64, nv.FLOAT32)
        ctx.finalize()
        a, b = np.arange(64, dtype=np.float32), np.zeros(64, np.float32)
        for send, recv in ((a.ctypes.data, b.ctypes.data), (C.c_void_p(a.ctypes.data), C.c_void_p(b.ctypes.data))):
            b[:] = 0
            ctx.run(0, send, recv)
            assert ctx.wait(0, 30000) == nv.SUCCESS
            assert (a == b).all()
        with pytest.raises(nv.DfcclError):
            ctx.run(0, None, b.ctypes.data)
        ctx.destroy()
        comm.destroy()
    finally:
        nv.set_backend(old)


@pytest.mark.parametrize("gcc", ["missing", "failing"])
def test_without_the_extension(monkeypatch, tmp_path, gcc):
    """No compiler, or none that finds the interpreter's headers, and no built extension: the library is compiled and linked
    all the same, and the same calls go through ctypes."""
    obj = tmp_path / "x.o"
    obj.touch()

    def run(cmd, **kw):
        if cmd[0] == _build.nvcc():
            (tmp_path / "libdfccl.so").touch()
        elif gcc == "missing":
            raise FileNotFoundError(cmd[0])
        return subprocess.CompletedProcess(cmd, 0 if cmd[0] == _build.nvcc() else 1, "", "no such header")

    monkeypatch.setattr(_build, "LIB", tmp_path / "libdfccl.so")
    monkeypatch.setattr(_build, "LIBDIR", tmp_path)
    monkeypatch.setattr(_build, "HOSTCALL", tmp_path / "dfccl_hostcall.so")
    monkeypatch.setattr(_build, "_compile", lambda *a: obj)
    monkeypatch.setattr(_build.subprocess, "run", run)
    monkeypatch.setattr(nv, "_hostcall", nv._hostcall.__wrapped__)
    monkeypatch.setattr(nv, "_entries", {})
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert _build.build().exists()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        assert nv._hostcall() is None
        test_submissions_take_what_ctypes_takes()


def test_a_stale_extension_is_built_again(monkeypatch, tmp_path):
    if nv._hostcall() is None:
        pytest.skip("no compiler or no interpreter headers")
    so = tmp_path / "dfccl_hostcall.so"
    monkeypatch.setattr(_build, "HOSTCALL", so)
    monkeypatch.setattr(_build, "LIBDIR", tmp_path)
    so.write_bytes(b"of another time")
    os.utime(so, (1, 1))
    assert nv._hostcall.__wrapped__() is not None
    assert so.stat().st_size > 1000
