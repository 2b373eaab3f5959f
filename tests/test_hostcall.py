"""Entry points called without ctypes: argument conversion, and what only ctypes converts."""
import ctypes as C

import numpy as np
import pytest

from dfccl_b200 import native as nv


def test_arguments():
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


def test_without_the_extension(monkeypatch):
    """No compiler and no built extension: the same calls through ctypes."""
    monkeypatch.setattr(nv, "_hostcall", lambda: None)
    monkeypatch.setattr(nv, "_entries", {})
    test_submissions_take_what_ctypes_takes()
