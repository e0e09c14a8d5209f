"""Device arrays of the caller's that are too short for a field are refused,
with the library's host code run over a stand-in for the CUDA runtime: a
conversion kernel never gets one."""
import ctypes as C

import numpy as np
import pytest

import hostlib

L, BS, NS = (8, 8, 8, 8), (4, 4, 4, 4), 4
NB = 8 ** 4 * 96       # bytes of an FP32 field


@pytest.fixture()
def qb():
    qb = hostlib.load()
    qb.geometry(L, BS, qb.even_first_ipt(L))
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.3, 1)
    qb.sw_term()
    qb.nv = qb.set_dfl_parms(BS, NS)
    for l in range(NS):
        qb.dfl_set_basis(l, np.ones(24 * 8 ** 4, np.float32))
    return qb


def _calls(qb):
    qb.vd = np.ones(2 * qb.nv)
    ptr = C.c_void_p * 1
    vds = ptr(qb.vd.ctypes.data)
    f = qb.lib()
    return {"s2vd": lambda p: f.b200_dfl_s2vd_multi(1, ptr(p), vds), "vd2s": lambda p: f.b200_dfl_vd2s_multi(1, vds, ptr(p)),
            "basis": lambda p: f.b200_dfl_set_basis(0, p)}


@pytest.mark.parametrize("call", ["s2vd", "vd2s", "basis"])
@pytest.mark.parametrize("short", [NB // 2, NB - 4])
def test_short_arrays(qb, call, short):
    f, do = qb.lib(), _calls(qb)[call]
    full, p = f.b200_dev_alloc(NB), f.b200_dev_alloc(short)
    assert do(full) == 0
    f.b200_clear_error()
    assert do(p) == -1 and f.b200_last_error()
    f.b200_clear_error()
    assert do(full) == 0 and f.b200_last_error() == b""
    off = f.b200_dev_alloc(NB + 32)       # a part of a longer array
    assert do(off + 32) == 0 and do(off + 48) == -1
