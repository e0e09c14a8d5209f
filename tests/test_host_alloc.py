"""Workspaces when memory runs out, with the library's host code run over a
stand-in for the CUDA runtime that lets a chosen allocation fail: the call
reports it, leaves nothing half made, and the next call starts afresh, without
a null pointer among its kernels' arguments."""
import numpy as np
import pytest

import hostlib

L, BS, NS = (8, 8, 8, 8), (4, 4, 4, 4), 4
V = 8 ** 4


@pytest.fixture()
def qb():
    qb = hostlib.load()
    qb.geometry(L, BS, qb.even_first_ipt(L))
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.3, 1)
    qb.sw_term()
    qb.set_sap_parms(BS, 1, 4, 2)
    return qb


@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_reduction_buffers(qb, n):
    f = qb.lib()
    x = qb.DevField(32)
    for arg, k in ((2, 2), (3, 1)):             # Fin {part, cnt}, out
        f.fake_watch(b"k_norm2", arg, k)
    live, launches = f.fake_live(), f.fake_launches()
    f.fake_fail_at(n)
    f.b200_clear_error()
    x.norm2()
    assert b"out of memory" in f.b200_last_error()
    assert f.fake_live() == live and f.fake_launches() == launches
    f.fake_fail_at(0)
    f.b200_clear_error()
    x.norm2()
    assert f.b200_last_error() == b"" and f.fake_launches() == launches + 1
    assert f.fake_null_args() == 0 and f.fake_live() == live + 4
