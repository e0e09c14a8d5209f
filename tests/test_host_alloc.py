"""Workspaces when memory runs out, with the library's host code run over a
stand-in for the CUDA runtime that lets a chosen allocation fail: the call
reports it, leaves nothing half made, and the next call starts afresh, without
a null pointer among its kernels' arguments."""
import ctypes as C

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


def _deflated(qb):
    nv = qb.set_dfl_parms(BS, NS)
    qb.set_dfl_pro_parms(2, 2, 1e-2, 2, 1e-2)
    for l in range(NS):
        qb.dfl_set_basis(l, np.ones(24 * V, np.float32))
    return nv


def _every_failure(prepare, call, watched):
    """call(qb, state) with its n-th allocation failing, for every n, and again
    without a failure, in a library of its own each time"""
    n, seen = 1, 0
    while True:
        qb = hostlib.load()
        qb.geometry(L, BS, qb.even_first_ipt(L))
        qb.set_parms(1.5, 0.0, 0)
        qb.random_ud(0.3, 1)
        qb.sw_term()
        qb.set_sap_parms(BS, 1, 4, 2)
        state = prepare(qb)
        f = qb.lib()
        for w in watched:
            f.fake_watch(*w)
        f.fake_fail_at(n)
        f.b200_clear_error()
        try:
            call(qb, state)
            error = f.b200_last_error().decode()
        except qb.B200Error as e:
            error = str(e)
        if "memory" in error or "allocation" in error:
            seen += 1
        elif f.fake_allocs() < n:
            assert not error or "unsafe" in error
            return n - 1, seen      # the call makes no more than that
        f.fake_fail_at(0)
        f.b200_clear_error()
        try:
            call(qb, state)
        except qb.B200Error as e:       # without its kernels' results a call may find its data degenerate
            assert "unsafe" in str(e)
        assert f.fake_null_args() == 0 and f.fake_bad_frees() == 0, n
        n += 1


def test_deflation_parameters():
    def call(qb, _):
        try:
            assert qb.set_dfl_parms(BS, NS) > 0
        except qb.B200Error:
            with pytest.raises(qb.B200Error, match="not set"):     # nothing works on what is left of it
                qb.dfl_s2vd(np.ones(24 * V, np.float32), 1)
            raise qb.B200Error("out of memory")
    total, seen = _every_failure(lambda qb: None, call, [])
    assert seen == total >= 13


@pytest.mark.parametrize("what", ["dfl_modes", "dfl_sap_gcr", "ltl_gcr", "ltl_gcr_ref", "batch", "network"])
def test_solver_workspaces(what):
    def prepare(qb):
        nv = _deflated(qb)
        qb.set_dfl_gen_parms(0.125, 0.0, 4, 4, 2)
        E, P = ([qb.DevField(64) for _ in range(2)] for _ in range(2))
        qb.dev_gcr_batch(2, 2, 0, 1e-10, [0.0] * 2, E, P)      # what a batch without deflation needs is there
        if what == "ltl_gcr_ref":
            qb.dfl_subspace([np.ones(24 * V, np.float32)] * NS)
            qb.set_ltl_solver(1)
        return nv, E, P, [qb.DevField(32) for _ in range(2)]

    def call(qb, s):
        nv, E, P, R = s
        if what == "dfl_modes":
            qb.dfl_modes(1)
        elif what == "dfl_sap_gcr":
            qb.dev_dfl_sap_gcr(2, 2, 0, 1e-10, 0.0, E[0], P[0])
        elif what == "batch":
            qb.dev_gcr_batch(2, 2, 0, 1e-10, [0.0] * 2, E, P, dfl=True)
        elif what == "network":
            qb.net_init(1, 0.25)
            qb.net_grad(*R)
        else:
            qb.ltl_gcr(0.0, np.ones(2 * nv))
    # the tables, partial sums, counters and results of the little solvers' sums
    watched = [(b"k_bmdot", k, 1) for k in (0, 3, 8, 9, 10)] + [(b"k_bcopy", 0, 1), (b"k_mdot", 0, 1), (b"k_cinv", 3, 1)]
    total, seen = _every_failure(prepare, call, watched)
    assert total >= 4 and seen >= total - 1      # the SAP input field has a stand-in


def test_subspace_generation_restores_the_mass():
    """the generation mass and the eo flag do not outlive a call that failed"""
    def prepare(qb):
        _deflated(qb)
        qb.set_dfl_gen_parms(0.11, 0.02, 4, 4, 2)
        qb.dirac_ref("Dw", 64, 0.0, np.ones(24 * V))
        return qb.lib().fake_launched

    def call(qb, launched):
        before = launched(b"k_sw_shift")
        try:
            qb.dfl_modes(1)
        finally:
            shifts = launched(b"k_sw_shift") - before
            try:
                qb.dirac_ref("Dw", 64, 0.0, np.ones(24 * V))
                assert shifts % 2 == 0              # there and back
            except qb.B200Error as e:
                assert "SW field" in str(e)         # or the SW term is gone, and said to be
                qb.sw_term()
    total, seen = _every_failure(prepare, call, [])
    assert seen == total >= 20


def test_larger_lattice_after_smaller():
    """what a call keeps is sized anew with the geometry: fields in copies,
    conversions, block solves and updates hold the new lattice"""
    qb = hostlib.load()
    qb.lib().fake_watch_room.argtypes = [C.c_char_p, C.c_int, C.c_size_t]
    for L in ((8, 8, 8, 8), (16, 8, 8, 8)):
        V = int(np.prod(L))
        qb.geometry(L, BS, qb.even_first_ipt(L))
        qb.lib().fake_unwatch()
        for kernel, args, site in ((b"k_copy_dd", (1, 2), 192), (b"k_copy_ff", (1, 2), 96), (b"k_sap_out", (1, 2, 3), 96),
                                   (b"k_fupd", (0, 1), 96), (b"k_scale_d", (1,), 192)):
            for a in args:
                qb.lib().fake_watch_room(kernel, a, V * site)
        qb.set_parms(1.5, 0.0, 0)
        qb.random_ud(0.3, 1)
        qb.sw_term()
        qb.set_sap_parms(BS, 1, 4, 2)
        s = np.ones(24 * V)
        qb.dirac_ref("Dwhat", 64, 0.1, s)
        qb.sap_ref(0.1, 1, 4, s.astype(np.float32), s.astype(np.float32))
        qb.sap_gcr(2, 2, 0, 1e-10, 0.0, s)
        qb.tmcg(128, 0, 1e-8, 0.1, s)
        nv = qb.set_dfl_parms(BS, NS)
        qb.set_dfl_pro_parms(2, 2, 1e-2, 2, 1e-2)
        for l in range(NS):
            qb.dfl_set_basis(l, np.ones(24 * V, np.float32))
        qb.dfl_s2vd_multi([s.astype(np.float32)] * 3, nv)
        E, P = ([qb.DevField(64) for _ in range(3)] for _ in range(2))
        for dfl in (False, True):
            qb.dev_gcr_batch(2, 2, 0, 1e-10, [0.0] * 3, E, P, dfl=dfl)
        assert qb.lib().b200_last_error() == b"" and qb.lib().fake_bad_frees() == 0
        assert qb.lib().fake_short_args() == 0
