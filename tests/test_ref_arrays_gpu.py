"""Conversions between the caller's arrays and the device layout: lattices whose
sites do not fill the conversion kernels' CTAs, both precisions, and the
deflation transfers on host arrays, on device arrays (converted in place) and
on device arrays that are not aligned for 16-byte accesses (staged): the same
bits from all of them."""
import ctypes as C

import numpy as np
import pytest

import openqcd_b200 as qb

pytestmark = pytest.mark.gpu

SHAPES = [((4, 4, 4, 4), (2, 2, 2, 2)), ((12, 4, 4, 4), (6, 2, 2, 2)), ((8, 12, 8, 12), (4, 6, 4, 6))]


@pytest.mark.parametrize("L,bs", SHAPES, ids=["x".join(map(str, l)) for l, _ in SHAPES])
def test_round_trip(L, bs):
    rng = np.random.default_rng(1)
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    for par in (slice(0, V // 2), slice(V // 2, V)):        # any order within a parity half
        q = np.nonzero((ipt >= par.start) & (ipt < par.stop))[0]
        ipt[q] = rng.permutation(np.arange(par.start, par.stop, dtype=np.int32))
    qb.geometry(L, bs, ipt)
    for prec, dt in ((64, np.float64), (32, np.float32)):
        x = rng.standard_normal(24 * V).astype(dt)
        f = qb.DevField(prec).from_ref(x)
        assert np.array_equal(f.to_ref(V), x)
        y, lex = (3, 1, 0, 1), np.ravel_multi_index((3, 1, 0, 1), L)
        p = qb.DevField(prec).point(y, 2, 1).to_ref(V).reshape(V, 24)
        assert np.count_nonzero(p) == 1 and p[ipt[lex], 2 * (3 * 2 + 1)] == 1.0


def _device(a, off):
    n = a.nbytes
    p = qb.lib().b200_dev_alloc(n + 16)
    qb.check(qb.lib().b200_memcpy(p + off, a.ctypes.data, n))
    return p


def test_transfers_on_device_arrays():
    L, bs, ns, nr = (8, 8, 8, 12), (4, 4, 4, 6), 4, 3
    qb.geometry(L, bs, qb.even_first_ipt(L))
    V = int(np.prod(L))
    rng = np.random.default_rng(2)
    nv = qb.set_dfl_parms(bs, ns)
    qb.dfl_subspace([rng.standard_normal(24 * V).astype(np.float32) for _ in range(ns)])
    fs = [rng.standard_normal(24 * V).astype(np.float32) for _ in range(nr)]
    vd = qb.dfl_s2vd_multi(fs, nv)
    out = qb.dfl_vd2s_multi(vd, V)
    for off in (0, 8):
        pf = [_device(f, off) for f in fs]
        po = [_device(np.zeros_like(f), off) for f in fs]
        v2 = [np.zeros_like(v) for v in vd]
        qb.check(qb.lib().b200_dfl_s2vd_multi(nr, (C.c_void_p * nr)(*[p + off for p in pf]),
                                              (C.c_void_p * nr)(*[v.ctypes.data for v in v2])))
        qb.check(qb.lib().b200_dfl_vd2s_multi(nr, (C.c_void_p * nr)(*[v.ctypes.data for v in v2]),
                                              (C.c_void_p * nr)(*[p + off for p in po])))
        for k in range(nr):
            o = np.zeros_like(fs[k])
            qb.check(qb.lib().b200_memcpy(o.ctypes.data, po[k] + off, o.nbytes))
            assert np.array_equal(v2[k], vd[k]) and np.array_equal(o, out[k])
            qb.lib().b200_dev_free(pf[k])
            qb.lib().b200_dev_free(po[k])
