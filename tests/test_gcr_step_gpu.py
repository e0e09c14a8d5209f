"""Reductions finished by the last block of their own launch, and the GCR step
that keeps its products on the device: lattices from less than one block of
threads to more blocks than the grid's limit, Krylov spaces of one vector
(no product), two, and more than a solve needs; residuals recomputed with the
CPU restatement of Dw_dble (oracle/qcd_oracle.c)."""
import numpy as np
import pytest

import openqcd_b200 as qb
import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [((4, 4, 4, 4), (2, 2, 2, 2)), ((12, 4, 4, 4), (6, 2, 2, 2)), ((8, 8, 8, 8), (4, 4, 4, 4)),
          ((32, 16, 16, 16), (4, 4, 4, 4))]


@pytest.mark.parametrize("L,bs", SHAPES, ids=["x".join(map(str, l)) for l, _ in SHAPES])
def test_reductions(L, bs):
    ipt = qb.even_first_ipt(L)
    qb.geometry(L, bs, ipt)
    x = np.random.default_rng(1).standard_normal(24 * ipt.size)
    for prec, tol in ((64, 1e-15), (32, 1e-7)):
        # FP64: double-double over the blocks, sums of at most 3e4 squares in
        # double within one (random roundings of 1e-16 / sqrt(3e4) each);
        # FP32: the four squares of an element are summed in FP32
        f = qb.DevField(prec).from_ref(x)
        q = x.astype(np.float32).astype(np.float64) if prec == 32 else x
        want = float(np.sum(q.astype(np.longdouble) ** 2))
        got = [f.norm2() for _ in range(3)]
        assert got[0] == got[1] == got[2]          # the same bits every time
        assert abs(got[0] - want) <= tol * want


@pytest.mark.parametrize("nkv", [1, 2, 16])
@pytest.mark.parametrize("L,bs", SHAPES[1:3], ids=["x".join(map(str, l)) for l, _ in SHAPES[1:3]])
def test_gcr_step(L, bs, nkv):
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.4, 99)
    assert qb.sw_term() == 0
    qb.set_sap_parms(bs, 1, 4, 3)
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = O.pauli_ref2lex(qb.download_swd(V), ipt)
    eta = np.random.default_rng(2).standard_normal(24 * V)
    psi, rho, ifail, status = qb.sap_gcr(nkv, 256, 0, 1e-10, 0.05, eta)
    r = O.spinor_ref2lex(eta, ipt) - O.dirac_dble(L, 0, 0.05, 0, U, sw, None, O.spinor_ref2lex(psi, ipt))
    assert ifail == 0 and 0 < status < 100
    assert np.linalg.norm(r) <= 1.0001e-10 * np.linalg.norm(eta)
    assert abs(rho - np.linalg.norm(r)) <= 1e-3 * rho
    z = qb.sap_gcr(nkv, 256, 0, 1e-10, 0.05, np.zeros_like(eta))     # no step at all
    assert z[2] == 0 and z[3] == 0 and not z[0].any()
