"""The stand-in for the reference on machines without its sources
(oracle/restated.py): its storage orders against each other, the distribution
of its links, and the smoke check's choice of it."""
import sys

import numpy as np
import pytest

import oracle as O
import reflib
import restated


@pytest.fixture(scope="module")
def r():
    r = restated.Restated((16, 8, 8, 8))
    r.init(csw=1.7, m0=-0.05)
    r.gen_links(0.3, 5)
    assert r.sw_term() == 0
    return r


def test_storage_orders(r):
    ipt = r.ipt()
    x = np.indices(r.L).reshape(4, -1)
    assert np.array_equal(np.sort(ipt), np.arange(r.vol))
    assert np.array_equal(ipt >= r.vol // 2, (x.sum(axis=0) & 1).astype(bool))
    assert np.array_equal(O.links_ref2lex(r.ud(), ipt, r.L), r.U)
    U = r.U.copy()
    r.set_ud(r.ud())
    assert np.array_equal(r.U, U)


def test_links(r):
    U = r.U.view(np.complex128).reshape(-1, 3, 3)
    assert np.abs(U @ U.conj().swapaxes(-1, -2) - np.eye(3)).max() <= 1e-14
    # tr X^2 has the mean -4 of random_alg's normalisation (eight components
    # with tr T^a T^b = -delta_ab / 2, each of variance 1), so Re tr U = 3 -
    # 2 eps^2 up to O(eps^4): checked by a field with a small eps
    r.gen_links(0.05, 7)
    spatial = r.U.view(np.complex128).reshape(-1, 4, 3, 3)[:, 1:]
    s = (3.0 - np.einsum("...ii->...", spatial).real) / 0.05 ** 2
    assert abs(s.mean() - 2.0) <= 5.0 * s.std() / np.sqrt(s.size) + 0.01
    r.gen_links(0.3, 5)


def test_inverted_sw_term(r):
    sw = O.pauli_ref2lex(r.swd(), r.ipt()).reshape(-1, 36)
    odd = np.repeat(np.indices(r.L).sum(axis=0).reshape(-1) & 1, 2).astype(bool)
    for which in (1, 2, 3):
        assert r.sw_term(which) == 0
        got = O.pauli_ref2lex(r.swd(), r.ipt()).reshape(-1, 36)
        inv = np.where(odd, which & 2, which & 1) != 0
        assert np.array_equal(got[~inv], sw[~inv])
        for i in np.flatnonzero(inv)[:20]:
            assert np.allclose(O.inv_pauli(0.0, sw[i])[0], got[i], rtol=1e-12, atol=0)
    r.sw_term(0)


def test_sums_and_matrices(r):
    s, t = r.random_sd(1), r.random_sd(2)
    z = r.spinor_prod_dble(s, t)
    assert abs(z[0] + 1j * z[2] - np.vdot(s.view(complex), t.view(complex))) <= 1e-12 * abs(np.vdot(s, s))
    # Dwee + Dwoo on all sites is the SW term
    d = r.dirac_dble(1, 0.2, s)
    h = 12 * r.vol
    assert np.allclose(r.apply_sw_dble(r.vol, 0.2, r.swd(), s)[:h], d[:h], rtol=0, atol=1e-13)
    w = r.apply_sw_dble(r.vol, 0.2, r.swd(), s)
    assert np.allclose(r.apply_swinv_dble(r.vol, 0.2, r.swd(), w)[0], s, rtol=0, atol=1e-12)
    # 1 - <Re tr U_p> / 3 = 4 x 2 eps^2 / 3 up to O(eps^4) for independent links
    assert abs(1.0 - r.plaq_sum() / (18 * r.vol) - 8 * 0.3 ** 2 / 3) <= 0.06


def test_phase_angles():
    """the SW term and the plaquette do not see them, the links do"""
    a, b = (restated.Restated((4, 4, 4, 4)) for _ in range(2))
    for x, theta in ((a, None), (b, (0.5, -0.8, 1.3))):
        x.init(csw=1.5, m0=0.0, theta=theta)
        x.gen_links(0.3, 5)
        x.sw_term()
    assert np.abs(a.U - b.U).max() > 0.1
    assert np.abs(a.sw - b.sw).max() <= 1e-13 and abs(a.plaq_sum() - b.plaq_sum()) <= 1e-10


def test_solver(r):
    r.set_sap_parms((4, 4, 4, 4), 1, 4, 3)
    eta = r.random_sd(3)
    psi, rho, ifail, status = r.sap_gcr(16, 64, 0, 1e-6, 0.0, eta)
    assert ifail == 0 and np.linalg.norm(eta - r.dirac_dble(0, 0.0, psi)) <= 1.1e-6 * np.linalg.norm(eta)


def test_what_it_does_not_cover(r):
    with pytest.raises(NotImplementedError):
        r.tmcg(1)
    with pytest.raises(NotImplementedError):
        r.init(isw=1)


def test_deflation():
    r = restated.Restated((8, 8, 8, 8))
    r.init(csw=1.5, m0=-0.2)
    r.gen_links(0.4, 5)
    r.sw_term()
    r.set_sap_parms((4, 4, 4, 4), 1, 4, 5)
    nv = r.dfl_init((4, 4, 4, 4), 4)
    assert nv == 64 and r.dfl_modes(7)[0] == 0
    g = np.random.default_rng(1)
    v = g.standard_normal(2 * nv)
    assert np.abs(r.dfl_s2vd(r.dfl_vd2s(v)) - v).max() <= 1e-5          # an orthonormal block basis
    # the little operator through fields, and the even-odd pieces through it
    s = r._prolong(v.view(complex), np.float64)
    assert np.allclose(r.little(0, 0.03, v)[0], r._restrict(r.dirac_dble(0, 0.03, s)).view(float), rtol=0, atol=1e-12)
    w = r.little(5, 0.03, v, r.little(0, 0.03, v)[0])[0][:nv]           # Aee v_e
    assert np.allclose(r.little(2, 0.03, np.concatenate([w, v[nv:]]))[0][:nv], v[:nv], rtol=0, atol=1e-10)
    x = r.little(1, 0.03, v)[0][:nv]
    y = r.little(3, 0.03, r.little(4, 0.03, v)[0])[0]
    z = r.little(2, 0.03, r.little(5, 0.03, y)[0])[0][:nv]              # -Aee^-1 Aeo Aoo^-1 Aoe v_e
    assert np.allclose(x, v[:nv] + z, rtol=0, atol=1e-12)
    assert np.allclose(r.little(0, 0.03, r.ltl_gcr(0.03, v)[0])[0], v, rtol=0, atol=1e-10)
    eta = r.random_sd(3)
    psi, rho, ifail, status = r.dfl_sap_gcr(16, 64, 0, 1e-10, 0.0, eta)
    assert ifail == 0 and status[0] < r.sap_gcr(16, 64, 0, 1e-10, 0.0, eta)[3] + 2
    assert np.linalg.norm(eta - r.dirac_dble(0, 0.0, psi)) <= 1.0001e-10 * np.linalg.norm(eta)


class _Device:
    """the calls of the binding that set-up and smoke check make, answered by
    the restatement"""

    def __init__(self, ref):
        self.ref = ref

    def __getattr__(self, name):
        return lambda *a, **k: 0

    def dirac_ref(self, op, prec, mu, s):
        return self.ref.dirac_dble(0, mu, s)

    def sap_gcr(self, *args):
        return self.ref.sap_gcr(*args)


def test_without_the_reference(monkeypatch):
    """the parity tests' set-up and the smoke check run where the reference's
    library is absent"""
    import __graft_entry__ as g
    import helpers
    ref = restated.Restated((8, 8, 8, 8))
    monkeypatch.setattr(reflib, "ensure_built", lambda *a, **k: False)
    monkeypatch.setattr(restated, "Restated", lambda L: ref)
    monkeypatch.setattr(helpers, "qb", _Device(ref))
    st = helpers.Setup((8, 8, 8, 8))
    assert st.vol == 4096 and st.ud.size == 4 * 4096 * 18 and st.source(1).size == 24 * 4096
    with pytest.raises(pytest.skip.Exception):
        st.ref.tmcg(1)
    ref.init(csw=1.5, m0=0.0)
    ref.gen_links(0.4, 1234)
    ref.sw_term()
    ref.set_sap_parms((4, 4, 4, 4), 1, 4, 5)
    monkeypatch.setitem(sys.modules, "openqcd_b200", _Device(ref))
    g.smoke()
