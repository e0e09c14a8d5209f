"""The operators with two lanes per site on blocks whose sites do not fill a
warp's 16 pairs: every operator and the host pipeline's block lists in both
precisions, with 12-real and 18-real links in FP32 and the residual-update
form, against the CPU restatement (oracle/qcd_oracle.c, modules/dirac/Dw.c:973,
Dw_dble.c:1377).  FP64 launches of three and of four CTAs per SM, in place, and
Dwhat_dble on its half-field scratch; Dwoe and Dweo in FP32 on lattices with one
lane per site in their two forms."""
import numpy as np
import pytest

import openqcd_b200 as qb
import oracle as O
from helpers import OPS, site_rel_err

pytestmark = pytest.mark.gpu

MU = 0.07
TOL = 2e-6      # FP32 rounding of one operator, the bar of the other parity tests
TOL64 = 1e-13

SHAPES = [((4, 4, 4, 4), (2, 2, 2, 2)), ((8, 4, 4, 12), (4, 2, 2, 6)), ((8, 12, 8, 8), (4, 6, 4, 4)),
          ((12, 12, 12, 12), (6, 6, 6, 6))]


@pytest.mark.parametrize("L,bs", SHAPES, ids=["x".join(map(str, b)) for _, b in SHAPES])
@pytest.mark.parametrize("eoflg", [0, 1])
def test_fp32_operators(L, bs, eoflg):
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, 0.0, eoflg)
    qb.random_ud(0.4, 99)
    assert qb.sw_term() == 0
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = [O.pauli_ref2lex(qb.download_swd(V, k), ipt) for k in (0, 1)]
    g = np.random.default_rng(3)
    s, r0 = (g.standard_normal(24 * V).astype(np.float32) for _ in range(2))
    ref = {op: O.spinor_lex2ref(O.dirac(L, k, MU, eoflg, U, sw[0], sw[1], O.spinor_ref2lex(s, ipt),
                                        O.spinor_ref2lex(r0, ipt)), ipt) for k, op in enumerate(OPS)}
    try:
        for l12 in (1, 0):
            qb.set_sap_link12(l12)
            assert not l12 or qb.links12_active()
            for op in OPS:
                assert site_rel_err(qb.dirac_ref(op, 32, MU, s, r0), ref[op], V) <= TOL, (op, l12)
            S, B, R = qb.DevField(32).from_ref(s), qb.DevField(32).from_ref(r0), qb.DevField(32)
            qb.dev_dirac_multi(MU, [S], [R], [B])
            assert site_rel_err(R.to_ref(V), r0 - ref["Dw"], V) <= TOL
            hs, hr = qb.HostArray(24 * V, np.float32), qb.HostArray(24 * V, np.float32)
            hs.a[:] = s
            qb.lib().Dw(MU, hs.ptr, hr.ptr)
            assert np.array_equal(np.array(hr.a), qb.dirac_ref("Dw", 32, MU, s))
            hs.free()
            hr.free()
    finally:
        qb.set_sap_link12(1)


# up to 444 CTAs of one lane per site, and more
@pytest.mark.parametrize("L,bs", [((16, 12, 16, 12), (4, 6, 4, 6)), ((24, 24, 24, 12), (6, 6, 6, 6))],
                         ids=["4x6x4x6", "6x6x6x6"])
def test_fp32_hops_large(L, bs):
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.4, 99)
    assert qb.sw_term() == 0
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = O.pauli_ref2lex(qb.download_swd(V), ipt)
    g = np.random.default_rng(3)
    s, r0 = (g.standard_normal(24 * V).astype(np.float32) for _ in range(2))
    try:
        for op in ("Dwoe", "Dweo"):
            ref = O.spinor_lex2ref(O.dirac(L, OPS.index(op), MU, 0, U, sw, sw, O.spinor_ref2lex(s, ipt),
                                           O.spinor_ref2lex(r0, ipt)), ipt)
            for l12 in (1, 0):
                qb.set_sap_link12(l12)
                assert site_rel_err(qb.dirac_ref(op, 32, MU, s, r0), ref, V) <= TOL, (op, l12)
        # the operator as a whole, which has two lanes per site, in its pieces
        qb.set_sap_link12(1)
        z = np.zeros_like(s)
        even = qb.dirac_ref("Dweo", 32, MU, -s, qb.dirac_ref("Dwee", 32, MU, s, z))
        odd = qb.dirac_ref("Dwoo", 32, MU, s, z) + qb.dirac_ref("Dwoe", 32, MU, s, z)
        h = 12 * V
        assert site_rel_err(np.concatenate([even[:h], odd[h:]]), qb.dirac_ref("Dw", 32, MU, s), V) <= TOL
    finally:
        qb.set_sap_link12(1)


# CTAs of a launch on one parity: 4 and 32, 164 and (four per SM) 512
@pytest.mark.parametrize("L,bs", [SHAPES[0], SHAPES[1], SHAPES[3], ((16, 16, 16, 16), (4, 4, 4, 4))],
                         ids=["2x2x2x2", "4x2x2x6", "6x6x6x6", "16^4"])
@pytest.mark.parametrize("eoflg", [0, 1])
def test_fp64_operators(L, bs, eoflg):
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, 0.0, eoflg)
    qb.random_ud(0.4, 99)
    assert qb.sw_term() == 0
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = [O.pauli_ref2lex(qb.download_swd(V, k), ipt) for k in (0, 1)]
    g = np.random.default_rng(3)
    s, r0 = (g.standard_normal(24 * V) for _ in range(2))
    ref = {op: O.spinor_lex2ref(O.dirac_dble(L, k, MU, eoflg, U, sw[0], sw[1], O.spinor_ref2lex(s, ipt),
                                             O.spinor_ref2lex(r0, ipt)), ipt) for k, op in enumerate(OPS)}
    for op in OPS:
        assert site_rel_err(qb.dirac_ref(op, 64, MU, s, r0), ref[op], V) <= TOL64, op
    # in place: Dwee and Dwoo change one parity, Dwhat reads the even sites and writes them
    for op in ("Dwee", "Dwoo", "Dwhat"):
        F = qb.DevField(64).from_ref(s)
        qb.dev_dirac(op, MU, F, F)
        half = slice(12 * V, None) if op == "Dwoo" else slice(0, 12 * V)
        assert site_rel_err(F.to_ref(V)[half], ref[op][half], V // 2) <= TOL64, op
    S, R = qb.DevField(64).from_ref(s), qb.DevField(64).from_ref(r0)
    qb.check(qb.lib().b200_dev_Dwhat_dble_noalloc(MU, S.ptr, R.ptr))
    assert np.array_equal(R.to_ref(V)[:12 * V], qb.dirac_ref("Dwhat", 64, MU, s, r0)[:12 * V])
    hs, hr = qb.HostArray(24 * V), qb.HostArray(24 * V)
    hs.a[:] = s
    qb.lib().Dw_dble(MU, hs.ptr, hr.ptr)
    assert np.array_equal(np.array(hr.a), qb.dirac_ref("Dw", 64, MU, s))
    hs.free()
    hr.free()
