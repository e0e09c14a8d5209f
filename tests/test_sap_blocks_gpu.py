"""The even-odd SAP block kernel on blocks of every kind of size: fewer sites
than a warp's lane pairs, remainders of the sites per pass, one and several
sites per lane pair, the largest block that fits; every launch variant, with
12-real and 18-real links and a twisted mass, against the CPU restatement of
the cycle (oracle/qcd_oracle.c, modules/sap/sap.c:720)."""
import numpy as np
import pytest

import openqcd_b200 as qb
import oracle as O

pytestmark = pytest.mark.gpu

MU = 0.07
# two cycles on FP32 fields: a site's residual is the difference of terms
# about 20 times as large, each with about ten roundings of 6e-8 that add at
# random
TOL = 2e-6

SHAPES = [((4, 4, 4, 4), (2, 2, 2, 2)), ((8, 4, 4, 12), (4, 2, 2, 6)), ((8, 8, 8, 8), (4, 4, 4, 4)),
          ((8, 12, 8, 8), (4, 6, 4, 4)), ((16, 8, 8, 8), (8, 4, 4, 4)), ((12, 12, 8, 8), (6, 6, 4, 4)),
          ((12, 12, 12, 12), (6, 6, 6, 6)), ((16, 16, 8, 12), (8, 8, 4, 6))]


@pytest.mark.parametrize("L,bs", SHAPES, ids=["x".join(map(str, b)) for _, b in SHAPES])
def test_sap_blocks(L, bs):
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.4, 99)
    assert qb.sw_term() == 0
    qb.set_sap_parms(bs, 1, 3, 2)
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = [O.pauli_ref2lex(qb.download_swd(V, k), ipt).astype(np.float32) for k in (0, 1)]
    eta = np.random.default_rng(5).standard_normal(24 * V).astype(np.float32)
    psi, rho = np.zeros_like(eta), O.spinor_ref2lex(eta, ipt)
    for _ in range(2):
        psi, rho = O.sap(L, bs, MU, 1, 3, 0, U, sw[0], sw[1], psi, rho)
    half = int(np.prod(bs)) // 2
    refused = [v for v, most in ((0, 256), (4, 320), (5, 128)) if half > most] + [6]
    try:
        for l12 in (1, 0):
            qb.set_sap_link12(l12)
            for v in range(-1, 7):
                if v in refused:
                    with pytest.raises(qb.B200Error):
                        qb.set_sap_variant(v)
                    continue
                qb.set_sap_variant(v)
                p, r = qb.DevField(32), qb.DevField(32).from_ref(eta)
                qb.dev_sap(MU, 1, 3, 2, p, r)
                for x, y in ((p, psi), (r, rho)):
                    d = O.spinor_ref2lex(x.to_ref(V), ipt)
                    assert np.linalg.norm(d - y) <= TOL * np.linalg.norm(y), (l12, v)
    finally:
        qb.set_sap_link12(1)
