"""The batched little solver's sums, finished by the last block of a row: little
vectors within one block of threads and over several, few and many Krylov
vectors (every width of the product kernel), one to three systems, a larger
lattice after a smaller one (the batch's fields are sized anew); checked by
the true residual of the outer solve (oracle/qcd_oracle.c) and against the
single-system solver."""
import numpy as np
import pytest

import openqcd_b200 as qb
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,ns,nkv,res", [((8, 8, 8, 8), 2, 2, 1e-1), ((8, 8, 8, 8), 8, 16, 1e-6),
                                          ((16, 8, 8, 8), 20, 32, 1e-9)])
def test_little_sums(L, ns, nkv, res):
    bs = (4, 4, 4, 4)
    ipt = qb.even_first_ipt(L)
    V = ipt.size
    qb.geometry(L, bs, ipt)
    qb.set_parms(1.5, -0.05, 0)
    qb.random_ud(0.3, 99)
    assert qb.sw_term() == 0
    qb.set_sap_parms(bs, 1, 4, 3)
    qb.set_dfl_parms(bs, ns)
    qb.set_dfl_pro_parms(nkv, 256, res, 24, 1e-2)
    qb.set_dfl_gen_parms(1.0 / (2.0 * 3.95), 0.0, 4, 4, 4)
    assert qb.dfl_modes(1)[0] == 0
    U = O.links_ref2lex(qb.download_ud(V), ipt, L)
    sw = O.pauli_ref2lex(qb.download_swd(V), ipt)
    rng = np.random.default_rng(4)
    eta = [rng.standard_normal(24 * V) for _ in range(3)]
    one = qb.dfl_sap_gcr(8, 256, 0, 1e-10, 0.0, eta[0])
    for nr in (1, 3):
        E = [qb.DevField(64).from_ref(e) for e in eta[:nr]]
        P = [qb.DevField(64) for _ in range(nr)]
        rho, ifail, status, little = qb.dev_gcr_batch(8, 256, 0, 1e-10, [0.0] * nr, E, P, dfl=True)
        assert not any(ifail) and min(little) >= 1
        assert abs(status[0] - one[3][0]) <= 1
        for e, p in zip(eta, P):
            r = O.spinor_ref2lex(e, ipt) - O.dirac_dble(L, 0, 0.0, 0, U, sw, None, O.spinor_ref2lex(p.to_ref(V), ipt))
            assert np.linalg.norm(r) <= 1.0001e-10 * np.linalg.norm(e)
