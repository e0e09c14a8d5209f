"""The part of reflib.RefLib's interface that the CPU restatement
(oracle/qcd_oracle.c) covers, for machines without the reference's sources:
gauge fields and SW term, the Dirac operators, SAP cycles and sap_gcr.  The
fields are its own (numpy's generators), drawn with the reference's
distributions; everything else goes through missing().  Test infrastructure
only."""
import numpy as np

import oracle as O
from reflib import GEOMETRIES


class Restated:
    def __init__(self, L):
        self.L = tuple(L)
        self.vol = int(np.prod(L))
        self.eoflg = 0
        self._x = np.indices(self.L).reshape(4, -1)

    def missing(self, what):
        raise NotImplementedError("the CPU restatement has no " + what)

    def __getattr__(self, name):
        if name.startswith("_"):
            raise AttributeError(name)
        return self.missing(name)

    def init(self, bc=3, seed=1234, csw=1.5, m0=0.0, eoflg=0, isw=0, theta=None):
        if bc != 3 or isw != 0 or (theta is not None and np.any(theta)):
            self.missing("boundary conditions other than type 3, exponential SW term or phase angles")
        self.csw, self.m0, self.eoflg = csw, m0, eoflg

    def set_sw_parms(self, m0):
        self.m0 = m0

    def set_tm_parms(self, eoflg):
        self.eoflg = eoflg

    def set_sap_parms(self, bs, isolv, nmr, ncy):
        self.sap_parms = (bs, isolv, nmr, ncy)

    def ipt(self):
        """an order of the reference's kind (modules/lattice/geometry.c:200-240):
        even sites first, the thread-local sub-lattices one after the other
        with x0 slowest, lexicographic within them"""
        T = GEOMETRIES.get(self.L, self.L)
        sub = np.ravel_multi_index([x // t for x, t in zip(self._x, T)], [n // t for n, t in zip(self.L, T)])
        order = np.lexsort((np.arange(self.vol), sub, self._x.sum(axis=0) & 1))
        out = np.empty(self.vol, dtype=np.int32)
        out[order] = np.arange(self.vol, dtype=np.int32)
        return out

    # ------------------------------------------------------------------ fields
    def gen_links(self, eps, seed):
        """U = exp(eps X), X distributed as by random_alg
        (modules/linalg/liealg.c:41-65); bc type 3 flips the sign of the time
        links of the last plane (modules/uflds/uflds.c:307-335)"""
        g = np.random.default_rng(seed).standard_normal((8, self.vol, 4)) / np.sqrt(2.0)
        a, b = (np.sqrt(3.0) + 1.0) / 6.0, (np.sqrt(3.0) - 1.0) / 6.0
        x1, x2 = a * g[0] + b * g[1], a * g[1] + b * g[0]
        off = (g[2::2] + 1j * g[3::2]) / np.sqrt(2.0)
        X = np.zeros((self.vol, 4, 3, 3), dtype=np.complex128)
        for i, d in enumerate((x1 + x2, x2 - 2 * x1, x1 - 2 * x2)):
            X[..., i, i] = 1j * d
        for z, (i, j) in zip(off, ((0, 1), (0, 2), (1, 2))):
            X[..., i, j], X[..., j, i] = z, -z.conj()
        w, v = np.linalg.eigh(-1j * eps * X)
        U = (v * np.exp(1j * w)[..., None, :]) @ v.conj().swapaxes(-1, -2)
        U[self._x[0] == self.L[0] - 1, 0] *= -1.0
        self.U = np.ascontiguousarray(U).view(np.float64).reshape(-1)

    def ud(self):
        """the eight links of every odd site (main/README.global:229-262)"""
        ipt, U, V = self.ipt(), self.U.reshape(self.vol, 4, 18), self.vol
        odd = ipt >= V // 2
        base = 8 * (ipt[odd] - V // 2)
        out = np.zeros((4 * V, 18))
        for mu in range(4):
            y = self._x[:, odd].copy()
            y[mu] = (y[mu] - 1) % self.L[mu]
            out[base + 2 * mu] = U[odd, mu]
            out[base + 2 * mu + 1] = U[np.ravel_multi_index(y, self.L), mu]
        return out.reshape(-1)

    def set_ud(self, ud):
        self.U = O.links_ref2lex(ud, self.ipt(), self.L)

    def sw_term(self, which=0):
        """which: 0 nothing, 1 the even, 2 the odd, 3 all sites inverted in
        swd(); the operators below need none of it"""
        self.sw = O.sw_term(self.L, self.csw, self.m0, self.U)
        self.swi, fail = O.invert_field(self.sw)
        self._which = which
        return fail if which else 0

    def swd(self):
        inv = np.where(self._x.sum(axis=0) & 1, self._which & 2, self._which & 1) != 0
        out = np.empty((self.vol, 72))
        out[self.ipt()] = np.where(inv[:, None], self.swi.reshape(-1, 72), self.sw.reshape(-1, 72))
        return out.reshape(-1)

    def random_sd(self, seed, sigma=1.0):
        """|s|^2 / sigma^2 distributed as by random_sd (modules/sflds/sflds.c)"""
        return np.random.default_rng(seed).standard_normal(24 * self.vol) * (sigma / np.sqrt(2.0))

    # --------------------------------------------------------------- operators
    def _call(self, dt, f, *fields):
        ipt = self.ipt()
        lex = [None if x is None else O.spinor_ref2lex(np.asarray(x, dtype=dt), ipt) for x in fields]
        out = f(*lex)
        if not isinstance(out, tuple):
            return O.spinor_lex2ref(out, ipt)
        return tuple(O.spinor_lex2ref(x, ipt) if isinstance(x, np.ndarray) else x for x in out)

    def dirac_dble(self, op, mu, s, r=None):
        return self._call(np.float64, lambda s, r: O.dirac_dble(self.L, op, mu, self.eoflg, self.U, self.sw, self.swi,
                                                                s, r), s, r)

    def dirac(self, op, mu, s, r=None):
        return self._call(np.float32, lambda s, r: O.dirac(self.L, op, mu, self.eoflg, self.U, self.sw, self.swi, s, r),
                          s, r)

    def sap(self, mu, isolv, nmr, ncy, psi, rho):
        sw, swi = self.sw.astype(np.float32), self.swi.astype(np.float32)

        def f(psi, rho):
            for _ in range(ncy):
                psi, rho = O.sap(self.L, self.sap_parms[0], mu, isolv, nmr, self.eoflg, self.U, sw, swi, psi, rho)
            return psi, rho, 0
        return self._call(np.float32, f, psi, rho)

    def sap_gcr(self, nkv, nmx, istop, res, mu, eta):
        bs, isolv, nmr, ncy = self.sap_parms
        return self._call(np.float64, lambda e: O.sap_gcr(self.L, bs, isolv, nmr, ncy, self.eoflg, self.U, self.sw,
                                                          self.sw.astype(np.float32), self.swi.astype(np.float32),
                                                          nkv, nmx, istop, res, mu, e), eta)
