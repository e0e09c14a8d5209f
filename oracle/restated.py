"""The part of reflib.RefLib's interface that the CPU restatement
(oracle/qcd_oracle.c) covers, for machines without the reference's sources:
gauge fields and SW term, the Dirac operators, SAP cycles and sap_gcr, and on
top of them, in numpy, the deflation: block basis, restriction and
prolongation, the little operators as dense matrices, and the deflated
solver.  The fields are its own (numpy's generators), drawn with the
reference's distributions; everything else goes through missing().  Test
infrastructure only."""
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
        if bc != 3 or isw != 0:
            self.missing("boundary conditions other than type 3 or exponential SW term")
        self.csw, self.m0, self.eoflg = csw, m0, eoflg
        self.theta = (0.0, 0.0, 0.0) if theta is None else theta

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
        links of the last plane (modules/uflds/uflds.c:307-335), and phase
        angles multiply U(x,k) by exp(i theta[k-1] / N[k]) (uflds.c:249-300)"""
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
        for k in range(3):
            U[:, k + 1] *= np.exp(1j * self.theta[k] / self.L[k + 1])
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

    def plaq_sum(self):
        """sum of Re tr of the plaquettes (modules/uflds/plaq_sum.c:161)"""
        U = self.U.view(np.complex128).reshape(self.L + (4, 3, 3)).copy()
        U[-1, :, :, :, 0] *= -1.0
        for k in range(3):
            U[..., k + 1, :, :] *= np.exp(-1j * self.theta[k] / self.L[k + 1])

        def up(a, mu):
            return np.roll(a, -1, axis=mu)
        out = 0.0
        for mu in range(4):
            for nu in range(mu):
                a, b = U[..., mu, :, :], U[..., nu, :, :]
                out += np.einsum("...ij,...jk,...lk,...il", a, up(b, mu), up(a, nu).conj(), b.conj(), optimize=True).real.sum()
        return out

    def random_sd(self, seed, sigma=1.0):
        """|s|^2 / sigma^2 distributed as by random_sd (modules/sflds/sflds.c)"""
        return np.random.default_rng(seed).standard_normal(24 * self.vol) * (sigma / np.sqrt(2.0))

    # ------------------------------------------------------- sums and matrices
    def spinor_prod_dble(self, s, r):
        a, b = (np.asarray(x, dtype=np.longdouble).reshape(-1, 2) for x in (s, r))
        z = (np.sum(a * b), np.sum(a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]))
        return np.array([f(x) for x in z for f in (float, lambda x: float(x - np.longdouble(float(x))))])

    def norm_square_dble(self, s):
        return self.spinor_prod_dble(s, s)[:2]

    def spinor_prod(self, s, r):
        return self.spinor_prod_dble(s, r)[::2].astype(np.float32)

    def norm_square(self, s):
        return np.float32(self.norm_square_dble(s)[0])

    @staticmethod
    def _pauli(m):
        """packed 6x6 matrices (modules/sw_term/pauli.c:953) -> full ones"""
        m = np.asarray(m, dtype=np.float64).reshape(-1, 36)
        out = np.zeros((len(m), 6, 6), dtype=np.complex128)
        out[:, range(6), range(6)] = m[:, :6]
        for k, (i, j) in enumerate((i, j) for i in range(6) for j in range(i + 1, 6)):
            out[:, i, j] = m[:, 6 + 2 * k] + 1j * m[:, 7 + 2 * k]
            out[:, j, i] = out[:, i, j].conj()
        return out

    def _sw_matrices(self, vol, mu, m):
        out = self._pauli(m)[:2 * vol]
        out[0::2, range(6), range(6)] += 1j * mu
        out[1::2, range(6), range(6)] -= 1j * mu
        return out

    def apply_sw_dble(self, vol, mu, m, s):
        s = np.ascontiguousarray(s, dtype=np.float64)
        w = s.view(np.complex128).reshape(-1, 6)[:2 * vol]
        return np.einsum("nij,nj->ni", self._sw_matrices(vol, mu, m), w).reshape(-1).view(np.float64)

    def apply_sw(self, vol, mu, m, s):
        return self.apply_sw_dble(vol, mu, m, s).astype(np.float32)

    def apply_swinv_dble(self, vol, mu, m, s):
        """and whether the Frobenius condition number of any matrix exceeds 100
        (modules/sw_term/pauli_dble.c:55-59)"""
        A = self._sw_matrices(vol, mu, m)
        inv = np.linalg.inv(A)
        w = np.ascontiguousarray(s, dtype=np.float64).view(np.complex128).reshape(-1, 6)[:2 * vol]
        cond = np.linalg.norm(A, axis=(1, 2)) * np.linalg.norm(inv, axis=(1, 2))
        return np.einsum("nij,nj->ni", inv, w).reshape(-1).view(np.float64), int(cond.max() > 100.0)

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

    # --------------------------------------------------------------- deflation
    # Little vectors: Ns numbers per block, the blocks of colour 0 first, each
    # colour in lexicographic order (modules/block/blk_grid.c:20-32).
    def dfl_init(self, bs, Ns, nkv=16, nmx=256, res=1e-2, nmx_gcr=24, res_gcr=1e-2, kappa=0.125, mu=0.0,
                 ninv=5, nmr=4, ncy=4):
        n = self._x // np.array(bs).reshape(4, 1)
        nb = [l // b for l, b in zip(self.L, bs)]
        lex = np.ravel_multi_index(n, nb)
        nbl = int(np.prod(nb))
        colour = np.indices(nb).reshape(4, -1).sum(axis=0) & 1
        order = np.lexsort((np.arange(nbl), colour))
        place = np.empty(nbl, dtype=int)
        place[order] = np.arange(nbl)
        sites = np.argsort(place[lex], kind="stable")       # of block 0, of block 1, ...
        self._blocks = sites.reshape(nbl, -1)
        self.Ns, self.nbl, self.nv = Ns, nbl, Ns * nbl
        self._little_of = None
        return self.nv

    def _by_block(self, s, dt=np.complex128):
        """storage order -> [block, component of the block's sites]"""
        f = np.asarray(s).reshape(self.vol, 24)[self.ipt()[self._blocks]]
        return np.ascontiguousarray(f.reshape(self.nbl, -1)).view(np.complex64 if f.dtype == np.float32
                                                                   else np.complex128).astype(dt)

    def _from_block(self, f, dt):
        out = np.empty((self.vol, 24), dtype=dt)
        out[self.ipt()[self._blocks]] = np.ascontiguousarray(f).view(np.float64).reshape(self.nbl, -1, 24)
        return out.reshape(-1)

    def dfl_subspace(self, modes):
        """the block orthonormal basis of the modes (dfl_subspace.c:171): Q of
        their QR decomposition with a positive diagonal of R"""
        M = np.stack([self._by_block(m) for m in modes], axis=-1)       # block, component, mode
        Q, R = np.linalg.qr(M)
        d = np.einsum("nll->nl", R)
        self._Q = (Q * (d / np.abs(d))[:, None, :]).astype(np.complex64).astype(np.complex128)
        self._little_of = None

    def dfl_modes(self, seed):
        """a subspace of random fields smoothed by one, two and three SAP cycles
        (dfl_modes.c:283-300), without the inverse iteration"""
        g = np.random.default_rng(seed)
        modes = []
        for _ in range(self.Ns):
            m = (g.random(24 * self.vol) - 0.5).astype(np.float32)
            for n in (1, 2, 3):
                m = self.sap(0.0, 1, 4, n, np.zeros_like(m), m)[0]
            modes.append(m)
        self.dfl_subspace(modes)
        return 0, [0, 0]

    def dfl_get_basis(self, l):
        return self._from_block(self._Q[:, :, l], np.float32)

    def _restrict(self, s):
        return np.einsum("ncl,nc->nl", self._Q.conj(), self._by_block(s)).reshape(-1)

    def _prolong(self, v, dt):
        return self._from_block(np.einsum("ncl,nl->nc", self._Q, v.reshape(self.nbl, self.Ns)), dt)

    def dfl_s2vd(self, s):
        return self._restrict(np.asarray(s, dtype=np.float32)).view(np.float64)

    def dfl_vd2s(self, vd):
        return self._prolong(np.ascontiguousarray(vd, dtype=np.float64).view(np.complex128), np.float32)

    def _Aw(self, mu):
        """the little operator as a matrix (Aw_ops.c:186): products of the basis
        with Dw on it and with i gamma5"""
        if self._little_of is None:
            A, G = (np.empty((self.nv, self.nv), dtype=np.complex128) for _ in range(2))
            e = np.zeros(self.nv, dtype=np.complex128)
            g5 = np.repeat([1.0, -1.0], 12)
            for j in range(self.nv):
                e[:] = 0.0
                e[j] = 1.0
                b = self._prolong(e, np.float64)
                A[:, j] = self._restrict(self.dirac_dble(0, 0.0, b))
                G[:, j] = 1j * self._restrict((b.reshape(-1, 24) * g5).reshape(-1))
            self._little_of = A, G
        A, G = self._little_of
        return A + mu * G

    def little(self, which, mu, v, w=None):
        """Aw, Awhat, Aweeinv, Awooinv, Awoe, Aweo (Aw_dble.c:122-361)"""
        v = np.ascontiguousarray(v, dtype=np.float64).view(np.complex128)
        w = np.zeros_like(v) if w is None else np.array(w, dtype=np.float64, copy=True).view(np.complex128)
        A, h = self._Aw(mu), self.nv // 2
        ee, oo = A[:h, :h].copy(), A[h:, h:].copy()
        for M in (ee, oo):                     # the diagonal blocks; blocks of one colour do not touch
            M[np.kron(np.eye(self.nbl // 2), np.ones((self.Ns, self.Ns))) == 0] = 0.0
        if which == 0:
            w = A @ v
        elif which == 1:
            w[:h] = v[:h] - np.linalg.solve(ee, A[:h, h:] @ np.linalg.solve(oo, A[h:, :h] @ v[:h]))
        elif which == 2:
            w[:h] = np.linalg.solve(ee, v[:h])
        elif which == 3:
            w[h:] = np.linalg.solve(oo, v[h:])
        elif which == 4:
            w[h:] = A[h:, :h] @ v[:h]
        elif which == 5:
            w[:h] -= A[:h, h:] @ v[h:]
        else:
            self.missing("little operator %d" % which)
        return w.view(np.float64), 0

    def little32(self, which, mu, v, w=None):
        w = None if w is None else np.asarray(w, dtype=np.float64)
        return self.little(which, mu, np.asarray(v, dtype=np.float64), w)[0].astype(np.float32)

    def ltl_gcr(self, mu, eta):
        """the solution itself; the steps it takes are not restated"""
        e = np.ascontiguousarray(eta, dtype=np.float64).view(np.complex128)
        return np.linalg.solve(self._Aw(mu), e).view(np.float64), 0.0, 0, [1, 1]

    def dfl_sap_gcr(self, nkv, nmx, istop, res, mu, eta):
        """GCR with the preconditioner of dfl_sap_gcr.c:212-241 (an exact little
        solve), in double precision, restarted after nkv steps"""
        bs, isolv, nmr, ncy = self.sap_parms
        A = np.linalg.inv(self._Aw(mu))
        psi, r = np.zeros_like(eta), np.array(eta)
        tol, steps = res * np.linalg.norm(eta), 0
        while np.linalg.norm(r) > tol and steps < nmx:
            chi = []
            while len(chi) < nkv and np.linalg.norm(r) > tol and steps < nmx:
                p = self._prolong(A @ self._restrict(r), np.float64)
                q = r - self.dirac_dble(0, mu, p)
                d = self.sap(mu, isolv, nmr, ncy, np.zeros(q.size, np.float32), q.astype(np.float32))[0]
                p = (p + d).view(np.complex128)
                q = self.dirac_dble(0, mu, p.view(np.float64)).view(np.complex128)
                for a, b in chi:
                    z = np.vdot(b, q)
                    p, q = p - z * a, q - z * b
                n = np.linalg.norm(q)
                p, q = p / n, q / n
                z = np.vdot(q, r.view(np.complex128))
                psi, r = psi + (z * p).view(np.float64), r - (z * q).view(np.float64)
                chi.append((p, q))
                steps += 1
            r = eta - self.dirac_dble(0, mu, psi)
        return psi, np.linalg.norm(r), 0 if np.linalg.norm(r) <= tol * 1.0001 else -1, [steps, 1, 0]
