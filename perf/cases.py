"""The work a user of this library has it do, as cases that can be timed and
checked: the Wilson-Dirac operator, the SAP preconditioner, the deflation
transfers and the two solvers, through the public entry points.

A gauge configuration is what a program keeps between calls (it is loaded
once and used for many sources), so the library's resident fields depend on
the case's lattice alone; the sources depend on the seed.

Fields returned by run() are in the library's device layout (even sites
first, per parity half blocks in lexicographic order, per block component
planes of consecutive sites) for the device entry points, and in the
reference's storage order for the drop-in ones.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "openqcd-2.4.2_b200"))

import openqcd_b200 as qb  # noqa: E402

BLOCK_MAX = 1536       # sites of the largest SAP block


# ------------------------------------------------------------------ the cases
def _case(path, L, bs, **kw):
    c = {"path": path, "eps": 0.3, "m0": -0.05, "csw": 1.7, "mu": 0.0}
    c.update({"L%d" % i: L[i] for i in range(4)})
    c.update({"b%d" % i: bs[i] for i in range(4)})
    c.update(kw)
    return c


def listed():
    b4, b6 = (4, 4, 4, 4), (6, 6, 6, 6)
    small = {"eps": 0.4, "m0": 0.0, "csw": 1.5}
    out = [
        # the smallest lattice of the tests and of the first configuration:
        # one application is launch latency
        ("dw_f64_small", _case("dirac", (8, 8, 8, 8), b4, op="Dw", prec=64, **small)),
        # the bandwidth configuration: 32^3x64, FP64 (residuals, CG)
        ("dw_f64_large", _case("dirac", (64, 32, 32, 32), b4, op="Dw", prec=64)),
        # the even-odd preconditioned FP64 operator of the CG solvers, on a
        # middling lattice
        ("dwhat_f64", _case("dirac", (32, 16, 16, 16), b4, op="Dwhat", prec=64, mu=0.02)),
        # the FP32 operator inside the solvers, with the 6^4 blocks of the
        # deflated configuration
        ("dw_f32_blocks6", _case("dirac", (48, 24, 24, 24), b6, op="Dw", prec=32)),
        # the drop-in call of a host program: page-locked fields in the
        # reference's order, copied in and out
        ("dw_host", _case("host", (32, 16, 16, 16), b4)),
        # the SAP preconditioner as sap_gcr applies it: five cycles of four MR
        # steps, on the training lattice of the learned preconditioner ...
        ("sap_small", _case("sap", (16, 16, 16, 16), b4, nmr=4, ncy=5)),
        # ... with the 6^4 blocks and the large field of the deflated
        # configuration (its two cycles of three steps) ...
        ("sap_blocks6", _case("sap", (48, 24, 24, 24), b6, nmr=3, ncy=2)),
        # ... and with oblong blocks and a twisted mass
        ("sap_oblong", _case("sap", (24, 24, 16, 8), (4, 6, 8, 4), nmr=4, ncy=2, mu=0.02)),
        # restriction and prolongation of four fields on 28 deflation modes
        ("transfer", _case("transfer", (48, 24, 24, 24), b6, ns=28, nr=4)),
        # the whole solver: sap_gcr to a relative residual of 1e-10 on 8^4
        # (the first configuration) and on 32x16^3
        ("solve_small", _case("solve", (8, 8, 8, 8), b4, nmr=4, ncy=5, nkv=16, **small)),
        ("solve", _case("solve", (32, 16, 16, 16), b4, nmr=4, ncy=5, nkv=16)),
        # the deflated solver on four sources at once
        ("solve_deflated", _case("deflated", (24, 12, 12, 12), b6, nmr=3, ncy=2, nkv=8, ns=20, nr=4)),
    ]
    return [dict(c, name=n) for n, c in out]


def _draw_lattice(rng, vmin, vmax, blocks=(4, 4, 6, 8)):
    while True:
        bs = [rng.choice(blocks) for _ in range(4)]
        if math.prod(bs) <= BLOCK_MAX and math.prod(2 * b for b in bs) <= vmax:
            break
    want = math.exp(rng.uniform(math.log(vmin), math.log(vmax)))
    nb = [2, 2, 2, 2]
    for _ in range(200):
        k = rng.choice((0, 0, 1, 2, 3))      # time is usually the longest
        nb[k] += 2
        if math.prod(n * b for n, b in zip(nb, bs)) > want:
            nb[k] -= 2
    return [n * b for n, b in zip(nb, bs)], bs


def draw(rng):
    path = rng.choice(("dirac", "dirac", "dirac", "dirac", "sap", "sap", "sap", "host", "transfer", "solve"))
    mu = rng.choice((0.0, 0.0, 0.02, 0.1))
    if path == "dirac":
        L, bs = _draw_lattice(rng, 4096, 2000000)
        return _case(path, L, bs, op=rng.choice(("Dw", "Dw", "Dw", "Dwhat", "Dwhat", "Dwoe", "Dwee")),
                     prec=rng.choice((64, 32)), mu=mu)
    if path == "sap":
        L, bs = _draw_lattice(rng, 4096, 660000)
        return _case(path, L, bs, nmr=rng.randint(2, 5), ncy=rng.choice((1, 2)), mu=mu)
    if path == "host":
        L, bs = _draw_lattice(rng, 4096, 131072)
        return _case(path, L, bs, mu=mu)
    if path == "transfer":
        L, bs = _draw_lattice(rng, 8192, 400000)
        return _case(path, L, bs, ns=2 * rng.randint(4, 14), nr=rng.choice((1, 2, 4, 5)))
    L, bs = _draw_lattice(rng, 4096, 100000)
    return _case(path, L, bs, nmr=4, ncy=rng.choice((3, 5)), nkv=16, mu=mu)


def _dims(case):
    return [case["L%d" % i] for i in range(4)], [case["b%d" % i] for i in range(4)]


def work(case):
    """Bytes: per application each field read or written once (spinor 192,
    links 576, SW matrices 576 bytes per site in FP64, half of that in FP32).
    Flops: 1824 a site for the hops and the SW term (1320 + 504)."""
    L, _ = _dims(case)
    V = math.prod(L)
    p, f = case["path"], 1824.0
    if p == "dirac":
        w = 8 if case["prec"] == 64 else 4
        per = {"Dw": 48 + 72 + 72, "Dwhat": (24 + 24 + 72) / 2 + 36 + 72, "Dwoe": 12 + 12 + 72, "Dwee": 12 + 12 + 36}
        fl = {"Dw": f, "Dwhat": f, "Dwoe": 660.0, "Dwee": 252.0}
        return {"bytes": V * w * per[case["op"]], "flops": V * fl[case["op"]]}
    if p == "host":
        return {"bytes": V * (1536 + 2 * 192), "flops": V * f}
    if p == "transfer":
        ns, nr = case["ns"], case["nr"]
        return {"bytes": V * 96.0 * (2 * ns + 2 * nr), "flops": V * 2.0 * 12 * 8 * ns * nr}
    # one SAP cycle: rho and psi in and out, links and SW matrices once;
    # nmr + 2 block operators
    cyc_b, cyc_f = V * (4 * 96 + 288 + 288), V * f * (case["nmr"] + 2)
    if p == "sap":
        return {"bytes": case["ncy"] * cyc_b + V * 96.0, "flops": case["ncy"] * cyc_f}
    # solvers: six steps (the fewest seen) of ncy cycles and the step's
    # vector work, and the final FP64 residual
    nr = case.get("nr", 1)
    by = 6 * (case["ncy"] * cyc_b + V * 96.0 * 6) + V * 1536
    return {"bytes": nr * by, "flops": nr * (6 * case["ncy"] * cyc_f + V * f)}


def tolerance(case):
    """about four times the distance to exact() that was measured"""
    p = case["path"]
    if p == "host":
        return {"rel": 1e-15}
    if p == "dirac":
        return {"rel": 1e-15} if case["prec"] == 64 else {"rel": 4e-7}
    if p == "sap":
        # 2e-7 to 3e-7 relative to the residual that the cycles leave, which
        # more of them make smaller
        return {"rel": 2e-6}
    if p == "transfer":
        return {"rel": 1e-6}
    # 5e-10: the relative residual of 1e-10 the solvers stop at
    return {"rel": 3e-9}


# ------------------------------------------------- fields made from seeds
def _gen(*seed):
    g = torch.Generator(device="cuda")
    s = 1469598103934665603
    for x in seed:
        s = ((s ^ int(x)) * 1099511628211) % (1 << 62)
    g.manual_seed(s)
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _links(L, eps):
    """U(x, mu) = exp(i eps H), H Gaussian traceless Hermitian with unit
    variance per su(3) generator, lexicographic sites; the time links of the
    last plane carry the sign of the antiperiodic quark boundary."""
    V = math.prod(L)
    c = _normal(_gen(17, *L), 8, V, 4) * (0.5 * eps)
    H = torch.zeros(V, 4, 3, 3, dtype=torch.complex128, device="cuda")
    d8 = c[7] / math.sqrt(3.0)
    H[..., 0, 0] = c[2] + d8
    H[..., 1, 1] = d8 - c[2]
    H[..., 2, 2] = -2.0 * d8
    for a, b, k in ((0, 1, 0), (0, 2, 3), (1, 2, 5)):
        H[..., a, b] = torch.complex(c[k], -c[k + 1])
        H[..., b, a] = torch.complex(c[k], c[k + 1])
    del c, d8
    # exp(A) by squaring exp(A/4), a Taylor series that ends below 1e-17
    A = H * 0.25j
    del H
    U = torch.eye(3, dtype=torch.complex128, device="cuda").expand(V, 4, 3, 3).clone()
    for n in range(14, 0, -1):
        U = _mm(A, U) / n
        for i in range(3):
            U[..., i, i] += 1.0
    U = _mm(U, U)
    U = _mm(U, U)
    U.view(L[0], -1, 4, 3, 3)[-1, :, 0] *= -1.0
    return U


def _mm(a, b):
    return sum(a[..., :, k, None] * b[..., None, k, :] for k in range(3))


@functools.lru_cache(maxsize=2)
def _ipt(L):
    return qb.even_first_ipt(L).astype(np.int64)


def _shift(x, L, mu, n):
    """x(s + n mu) for an array over lexicographic sites (first axis)"""
    return torch.roll(x.view(*L, *x.shape[1:]), -n, mu).reshape(x.shape)


def _links_storage(U, L):
    """the reference's array of the eight links of every odd site"""
    ipt = torch.from_numpy(_ipt(tuple(L))).cuda()
    V = ipt.numel()
    odd = torch.nonzero(ipt >= V // 2).flatten()
    base = 8 * (ipt[odd] - V // 2)
    out = torch.empty(4 * V, 3, 3, dtype=torch.complex128, device="cuda")
    for mu in range(4):
        out[base + 2 * mu] = U[odd, mu]
        out[base + 2 * mu + 1] = _shift(U[:, mu], L, mu, -1)[odd]
    return out


def _source(L, seed, k, prec):
    """Gaussian spinor field, [V, 4, 3] complex, lexicographic"""
    f = torch.view_as_complex(_normal(_gen(29, seed, k, *L), math.prod(L), 4, 3, 2))
    return f if prec == 64 else f.to(torch.complex64)


def _modes(L, l):
    return torch.view_as_complex(_normal(_gen(31, l, *L), math.prod(L), 4, 3, 2)).to(torch.complex64)


def _to_storage(f, L):
    """lexicographic -> the reference's storage order, real view"""
    out = torch.empty_like(f)
    out[torch.from_numpy(_ipt(tuple(L))).cuda()] = f
    return torch.view_as_real(out).reshape(-1)


@functools.lru_cache(maxsize=2)
def _device_sites(L, bs):
    """lexicographic site of every device site (parity, block, site)"""
    x = np.indices(L).reshape(4, -1)
    b = np.array(bs).reshape(4, 1)
    nb = [n // m for n, m in zip(L, bs)]
    blk = np.ravel_multi_index(tuple(x // b), nb)
    s = np.ravel_multi_index(tuple(x % b), bs) // 2
    vbh = math.prod(bs) // 2
    dev = ((x.sum(axis=0) & 1) * math.prod(nb) + blk) * vbh + s
    out = np.empty_like(dev)
    out[dev] = np.arange(dev.size)
    return out


def _to_device(f, L, bs, prec):
    """lexicographic [V, 4, 3] -> the device layout, flat reals"""
    vbh = math.prod(bs) // 2
    g = torch.view_as_real(f[torch.from_numpy(_device_sites(tuple(L), tuple(bs))).cuda()])   # V, 4, 3, 2
    per = 1 if prec == 64 else 2            # complex components of one plane's element
    g = g.reshape(-1, vbh, 12 // per, per * 2).transpose(1, 2)
    return g.reshape(-1).contiguous()


# ------------------------------------------------------------ what is resident
_resident = None
_fields = ("L0", "L1", "L2", "L3", "b0", "b1", "b2", "b3", "eps", "m0", "csw", "path", "nmr", "ncy", "ns")


def _load(case):
    """the case's gauge field, SW term, SAP parameters and deflation subspace
    in the library, if they are not there yet"""
    global _resident
    key = tuple(case.get(k) for k in _fields)
    if _resident == key:
        return
    _resident = None
    L, bs = _dims(case)
    qb.release_workspace()
    qb.geometry(L, bs, _ipt(tuple(L)))
    qb.set_parms(case["csw"], case["m0"], 0)
    ud = _links_storage(_links(L, case["eps"]), L)
    torch.cuda.synchronize()
    qb.check(qb.lib().b200_upload_ud(ud.data_ptr()))
    del ud
    if qb.sw_term() != 0:
        raise RuntimeError("the SW term is not safely invertible")
    if "nmr" in case:
        qb.set_sap_parms(bs, 1, case["nmr"], case["ncy"])
    if "ns" in case:
        qb.set_dfl_parms(bs, case["ns"])
        qb.set_dfl_pro_parms(24, 256, 1e-2, 24, 1e-2)
        if case["path"] == "transfer":
            m = [_to_storage(_modes(L, l), L) for l in range(case["ns"])]
            torch.cuda.synchronize()
            qb._void(qb.lib().dfl_subspace, (ctypes.c_void_p * len(m))(*[x.data_ptr() for x in m]))
            del m
        else:
            qb.set_dfl_gen_parms(1.0 / (2.0 * (4.0 + case["m0"])), 0.0, 6, 4, 4)
            if qb.dfl_modes(1)[0] != 0:
                raise RuntimeError("subspace generation failed")
            qb.release_workspace()
    torch.cuda.empty_cache()
    _resident = key


class _Field:
    """a spinor field in the device layout, held by a tensor"""

    def __init__(self, case, prec):
        self.prec = prec
        self.data = torch.zeros(24 * math.prod(_dims(case)[0]), dtype=torch.float64 if prec == 64 else torch.float32,
                                device="cuda")
        self.ptr = self.data.data_ptr()


def _dev_source(case, seed, k, prec):
    L, _ = _dims(case)
    q = _to_storage(_source(L, seed, k, prec), L)
    f = _Field(case, prec)
    torch.cuda.synchronize()
    qb.check(qb.lib().b200_dev_from_ref(prec, q.data_ptr(), f.ptr))
    return f


def prepare(case, seed):
    _load(case)
    L, _ = _dims(case)
    p, st = case["path"], {"case": case, "key": _resident}
    if p == "dirac":
        st["s"], st["r"] = _dev_source(case, seed, 0, case["prec"]), _Field(case, case["prec"])
    elif p == "host":
        st["s"] = _to_storage(_source(L, seed, 0, 64), L).cpu().pin_memory()
        st["r"] = torch.zeros_like(st["s"]).pin_memory()
    elif p == "sap":
        st["eta"], st["zero"] = _dev_source(case, seed, 0, 32), _Field(case, 32)
        st["psi"], st["rho"] = _Field(case, 32), _Field(case, 32)
    elif p == "transfer":
        nr, nv = case["nr"], qb.lib().b200_dfl_nv()
        st["f"] = [_to_storage(_source(L, seed, k, 32), L) for k in range(nr)]
        st["v"] = [_normal(_gen(37, seed, k), 2 * nv) for k in range(nr)]
        st["vd"] = [torch.zeros_like(v) for v in st["v"]]
        st["s"] = [torch.zeros_like(f) for f in st["f"]]
        for k in ("f", "v", "vd", "s"):
            st["p" + k] = (ctypes.c_void_p * nr)(*[t.data_ptr() for t in st[k]])
    else:
        nr = case.get("nr", 1)
        st["eta"] = [_dev_source(case, seed, k, 64) for k in range(nr)]
        st["psi"] = [_Field(case, 64) for _ in range(nr)]
    torch.cuda.synchronize()
    return st


def run(st):
    case, lib = st["case"], qb.lib()
    if st["key"] != _resident:
        _load(case)
    p = case["path"]
    if p == "dirac":
        qb.dev_dirac(case["op"], case["mu"], st["s"], st["r"])
        return st["r"].data
    if p == "host":
        lib.Dw_dble(case["mu"], st["s"].data_ptr(), st["r"].data_ptr())
        return st["r"]
    if p == "sap":
        # the preconditioner: psi = 0, rho = eta, then the cycles
        nb = st["eta"].data.numel() * 4
        qb.check(lib.b200_memcpy(st["rho"].ptr, st["eta"].ptr, nb))
        qb.check(lib.b200_memcpy(st["psi"].ptr, st["zero"].ptr, nb))
        qb.dev_sap(case["mu"], 1, case["nmr"], case["ncy"], st["psi"], st["rho"])
        return [st["psi"].data, st["rho"].data]
    if p == "transfer":
        qb.check(lib.b200_dfl_s2vd_multi(case["nr"], st["pf"], st["pvd"]))
        qb.check(lib.b200_dfl_vd2s_multi(case["nr"], st["pv"], st["ps"]))
        return [st["vd"], st["s"]]
    if p == "solve":
        _, ifail, _ = qb.dev_sap_gcr(case["nkv"], 256, 0, 1e-10, case["mu"], st["eta"][0], st["psi"][0])
        fails = [ifail]
    else:
        nr = case["nr"]
        _, fails, _, _ = qb.dev_gcr_batch(case["nkv"], 256, 0, 1e-10, [case["mu"]] * nr, st["eta"], st["psi"], dfl=True)
    if any(fails):
        raise RuntimeError("the solver failed: %s" % (fails,))
    return [x.data for x in st["psi"]]


# -------------------------------------------------- the same in 64 bits, plainly
# (1 - gamma_mu): component 0 couples to a0 with f0, component 1 to a1 with f1
_PROJ = ((2, 1, 3, 1), (3, 1j, 2, 1j), (3, 1, 2, -1), (2, 1j, 3, -1j))


class _Plain:
    """Wilson-Dirac operator with the SW term on lexicographic complex128
    fields [V, 4, 3], written from its definition."""

    def __init__(self, case):
        L, bs = self.L, self.bs = _dims(case)
        self.V = math.prod(L)
        self.U = _links(L, case["eps"])
        self.A = self._sw(case["csw"], case["m0"])          # V, 2, 6, 6
        x = np.indices(L).reshape(4, -1)
        self.odd = torch.from_numpy((x.sum(axis=0) & 1).astype(bool)).cuda()[:, None, None]
        b = np.array(bs).reshape(4, 1)
        nb = [n // m for n, m in zip(L, bs)]
        self.nbl = math.prod(nb)
        self.blk = torch.from_numpy(np.ravel_multi_index(tuple(x // b), nb)).cuda()
        self.colour = torch.from_numpy(((x // b).sum(axis=0) & 1)).cuda()[:, None, None]
        # inside[mu]: x + mu lies in the block of x
        self.inside = [torch.from_numpy(x[m] % bs[m] + 1 < bs[m]).cuda()[:, None, None] for m in range(4)]
        self.g5 = torch.tensor([1, 1, -1, -1], dtype=torch.complex128, device="cuda")[None, :, None]

    def _field(self, mu, nu):
        """anti-Hermitian clover field: the sum over the four leaves of
        (m - m^dagger)/8"""
        L, U = self.L, self.U
        u, v = U[:, mu], U[:, nu]
        dag = lambda m: m.conj().transpose(-1, -2)   # noqa: E731
        u_nu, v_mu = _shift(u, L, nu, 1), _shift(v, L, mu, 1)
        w1, w2 = _mm(u, v_mu), _mm(dag(u_nu), dag(v))       # around the plaquette at x
        w3, w4 = _mm(dag(v), u), _mm(v_mu, dag(u_nu))
        m = _mm(w1, w2)
        # m(x) of the leaf at x; those of the plaquettes at x - mu - nu, x - nu, x - mu
        m = m + _shift(_shift(_mm(w2, w1), L, mu, -1), L, nu, -1)
        m = m + _shift(_mm(w3, w4), L, nu, -1) + _shift(_mm(w4, w3), L, mu, -1)
        return (m - dag(m)) / 8.0

    def _sw(self, csw, m0):
        A = torch.zeros(self.V, 2, 2, 3, 2, 3, dtype=torch.complex128, device="cuda")
        sig = (((0, 1, 1), (1, 0, 1)), ((0, 1, -1j), (1, 0, 1j)), ((0, 0, 1), (1, 1, -1)))
        for k, (el, mag) in enumerate((((0, 1), (2, 3)), ((0, 2), (3, 1)), ((0, 3), (1, 2)))):
            E, B = self._field(*el), self._field(*mag)
            for h, F in ((0, B - E), (1, B + E)):
                for i, j, z in sig[k]:
                    A[:, h, i, :, j, :] += (-0.5 * csw * 1j * z) * F
        A = A.view(self.V, 2, 6, 6)
        for i in range(6):
            A[:, :, i, i] += 4.0 + m0
        return A

    def sw(self, s, mu=0.0, inverse=False):
        """(A + i mu g5) s, or A^-1 s"""
        if inverse and not hasattr(self, "Ai"):
            self.Ai = torch.linalg.inv(self.A)
        M, w = (self.Ai if inverse else self.A), s.reshape(self.V, 2, 6)
        r = sum(M[..., k] * w[..., None, k] for k in range(6)).view(s.shape)
        return r + 1j * mu * self.g5 * s if mu else r

    def hop(self, s, masks=None):
        """-1/2 sum over mu of U (1 - g) s(x + mu) + U^dagger (1 + g) s(x - mu);
        masks[mu]: the links (x, x + mu) to keep"""
        acc = torch.zeros_like(s)
        for mu, (a0, f0, a1, f1) in enumerate(_PROJ):
            U = self.U[:, mu]
            for sgn in (1, -1):
                t = _shift(s, self.L, mu, 1) if sgn > 0 else s
                h = torch.stack((t[:, 0] + sgn * f0 * t[:, a0], t[:, 1] + sgn * f1 * t[:, a1]), 1)
                if sgn > 0:
                    c = sum(U[:, None, :, k] * h[:, :, None, k] for k in range(3))
                else:
                    c = sum(U.conj()[:, None, k, :] * h[:, :, None, k] for k in range(3))
                if masks is not None:
                    c = c * masks[mu]
                if sgn < 0:
                    c = _shift(c, self.L, mu, -1)
                acc[:, :2] += c
                acc[:, a0] += sgn * complex(f0).conjugate() * c[:, 0]
                acc[:, a1] += sgn * complex(f1).conjugate() * c[:, 1]
        return acc.mul_(-0.5)

    def even(self, s):
        return torch.where(self.odd, 0.0, s)

    def odds(self, s):
        return torch.where(self.odd, s, 0.0)

    def apply(self, op, mu, s):
        if op == "Dw":
            return self.sw(s, mu) + self.hop(s)
        if op == "Dwee":
            return self.even(self.sw(s, mu))
        if op == "Dwoe":
            return self.odds(self.hop(self.even(s)))
        e = self.even(s)                                     # Dwhat
        t = self.odds(self.sw(self.hop(e), inverse=True))
        return self.even(self.sw(e, mu) - self.hop(t))

    def blocks(self, a, b):
        """(a, b) summed over every block, at every site"""
        v = (a.conj() * b).sum((1, 2))
        out = torch.zeros(self.nbl, dtype=v.dtype, device="cuda").index_add_(0, self.blk, v)
        return out[self.blk][:, None, None]

    def sap(self, mu, nmr, ncy, eta):
        """multiplicative Schwarz cycles from psi = 0: per block nmr MR steps
        on the even-odd preconditioned block operator"""
        psi, rho = torch.zeros_like(eta), eta.clone()
        cross = [~m for m in self.inside]
        bhop = lambda x: self.hop(x, self.inside)   # noqa: E731
        for ic in list(range(2)) * ncy:
            on = self.colour == ic
            r = torch.where(on, rho, 0.0)
            v = self.odds(self.sw(r, inverse=True))
            s1 = self.even(r - bhop(v))
            s0 = torch.zeros_like(s1)
            for _ in range(nmr):
                w = self.odds(self.sw(bhop(s1), inverse=True))
                s2 = self.even(self.sw(s1, mu) - bhop(w))
                n = self.blocks(s2, s2)
                z = torch.where(n.real > 0, self.blocks(s2, s1) / n, 0.0)
                s0, s1 = s0 + z * s1, s1 - z * s2
            phi = s0 + v - self.odds(self.sw(bhop(s0), inverse=True))
            psi = psi + phi
            rho = torch.where(on, s1 - 1j * mu * self.g5 * self.odds(phi), rho)
            rho = torch.where(on, rho, rho - self.hop(phi, cross))
        return psi, rho

    def solve(self, mu, eta):
        """Dw psi = eta by BiCGstab on the even-odd preconditioned system"""
        if mu:          # the inverse of A + i mu g5 on the odd sites
            sh = torch.tensor([1, -1], dtype=torch.complex128, device="cuda")[None, :, None, None] * (1j * mu)
            self.Ai = torch.linalg.inv(self.A + sh * torch.eye(6, device="cuda", dtype=torch.complex128))
        oinv = lambda x: self.odds(self.sw(x, inverse=True))   # noqa: E731
        hat = lambda x: self.even(self.sw(x, mu) - self.hop(oinv(self.hop(x))))   # noqa: E731
        dot = lambda a, b: torch.vdot(a.flatten(), b.flatten())   # noqa: E731
        b = self.even(eta - self.hop(oinv(eta)))
        x, r = torch.zeros_like(b), b.clone()
        rt, p = r.clone(), r.clone()
        rho, tol = dot(rt, r), 1e-14 * b.norm()
        for it in range(1500):
            v = hat(p)
            al = rho / dot(rt, v)
            s = r - al * v
            t = hat(s)
            om = dot(t, s) / dot(t, t)
            x = x + al * p + om * s
            r = s - om * t
            if it % 20 == 19:
                r = b - hat(x)
            if r.norm() <= tol or (it % 20 == 19 and it > 400 and r.norm() <= 20 * tol):
                break
            rho_new = dot(rt, r)
            p = r + (rho_new / rho) * (al / om) * (p - om * v)
            rho = rho_new
        if (b - hat(x)).norm() > 1e-12 * b.norm():
            return None
        return x + oinv(eta - self.hop(x))


def _dfl_order(L, bs):
    """blocks in the order of the little vectors: colour 0 first"""
    nb = [n // m for n, m in zip(L, bs)]
    col = np.indices(nb).reshape(4, -1).sum(axis=0) & 1
    return np.argsort(col, kind="stable")


def _block_fields(f, L, bs):
    """[V, 4, 3] -> [blocks, components], blocks in little-vector order"""
    nb = [n // m for n, m in zip(L, bs)]
    x = f.reshape(nb[0], bs[0], nb[1], bs[1], nb[2], bs[2], nb[3], bs[3], 12)
    x = x.permute(0, 2, 4, 6, 1, 3, 5, 7, 8).reshape(math.prod(nb), -1)
    return x[torch.from_numpy(_dfl_order(L, bs)).cuda()]


def _unblock(x, L, bs):
    nb = [n // m for n, m in zip(L, bs)]
    f = torch.empty_like(x)
    f[torch.from_numpy(_dfl_order(L, bs)).cuda()] = x
    f = f.reshape(*nb, *bs, 12).permute(0, 4, 1, 5, 2, 6, 3, 7, 8)
    return f.reshape(-1, 4, 3)


def exact(case, seed):
    L, bs = _dims(case)
    p = case["path"]
    if p == "transfer":
        # block orthonormal basis: QR with a positive diagonal
        B = torch.stack([_block_fields(_modes(L, l).to(torch.complex128), L, bs) for l in range(case["ns"])], 2)
        for l in range(case["ns"]):
            for _ in range(2):
                if l:
                    c = B[:, :, :l].conj().transpose(1, 2) @ B[:, :, l:l + 1]
                    B[:, :, l] -= (B[:, :, :l] @ c)[..., 0]
            B[:, :, l] /= B[:, :, l].norm(dim=1, keepdim=True)
        vd, fs = [], []
        for k in range(case["nr"]):
            f = _block_fields(_source(L, seed, k, 32).to(torch.complex128), L, bs)
            c = (B.conj() * f[:, :, None]).sum(1)
            vd.append(torch.view_as_real(c).reshape(-1))
            v = torch.view_as_complex(_normal(_gen(37, seed, k), c.numel() * 2).view(-1, case["ns"], 2))
            fs.append(_to_storage(_unblock((B * v[:, None, :]).sum(2), L, bs), L))
        return [vd, fs]
    D = _Plain(case)
    mu = case["mu"]
    if p == "dirac":
        s = _source(L, seed, 0, case["prec"]).to(torch.complex128)
        return _to_device(D.apply(case["op"], mu, s), L, bs, case["prec"])
    if p == "host":
        return _to_storage(D.apply("Dw", mu, _source(L, seed, 0, 64)), L)
    if p == "sap":
        out = D.sap(mu, case["nmr"], case["ncy"], _source(L, seed, 0, 32).to(torch.complex128))
        return [_to_device(x, L, bs, 32) for x in out]
    out = [D.solve(mu, _source(L, seed, k, 64)) for k in range(case.get("nr", 1))]
    return None if any(x is None for x in out) else [_to_device(x, L, bs, 64) for x in out]
