// Wilson-Dirac operator kernels (full, even/odd pieces, Dwhat) in FP64 and
// FP32 on the block-major layout of qcd.cuh.
//
// One templated body (pair_body) covers every operator of the reference's
// modules/dirac/Dw_dble.c and modules/dirac/Dw.c.  Per site x of the selected
// parity it forms
//     acc  = (A(x) + i mu_x gamma5) s(x)                    if OP_SW
//     h    = -1/2 sum_mu [hop terms of t around x]          if OP_HOP/OP_HOPSUB
//     h    = A(x)^-1 h                                      if OP_INV
//     acc += h  (OP_HOP)   or   acc -= h  (OP_HOPSUB)
//     r(x) = acc  or  r(x) += acc (OP_ACC)
// which gives
//     Dw    : all sites, SW|HOP            (Dw_dble.c:1377)
//     Dwee  : even,      SW                (Dw_dble.c:1507)
//     Dwoo  : odd,       SW                (Dw_dble.c:1565)
//     Dwoe  : odd,       HOP               (Dw_dble.c:1627)
//     Dweo  : even,      HOPSUB|ACC        (Dw_dble.c:1705, subtracts from r)
//     Dwhat : odd HOP|INV into a scratch field, then even SW|HOPSUB
//                                          (Dw_dble.c:1792)
// It is a pure gather: each pair of lanes reads the spinors of its site's 8
// neighbours and the 8 links that touch the site, and writes only that site.
#include "lib.h"
#include "pairs.cuh"
#include <algorithm>

namespace qcd {

enum { OP_SW = 1, OP_HOP = 2, OP_HOPSUB = 4, OP_INV = 8, OP_ACC = 16, OP_SUB = 32 };

// L2 residency in FP64: the SW matrices are read once per application and the
// output is not read back by the launch, so both go through L2 with the
// evict-first policy (ld.global.cs, and st.global.cs in eo_store).  The
// neighbour spinors and links, read by several CTAs at different times (block
// faces), then stay in L2 longer.  FP32 reads and writes with the default policy.
__device__ __forceinline__ void load_pauli_cs(const double2 *base, int chunk, int half, int s, int vbh,
                                              double u[36]) {
  const double2 *p = base + ((size_t)chunk * 36 + 18 * half) * vbh + s;
#pragma unroll
  for (int k = 0; k < 18; k++) {
    const double2 v = __ldcs(p + (size_t)k * vbh);
    u[2 * k] = v.x;
    u[2 * k + 1] = v.y;
  }
}
// ------------------------------------------------------------------------
// Two lanes per site (pairs.cuh): a warp takes 16 sites of one parity of a
// block, warp w of a launch parity w & 1 when both are done.
//
// Bound by the latency of the gathers.  Against one thread per site (the same
// 128 registers and 16 warps per SM) a lane's chain is half as long and its
// four hops' loads are in flight together.  FP32: Dw on 32^3x64 335 -> 275 us (5.1
// TB/s of the 672 algorithmic bytes per site), on 48x24^3 with 6^4 blocks 107.6
// -> 94.5 us, on 8^4 8.2 -> 4.1 us; five CTAs per SM (96 registers) 312 and
// 98.8 us, six (80) 294 and 94.3 us.
constexpr int DW_MINB32 = 4;
__device__ __forceinline__ void pair_load_sw(const void *m, int chunk, int half, int s, int vbh, float (&a)[36]) {
  Store<float>::load_pauli(m, chunk, half, s, vbh, a);
}
__device__ __forceinline__ void pair_load_sw(const void *m, int chunk, int half, int s, int vbh, double (&a)[36]) {
  load_pauli_cs((const double2 *)m, chunk, half, s, vbh, a);
}
// the sums up, lo of a role's four hops of t around site (p, blk, si)
template <class LP, int DD, typename R = typename LP::R, typename E = typename Prec<R>::E>
__device__ __forceinline__ void role_hops(const Geom &g, const DDGeom &dg, const Site &x, int p, int blk, int si,
                                          const EoRole &ro, const E *__restrict__ t, const void *__restrict__ u,
                                          Pair3<R> &up, Pair3<R> &lo) {
  const int vbh = g.vbh, chunk = p * g.nbl + blk;
  // the two directions of the role: coordinates and blocks
  const int ya = ro.role ? x.y[2] : x.y[0], yb = ro.role ? x.y[1] : x.y[3];
  const int na = ro.role ? x.n[2] : x.n[0], nba = ro.role ? g.nb[2] : g.nb[0], bsta = ro.role ? g.bstr[2] : g.bstr[0];
  const int nb = ro.role ? x.n[1] : x.n[3], nbb = ro.role ? g.nb[1] : g.nb[3], bstb = ro.role ? g.bstr[1] : 1;
  auto fwd = [&](int y, int n, int nbk, int bstr, int bs, int str, int &c2, int &s2) {
    const bool in = y + 1 < bs;
    s2 = (in ? x.l + str : x.l - (bs - 1) * str) >> 1;
    c2 = (1 - p) * g.nbl + blk + (in ? 0 : (n + 1 < nbk ? bstr : -(nbk - 1) * bstr));
  };
  auto bwd = [&](int y, int n, int nbk, int bstr, int bs, int str, int &c2, int &s2) {
    const bool in = y > 0;
    s2 = (in ? x.l - str : x.l + (bs - 1) * str) >> 1;
    c2 = (1 - p) * g.nbl + blk + (in ? 0 : (n > 0 ? -bstr : (nbk - 1) * bstr));
  };
  // global time coordinate: the time links at x0 = N0-1 carry the boundary sign
  const int x0 = (DD ? dg.x0off : 0) + x.n[0] * g.bs[0] + x.y[0], xlast = (DD ? dg.N0 : g.L[0]) - 1;
  pair_zero(up);
  pair_zero(lo);
  int c2, s2;
  if (DD && ro.role == 0 && na + 1 == nba && ya + 1 == ro.bsa) {
    eo_face_fwd<LP>(dg.hup, face_sites(g), face_index_of(g, x.n, x.y), u, vbh, chunk, si, x0 == xlast, up, lo);
  } else {
    fwd(ya, na, nba, bsta, ro.bsa, ro.stra, c2, s2);
    eo_field_hop<0, 0, LP>(ro, t, u, vbh, c2, s2, chunk, ro.mua, si, (R)ro.s, ro.role == 0 && x0 == xlast, up, lo);
  }
  if (DD && ro.role == 0 && na == 0 && ya == 0) {
    eo_face_bwd(dg.hdn, face_sites(g), face_index_of(g, x.n, x.y), up, lo);
  } else {
    bwd(ya, na, nba, bsta, ro.bsa, ro.stra, c2, s2);
    eo_field_hop<0, 1, LP>(ro, t, u, vbh, c2, s2, c2, ro.mua, s2, (R)-ro.s, ro.role == 0 && x0 == 0, up, lo);
  }
  fwd(yb, nb, nbb, bstb, ro.bsb, ro.strb, c2, s2);
  eo_field_hop<1, 0, LP>(ro, t, u, vbh, c2, s2, chunk, ro.mub, si, (R)ro.t, false, up, lo);
  bwd(yb, nb, nbb, bstb, ro.bsb, ro.strb, c2, s2);
  eo_field_hop<1, 1, LP>(ro, t, u, vbh, c2, s2, c2, ro.mub, s2, (R)-ro.t, false, up, lo);
}

template <int OPS, int PAR, class LP, int DD, typename R = typename LP::R, typename E = typename Prec<R>::E>
__device__ __forceinline__ void pair_body(const Geom &g, const DDGeom &dg, int w, const E *__restrict__ s,
                                          const E *__restrict__ t, E *r, const void *__restrict__ u,
                                          const void *__restrict__ sw, const void *__restrict__ swinv, R mu_e, R mu_o,
                                          const int *__restrict__ sched, const E *__restrict__ sub) {
  const int lane = threadIdx.x & 31, vbh = g.vbh, tpb = (vbh + 15) >> 4;
  const int p = PAR == 2 ? w & 1 : PAR, wb = PAR == 2 ? w >> 1 : w;
  int blk = wb / tpb;
  const int s0 = (wb - blk * tpb) * 16 + (lane & 15);
  if (sched) blk = __ldg(sched + blk);
  // lanes beyond the last site work on it again (every lane takes part in
  // the exchange) and store nothing
  const bool act = s0 < vbh;
  const int si = act ? s0 : vbh - 1;
  Site x;
  site_decode(g, p, blk, si, x);
  const int chunk = p * g.nbl + blk;
  const EoRole ro = eo_role(g, lane >> 4);
  const size_t own = ((size_t)chunk * 2 + ro.role) * Prec<R>::NP * vbh + si;   // this role's chirality of a field
  cpx<R> acc[6], h[6];
  if (OPS & (OP_HOP | OP_HOPSUB)) {
    Pair3<R> up, lo;
    role_hops<LP, DD>(g, dg, x, p, blk, si, ro, t, u, up, lo);
    if (DD) __syncwarp();
    eo_exchange(ro.role, up, lo, h);
#pragma unroll
    for (int i = 0; i < 6; i++) h[i] = mk<R>((R)-0.5 * h[i].re, (R)-0.5 * h[i].im);
    if (OPS & OP_INV) {
      cpx<R> q[6];
      R m[36];
      pair_load_sw(swinv, chunk, ro.role, si, vbh, m);
      eo_pauli((R)0, m, h, q);
#pragma unroll
      for (int i = 0; i < 6; i++) h[i] = q[i];
    }
  }
  if (OPS & OP_SW) {
    cpx<R> in[6];
    eo_load(s + own, vbh, in);
    R m[36];
    pair_load_sw(sw, chunk, ro.role, si, vbh, m);
    const R mu = p == 0 ? mu_e : mu_o;
    eo_pauli(ro.role ? -mu : mu, m, in, acc);
  } else {
#pragma unroll
    for (int i = 0; i < 6; i++) acc[i] = mk<R>(0, 0);
  }
  if (OPS & (OP_HOP | OP_HOPSUB)) {
    const R sg = (OPS & OP_HOP) ? (R)1 : (R)-1;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      acc[i] = mk<R>(fm(sg, h[i].re, acc[i].re), fm(sg, h[i].im, acc[i].im));
    }
  }
  if (!act) return;
  if (OPS & (OP_SUB | OP_ACC)) {   // r = sub - acc (the residual update of a preconditioner), r += acc
    cpx<R> v[6];
    eo_load(((OPS & OP_SUB) ? sub : (const E *)r) + own, vbh, v);
    const R sg = (OPS & OP_SUB) ? (R)-1 : (R)1;
#pragma unroll
    for (int i = 0; i < 6; i++) acc[i] = mk<R>(fm(sg, acc[i].re, v[i].re), fm(sg, acc[i].im, v[i].im));
  }
  eo_store(r + own, vbh, acc);
}

// CTAs of four warps for nblk blocks (a multiple of eight in every use, since
// every lattice direction has an even number of blocks: no warp is left over)
static unsigned pair_grid(const Geom &g, int par, int nblk) {
  return (unsigned)(((g.vbh + 15) / 16) * nblk * (par == 2 ? 2 : 1) / 4);
}
__device__ __forceinline__ int pair_warp(int cta) { return cta * 4 + (threadIdx.x >> 5); }

// CTAs per SM: FP32 4 of 128 registers (see above); FP64 with hops 3 of 168,
// which run faster than 2 of up to 226 (620 against 696 us for Dw on 32^3x64,
// 42.8 and 46.9 us on 32x16^3) and than 4 of 128 (666 and 46.1 us), unless the
// launch fits the chip in one wave of 4 and not of 3: Dwhat on 16^4 (512 CTAs)
// 26.6 us with 3, 24.6 with 4, on 24^2x16x8 (576) 28.7 and 25.3 us; beyond that
// wave, on 32x16^3 (1024), 56.3 and 57.9 us.  Without hops the kernel has 120
// registers anyway.
template <int OPS, int PAR, class LP, int MINB, typename R = typename LP::R, typename E = typename Prec<R>::E>
__global__ void __launch_bounds__(128, MINB)
    dirac_pair_kernel(Geom g, const E *__restrict__ s, const E *__restrict__ t, E *r, const void *__restrict__ u,
                      const void *__restrict__ sw, const void *__restrict__ swinv, R mu_e, R mu_o,
                      const int *__restrict__ sched, const E *__restrict__ sub) {
  pair_body<OPS, PAR, LP, 0>(g, DDGeom{0, 0, nullptr, nullptr}, pair_warp(blockIdx.x), s, t, r, u, sw, swinv, mu_e, mu_o,
                             sched, sub);
}
template <int OPS, int PAR, class LP, typename R = typename LP::R, typename E = typename Prec<R>::E>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 3 : DW_MINB32)
    dirac_pair_dd_kernel(Geom g, DDGeom dg, const E *__restrict__ s, const E *__restrict__ t, E *r,
                         const void *__restrict__ u, const void *__restrict__ sw, const void *__restrict__ swinv,
                         R mu_e, R mu_o, const int *__restrict__ sched) {
  pair_body<OPS, PAR, LP, 1>(g, dg, pair_warp(blockIdx.x), s, t, r, u, sw, swinv, mu_e, mu_o, sched, (const E *)nullptr);
}

// Hops alone in FP32 (OP_HOP, or OP_HOPSUB | OP_ACC) with one lane per site,
// which goes through the two roles one after the other: the same sums in the
// same order as with two lanes.  Without SW matrices there is little to do per
// byte, and what counts are the bytes that the gathers have in flight; a lane's
// eight neighbours and links are twice those of a lane of a pair.  Dwoe with
// 12-real links on 32^3x64 145 us with two lanes, 113 with one (its 288 bytes
// per site take 92), on 48x24^3 with 6^4 blocks 51.7 and 41.9 us; Dweo 156 and
// 135 us, 53.5 and 49.2 us; on 32^3x64 with 18-real links 158 and 137 us, 170 and
// 161 us.
template <int OPS, int PAR, class LP, int DD, typename R = typename LP::R, typename E = typename Prec<R>::E>
__device__ __forceinline__ void site_body(const Geom &g, const DDGeom &dg, int n, const E *__restrict__ t, E *r,
                                          const void *__restrict__ u, const int *__restrict__ sched) {
  const int i = blockIdx.x * 128 + threadIdx.x, vbh = g.vbh;
  if (i >= n) return;
  int blk = i / vbh;
  const int si = i - blk * vbh;
  if (sched) blk = __ldg(sched + blk);
  Site x;
  site_decode(g, PAR, blk, si, x);
  Pair3<R> up[2], lo[2];
#pragma unroll
  for (int k = 0; k < 2; k++) role_hops<LP, DD>(g, dg, x, PAR, blk, si, eo_role(g, k), t, u, up[k], lo[k]);
  E *own = r + ((size_t)PAR * g.nbl + blk) * 2 * Prec<R>::NP * vbh + si;
  const R sg = (OPS & OP_HOP) ? (R)-0.5 : (R)0.5;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    cpx<R> h[6];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const auto ar = k ? mk2(lo[1].re[c].y, lo[1].re[c].x) : up[0].re[c], br = k ? lo[0].re[c] : up[1].re[c];
      const auto ai = k ? mk2(lo[1].im[c].y, lo[1].im[c].x) : up[0].im[c], bi = k ? lo[0].im[c] : up[1].im[c];
      h[c] = mk<R>(fm(sg, ar.x + br.x, (R)0), fm(sg, ai.x + bi.x, (R)0));   // (no negative zeros, as in pair_body)
      h[3 + c] = mk<R>(fm(sg, ar.y + br.y, (R)0), fm(sg, ai.y + bi.y, (R)0));
    }
    E *o = own + (size_t)k * Prec<R>::NP * vbh;
    if (OPS & OP_ACC) {
      cpx<R> v[6];
      eo_load((const E *)o, vbh, v);
#pragma unroll
      for (int j = 0; j < 6; j++) h[j] = mk<R>(h[j].re + v[j].re, h[j].im + v[j].im);
    }
    eo_store(o, vbh, h);
  }
}
template <int OPS, int PAR, class LP, int MINB, typename E = typename Prec<typename LP::R>::E>
__global__ void __launch_bounds__(128, MINB)
    dirac_site_kernel(Geom g, int n, const E *__restrict__ t, E *r, const void *__restrict__ u,
                      const int *__restrict__ sched) {
  site_body<OPS, PAR, LP, 0>(g, DDGeom{0, 0, nullptr, nullptr}, n, t, r, u, sched);
}
template <int OPS, int PAR, class LP, typename E = typename Prec<typename LP::R>::E>
__global__ void __launch_bounds__(128, DW_MINB32)
    dirac_site_dd_kernel(Geom g, DDGeom dg, int n, const E *__restrict__ t, E *r, const void *__restrict__ u,
                         const int *__restrict__ sched) {
  site_body<OPS, PAR, LP, 1>(g, dg, n, t, r, u, sched);
}

// Several systems of the batched solvers (SAP_MS at most): r_j = sub_j -
// Dw(mu_j) s_j, FP32, in one launch whose CTAs of one tile of sites
// are adjacent (CTA x: tile x / n, system x % n), so the links and SW
// matrices of a tile serve every system while they are in L2.
struct DwSys {
  const void *s[SAP_MS];
  void *r[SAP_MS];
  const void *sub[SAP_MS];
  float mu[SAP_MS];
};
template <class LP>
__global__ void __launch_bounds__(128, DW_MINB32)
    dirac_sys_kernel(Geom g, DwSys f, int n, const void *__restrict__ u, const void *__restrict__ sw, int eoflg,
                     const int *__restrict__ sched) {
  const int j = blockIdx.x % n;
  // selected without indexing the parameter arrays by a variable (which
  // would copy them to local memory)
  const void *s = f.s[0], *sb = f.sub[0];
  void *r = f.r[0];
  float mu = f.mu[0];
#pragma unroll
  for (int q = 1; q < SAP_MS; q++)
    if (j == q) {
      s = f.s[q];
      r = f.r[q];
      sb = f.sub[q];
      mu = f.mu[q];
    }
  pair_body<OP_SW | OP_HOP | OP_SUB, 2, LP, 0>(g, DDGeom{0, 0, nullptr, nullptr}, pair_warp(blockIdx.x / n),
                                               (const float4 *)s, (const float4 *)s, (float4 *)r, u, sw, nullptr, mu,
                                               eoflg ? 0.0f : mu, sched, (const float4 *)sb);
}

// the operators on the listed blocks (all of them in the order sched), two
// lanes per site, with the links u read by LP
template <int OPS, int PAR, class LP>
static void launch_pairs(const Ctx &c, const DDGeom *dg, const void *s, const void *t, void *r, const void *u,
                         typename LP::R mu_e, typename LP::R mu_o, const int *sched, int nblk, const void *sub,
                         cudaStream_t st) {
  using R = typename LP::R;
  using E = typename Prec<R>::E;
  constexpr bool F64 = sizeof(R) == 8;
  const unsigned nb = pair_grid(c.g, PAR, nblk);
  const void *sw = F64 ? (const void *)c.swd : (const void *)c.sw32;
  const void *swinv = F64 ? (const void *)c.swd_inv : (const void *)c.sw32_inv;
  const E *es = (const E *)s, *et = (const E *)t, *eb = (const E *)sub;
  E *er = (E *)r;
  if constexpr (!F64 && !(OPS & (OP_SW | OP_INV))) {
    // hops alone: one lane per site, unless that leaves half of the warp slots
    // empty (8^4: 6.2 us with one lane, 4.2 with two; 16^4: 6.2 and 6.2 to 6.9).
    // CTAs per SM: Dwoe 4 (3 are 8 % slower on 32^3x64, 5 are 5 %).  Dweo,
    // which reads its output too, 3 with 18-real links (161 us on 32^3x64; 4:
    // 168), with 12-real ones 5 (135 us; 4: 137, 3: 143), or 3 if the launch is
    // one wave then (16^4: 6.2 us; 4: 7.2, 5: 8.2)
    const int n = nblk * c.g.vbh, ns = (n + 127) / 128;
    if (nb > 2 * 148) {
      constexpr int MINB = OPS & OP_ACC ? (LP::NRAW == 12 ? 5 : 3) : 4;
      if (dg) dirac_site_dd_kernel<OPS, PAR, LP><<<ns, 128, 0, st>>>(c.g, *dg, n, et, er, u, sched);
      else if (ns > 3 * 148) dirac_site_kernel<OPS, PAR, LP, MINB><<<ns, 128, 0, st>>>(c.g, n, et, er, u, sched);
      else dirac_site_kernel<OPS, PAR, LP, MINB == 5 ? 3 : MINB><<<ns, 128, 0, st>>>(c.g, n, et, er, u, sched);
      return;
    }
  }
  if constexpr (!(OPS & OP_SUB)) {
    if (dg) {
      dirac_pair_dd_kernel<OPS, PAR, LP><<<nb, 128, 0, st>>>(c.g, *dg, es, et, er, u, sw, swinv, mu_e, mu_o, sched);
      return;
    }
  }
  if constexpr (F64 && (OPS & (OP_HOP | OP_HOPSUB))) {
    if (nb <= 3 * 148 || nb > 4 * 148) {
      dirac_pair_kernel<OPS, PAR, LP, 3><<<nb, 128, 0, st>>>(c.g, es, et, er, u, sw, swinv, mu_e, mu_o, sched, eb);
      return;
    }
  }
  dirac_pair_kernel<OPS, PAR, LP, 4><<<nb, 128, 0, st>>>(c.g, es, et, er, u, sw, swinv, mu_e, mu_o, sched, eb);
}

// With domain decomposition the operators that hop (all but Dwee, Dwoo)
// first exchange the x0-faces of the field they hop on.
template <typename R, int OPS, int PAR>
static void launch(const Ctx &c, const void *s, const void *t, void *r, R mu_e, R mu_o, cudaStream_t st) {
  constexpr bool HOPS = (OPS & (OP_HOP | OP_HOPSUB)) != 0;
  const void *u = sizeof(R) == 8 ? (const void *)c.ud : (const void *)c.u32;
  const void *u12 = nullptr;
  if constexpr (sizeof(R) == 4 && HOPS) u12 = links12(const_cast<Ctx &>(c), st);
  DDGeom g = c.ddg;
  const bool dd = HOPS && dd_on(c);
  if (dd && dd_faces(const_cast<Ctx &>(c), sizeof(R) == 8 ? 64 : 32, t, u12 ? u12 : u, u12 != nullptr, st, g))
    return;
  if constexpr (sizeof(R) == 4) {
    if (u12) launch_pairs<OPS, PAR, EoTwoRow>(c, dd ? &g : nullptr, s, t, r, u12, mu_e, mu_o, c.sched, c.g.nbl, nullptr, st);
    else launch_pairs<OPS, PAR, EoFull>(c, dd ? &g : nullptr, s, t, r, u, mu_e, mu_o, c.sched, c.g.nbl, nullptr, st);
  } else {
    launch_pairs<OPS, PAR, EoDouble>(c, dd ? &g : nullptr, s, t, r, u, mu_e, mu_o, c.sched, c.g.nbl, nullptr, st);
  }
}

// op: 0 Dw, 1 Dwee, 2 Dwoo, 3 Dwoe, 4 Dweo, 5 Dwhat.  tmp: a scratch field
// (same precision) used by Dwhat for its odd intermediate.
template <typename R>
int dirac_op(const Ctx &c, int op, R mu, const void *s, void *r, void *tmp, cudaStream_t st) {
  R muo = c.eoflg ? (R)0 : mu;
  switch (op) {
    case 0: launch<R, OP_SW | OP_HOP, 2>(c, s, s, r, mu, muo, st); break;
    case 1: launch<R, OP_SW, 0>(c, s, s, r, mu, mu, st); break;
    case 2: launch<R, OP_SW, 1>(c, s, s, r, muo, muo, st); break;
    case 3: launch<R, OP_HOP, 1>(c, s, s, r, mu, mu, st); break;
    case 4: launch<R, OP_HOPSUB | OP_ACC, 0>(c, s, s, r, mu, mu, st); break;
    case 5:
      launch<R, OP_HOP | OP_INV, 1>(c, s, s, tmp, (R)0, (R)0, st);
      launch<R, OP_SW | OP_HOPSUB, 0>(c, s, tmp, r, mu, mu, st);
      break;
    default: return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Dw on all sites of the listed blocks (block indices in device memory):
// the launches of dirac_op(0) with the block list as the traversal order
template <typename R>
int dirac_dw_blocks(const Ctx &c, R mu, const void *s, void *r, const int *blocks, int nblk, cudaStream_t st) {
  const R muo = c.eoflg ? (R)0 : mu;
  constexpr int OPS = OP_SW | OP_HOP;
  if constexpr (sizeof(R) == 4) {
    if (const void *u12 = links12(const_cast<Ctx &>(c), st))
      launch_pairs<OPS, 2, EoTwoRow>(c, nullptr, s, s, r, u12, mu, muo, blocks, nblk, nullptr, st);
    else
      launch_pairs<OPS, 2, EoFull>(c, nullptr, s, s, r, c.u32, mu, muo, blocks, nblk, nullptr, st);
  } else {
    launch_pairs<OPS, 2, EoDouble>(c, nullptr, s, s, r, c.ud, mu, muo, blocks, nblk, nullptr, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
template int dirac_dw_blocks<double>(const Ctx &, double, const void *, void *, const int *, int, cudaStream_t);
template int dirac_dw_blocks<float>(const Ctx &, float, const void *, void *, const int *, int, cudaStream_t);

// Dwhat_dble with the odd intermediate in a caller-provided half-field
// (odd chunks only, volh sites); used by the allocation-free entry point.
int dwhat_dble_halfscratch(const Ctx &c, double mu, const void *s, void *r, void *odd_scratch, cudaStream_t st) {
  // the full field whose odd half the scratch is
  double2 *odd = (double2 *)odd_scratch - (size_t)c.g.nbl * 12 * c.g.vbh;
  launch_pairs<OP_HOP | OP_INV, 1, EoDouble>(c, nullptr, s, s, odd, c.ud, 0.0, 0.0, nullptr, c.g.nbl, nullptr, st);
  launch_pairs<OP_SW | OP_HOPSUB, 0, EoDouble>(c, nullptr, s, odd, r, c.ud, mu, mu, nullptr, c.g.nbl, nullptr, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// r[j] = Dw(mu) s[j], or r[j] = sub[j] - Dw s[j] when sub is given (the
// residual update of the deflated preconditioner fused into the operator),
// for n FP32 fields
int dirac_multi32(const Ctx &c, int n, float mu, void *const *sv, void *const *rv, void *const *subv,
                  cudaStream_t st) {
  // one single-field launch per field, the residual update fused into its
  // store: on B200 the four-field kernel (links and SW read once, 255
  // registers, 8 warps per SM) took 13.0 ms for four fields at 48^3x96 with
  // 6^4 blocks against 6.9 ms for four single-field launches
  const float muo = c.eoflg ? 0.0f : mu;
  const void *u12 = links12(const_cast<Ctx &>(c), st);
  constexpr int OPS = OP_SW | OP_HOP;
  for (int j = 0; j < n; j++) {
    const void *b = subv ? subv[j] : nullptr;
    if (b && u12) launch_pairs<OPS | OP_SUB, 2, EoTwoRow>(c, nullptr, sv[j], sv[j], rv[j], u12, mu, muo, c.sched, c.g.nbl, b, st);
    else if (b) launch_pairs<OPS | OP_SUB, 2, EoFull>(c, nullptr, sv[j], sv[j], rv[j], c.u32, mu, muo, c.sched, c.g.nbl, b, st);
    else if (u12) launch_pairs<OPS, 2, EoTwoRow>(c, nullptr, sv[j], sv[j], rv[j], u12, mu, muo, c.sched, c.g.nbl, b, st);
    else launch_pairs<OPS, 2, EoFull>(c, nullptr, sv[j], sv[j], rv[j], c.u32, mu, muo, c.sched, c.g.nbl, b, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// r_j = sub_j - Dw(mu_j) s_j for n <= SAP_MS systems in one launch (FP32)
int dirac_sys32(const Ctx &c, int n, const float *mu, void *const *sv, void *const *rv, void *const *subv,
                cudaStream_t st) {
  if (n < 1 || n > SAP_MS) return -2;
  DwSys f;
  for (int j = 0; j < SAP_MS; j++) {
    const int k = j < n ? j : 0;
    f.s[j] = sv[k];
    f.r[j] = rv[k];
    f.sub[j] = subv[k];
    f.mu[j] = mu[k];
  }
  const unsigned nb = pair_grid(c.g, 2, c.g.nbl) * n;
  const void *u12 = links12(const_cast<Ctx &>(c), st);
  if (u12) dirac_sys_kernel<EoTwoRow><<<nb, 128, 0, st>>>(c.g, f, n, u12, c.sw32, c.eoflg, c.sched);
  else dirac_sys_kernel<EoFull><<<nb, 128, 0, st>>>(c.g, f, n, c.u32, c.sw32, c.eoflg, c.sched);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

template int dirac_op<double>(const Ctx &, int, double, const void *, void *, void *, cudaStream_t);
template int dirac_op<float>(const Ctx &, int, float, const void *, void *, void *, cudaStream_t);

}  // namespace qcd
