// Wilson-Dirac operator kernels (full, even/odd pieces, Dwhat) in FP64 and
// FP32 on the block-major layout of qcd.cuh.
//
// One templated form (FP64: dirac_body, FP32: pair_body) covers every operator of the reference's
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
// It is a pure gather: each thread (FP64) or pair of lanes (FP32) reads the
// spinors of its 8 neighbours and the 8 links that touch its site, and writes
// only its own site.
#include "lib.h"
#include "pairs.cuh"
#include "tma.cuh"
#include <algorithm>

namespace qcd {

enum { OP_SW = 1, OP_HOP = 2, OP_HOPSUB = 4, OP_INV = 8, OP_ACC = 16, OP_SUB = 32 };

// L2 residency: the SW matrices are read once per application and the
// output is not read back by the launch, so both go through L2 with the
// evict-first policy (ld.global.cs / st.global.cs, or a cache hint on the
// bulk copies).  The neighbour spinors and links, read by several CTAs at
// different times (block faces), then stay in L2 longer.
#ifndef DW_NO_HINTS
#define DW_HINTS 1
#else
#define DW_HINTS 0
#endif

__device__ __forceinline__ void load_pauli_cs(const double2 *base, int chunk, int half, int s, int vbh,
                                              double u[36]) {
  const double2 *p = base + ((size_t)chunk * 36 + 18 * half) * vbh + s;
#pragma unroll
  for (int k = 0; k < 18; k++) {
    const double2 v = DW_HINTS ? __ldcs(p + (size_t)k * vbh) : __ldg(p + (size_t)k * vbh);
    u[2 * k] = v.x;
    u[2 * k + 1] = v.y;
  }
}
__device__ __forceinline__ spinor<double> apply_sw_site_cs(const void *sw, int chunk, int s, int vbh, double mu,
                                                           const spinor<double> &in) {
  spinor<double> out;
  double u[36];
  cpx<double> w[6], r[6];
#pragma unroll
  for (int half = 0; half < 2; half++) {
    load_pauli_cs((const double2 *)sw, chunk, half, s, vbh, u);
    weyl_get(in, half, w);
    mul_pauli<double>(half == 0 ? mu : -mu, u, w, r);
    weyl_put(out, half, r);
  }
  return out;
}

__device__ __forceinline__ void store_spinor_cs(double2 *base, int chunk, int s, int vbh, const spinor<double> &r) {
  double2 *p = base + (size_t)chunk * 12 * vbh + s;
#pragma unroll
  for (int k = 0; k < 12; k++) {
    const double2 v = make_double2(r.c[k / 3].c[k % 3].re, r.c[k / 3].c[k % 3].im);
    if (DW_HINTS) __stcs(p + (size_t)k * vbh, v);
    else p[(size_t)k * vbh] = v;
  }
}

// RHALF / THALF = 1: the output r / the hop field t is a half-field holding
// only the odd chunks (chunk index counted from the first odd chunk).
// Resident CTAs per SM asked of the compiler: the FP64 kernel keeps 255
// registers (more CTAs made it spill and run slower).
#ifndef DW_MINB64
#define DW_MINB64 1
#endif
#ifndef DW_UNROLL
#define DW_UNROLL 4
#endif
constexpr int kDwUnroll = DW_UNROLL;

template <typename R, int OPS, int PAR, int RHALF, int THALF, int DD>
__device__ __forceinline__ void dirac_body(const Geom &g, const DDGeom &dg, int i, const void *__restrict__ s,
                                           const void *__restrict__ t, void *r, const void *__restrict__ u,
                                           const void *__restrict__ sw, const void *__restrict__ swinv, R mu_e,
                                           R mu_o, const int *__restrict__ sched, const void *__restrict__ sub) {
  int p, blk, si;
  if (PAR == 2) {
    if (i >= g.vol) return;
    int b = i / g.vb;
    int rr = i - b * g.vb;
    p = rr >= g.vbh;
    si = rr - p * g.vbh;
    blk = sched ? __ldg(sched + b) : b;
  } else {
    if (i >= g.volh) return;
    p = PAR;
    blk = i / g.vbh;
    si = i - blk * g.vbh;
    if (sched) blk = __ldg(sched + blk);
  }
  Site x;
  site_decode(g, p, blk, si, x);
  const int chunk = p * g.nbl + blk;

  spinor<R> acc;
  if (OPS & OP_SW) {
    spinor<R> in = Store<R>::load_spinor(s, chunk, si, g.vbh);
    acc = apply_sw_site_cs(sw, chunk, si, g.vbh, p == 0 ? mu_e : mu_o, in);
  } else {
    szero(acc);
  }

  if (OPS & (OP_HOP | OP_HOPSUB)) {
    spinor<R> h;
    szero(h);
    if constexpr (DD == 0) {
#pragma unroll kDwUnroll
      for (int mu = 0; mu < 4; mu++) {
        int c2, s2;
        site_nbr(g, x, mu, +1, c2, s2);
        {
          spinor<R> sp = Store<R>::load_spinor(t, THALF ? c2 - g.nbl : c2, s2, g.vbh);
          const su3<R> uu = Store<R>::load_link(u, chunk, mu, si, g.vbh);
          hop_fwd<R>(mu, uu, sp, h);
        }
        site_nbr(g, x, mu, -1, c2, s2);
        {
          spinor<R> sm = Store<R>::load_spinor(t, THALF ? c2 - g.nbl : c2, s2, g.vbh);
          const su3<R> uu = Store<R>::load_link(u, c2, mu, s2, g.vbh);
          hop_bwd<R>(mu, uu, sm, h);
        }
      }
    } else {
      // domain decomposition: the x0-neighbours across the rank boundary from
      // the faces
      const bool up = x.n[0] + 1 == g.nb[0] && x.y[0] + 1 == g.bs[0];
      const bool dn = x.n[0] == 0 && x.y[0] == 0;
#pragma unroll kDwUnroll
      for (int mu = 0; mu < 4; mu++) {
        int c2, s2;
        const su3<R> uu = Store<R>::load_link(u, chunk, mu, si, g.vbh);
        if (mu == 0 && up) {
          vec3<R> h0, h1;
          Half<R>::load(dg.hup, face_sites(g), face_index_of(g, x.n, x.y), h0, h1);
          dd_hop_fwd<R>(uu, h0, h1, h);
        } else {
          site_nbr(g, x, mu, +1, c2, s2);
          spinor<R> sp = Store<R>::load_spinor(t, THALF ? c2 - g.nbl : c2, s2, g.vbh);
          hop_fwd<R>(mu, uu, sp, h);
        }
        if (mu == 0 && dn) {
          vec3<R> c0, c1;
          Half<R>::load(dg.hdn, face_sites(g), face_index_of(g, x.n, x.y), c0, c1);
          dd_hop_bwd<R>(c0, c1, h);
        } else {
          site_nbr(g, x, mu, -1, c2, s2);
          spinor<R> sm = Store<R>::load_spinor(t, THALF ? c2 - g.nbl : c2, s2, g.vbh);
          const su3<R> ub = Store<R>::load_link(u, c2, mu, s2, g.vbh);
          hop_bwd<R>(mu, ub, sm, h);
        }
      }
    }
    sscale<R>(h, (R)-0.5);
    if (OPS & OP_INV) h = apply_sw_site_cs(swinv, chunk, si, g.vbh, 0.0, h);
    if (OPS & OP_HOP) sadd(acc, h);
    else ssub(acc, h);
  }

  const int rchunk = RHALF ? chunk - g.nbl : chunk;
  if (OPS & OP_SUB) {   // r = sub - acc (the residual update of a preconditioner)
    spinor<R> v = Store<R>::load_spinor(sub, rchunk, si, g.vbh);
    ssub(v, acc);
    store_spinor_cs((double2 *)r, rchunk, si, g.vbh, v);
  } else if (OPS & OP_ACC) {
    spinor<R> old = Store<R>::load_spinor_rw(r, rchunk, si, g.vbh);
    sadd(old, acc);
    Store<R>::store_spinor(r, rchunk, si, g.vbh, old);
  } else {
    store_spinor_cs((double2 *)r, rchunk, si, g.vbh, acc);
  }
}


// ------------------------------------------------------------------------
// The FP32 operators, two lanes per site (pairs.cuh): a warp takes 16 sites
// of one parity of a block, warp w of a launch parity w & 1 when both are
// done.
//
// Bound by the latency of the gathers.  Against one thread per site (the same
// 128 registers and 16 warps per SM) a lane's chain is half as long and its
// four hops' loads are in flight together: Dw on 32^3x64 335 -> 275 us (5.1
// TB/s of the 672 algorithmic bytes per site), on 48x24^3 with 6^4 blocks 107.6
// -> 94.5 us, on 8^4 8.2 -> 4.1 us; five CTAs per SM (96 registers) 312 and
// 98.8 us, six (80) 294 and 94.3 us.
#ifndef DW_MINB32
#define DW_MINB32 4
#endif
template <int OPS, int PAR, class LP, int DD>
__device__ __forceinline__ void pair_body(const Geom &g, const DDGeom &dg, int w, const float4 *__restrict__ s,
                                          const float4 *__restrict__ t, float4 *r, const void *__restrict__ u,
                                          const void *__restrict__ sw, const void *__restrict__ swinv, float mu_e,
                                          float mu_o, const int *__restrict__ sched, const float4 *__restrict__ sub) {
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
  const size_t own = ((size_t)chunk * 6 + 3 * ro.role) * vbh + si;   // this role's chirality of a field
  cpx<float> acc[6], h[6];
  if (OPS & (OP_HOP | OP_HOPSUB)) {
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
    Pair3 up, lo;
#pragma unroll
    for (int k = 0; k < 3; k++) up.re[k] = up.im[k] = lo.re[k] = lo.im[k] = make_float2(0.0f, 0.0f);
    int c2, s2;
    if (DD && ro.role == 0 && na + 1 == nba && ya + 1 == ro.bsa) {
      eo_face_fwd<LP>(dg.hup, face_sites(g), face_index_of(g, x.n, x.y), u, vbh, chunk, si, x0 == xlast, up, lo);
    } else {
      fwd(ya, na, nba, bsta, ro.bsa, ro.stra, c2, s2);
      eo_field_hop<0, 0, LP>(ro, t, u, vbh, c2, s2, chunk, ro.mua, si, ro.s, ro.role == 0 && x0 == xlast, up, lo);
    }
    if (DD && ro.role == 0 && na == 0 && ya == 0) {
      eo_face_bwd(dg.hdn, face_sites(g), face_index_of(g, x.n, x.y), up, lo);
    } else {
      bwd(ya, na, nba, bsta, ro.bsa, ro.stra, c2, s2);
      eo_field_hop<0, 1, LP>(ro, t, u, vbh, c2, s2, c2, ro.mua, s2, -ro.s, ro.role == 0 && x0 == 0, up, lo);
    }
    fwd(yb, nb, nbb, bstb, ro.bsb, ro.strb, c2, s2);
    eo_field_hop<1, 0, LP>(ro, t, u, vbh, c2, s2, chunk, ro.mub, si, ro.t, false, up, lo);
    bwd(yb, nb, nbb, bstb, ro.bsb, ro.strb, c2, s2);
    eo_field_hop<1, 1, LP>(ro, t, u, vbh, c2, s2, c2, ro.mub, s2, -ro.t, false, up, lo);
    if (DD) __syncwarp();
    eo_exchange(ro.role, up, lo, h);
#pragma unroll
    for (int i = 0; i < 6; i++) h[i] = mk<float>(-0.5f * h[i].re, -0.5f * h[i].im);
    if (OPS & OP_INV) {
      cpx<float> q[6];
      float m[36];
      Store<float>::load_pauli(swinv, chunk, ro.role, si, vbh, m);
      eo_pauli(0.0f, m, h, q);
#pragma unroll
      for (int i = 0; i < 6; i++) h[i] = q[i];
    }
  }
  if (OPS & OP_SW) {
    cpx<float> in[6];
    eo_load(s + own, vbh, in);
    float m[36];
    Store<float>::load_pauli(sw, chunk, ro.role, si, vbh, m);
    const float mu = p == 0 ? mu_e : mu_o;
    eo_pauli(ro.role ? -mu : mu, m, in, acc);
  } else {
#pragma unroll
    for (int i = 0; i < 6; i++) acc[i] = mk<float>(0.0f, 0.0f);
  }
  if (OPS & (OP_HOP | OP_HOPSUB)) {
    const float sg = (OPS & OP_HOP) ? 1.0f : -1.0f;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      acc[i] = mk<float>(fmaf(sg, h[i].re, acc[i].re), fmaf(sg, h[i].im, acc[i].im));
    }
  }
  if (!act) return;
  if (OPS & (OP_SUB | OP_ACC)) {   // r = sub - acc (the residual update of a preconditioner), r += acc
    cpx<float> v[6];
    eo_load(((OPS & OP_SUB) ? sub : (const float4 *)r) + own, vbh, v);
    const float sg = (OPS & OP_SUB) ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 6; i++) acc[i] = mk<float>(fmaf(sg, acc[i].re, v[i].re), fmaf(sg, acc[i].im, v[i].im));
  }
  eo_store(r + own, vbh, acc);
}

// CTAs of four warps for nblk blocks (a multiple of eight in every use, since
// every lattice direction has an even number of blocks: no warp is left over)
static unsigned pair_grid(const Geom &g, int par, int nblk) {
  return (unsigned)(((g.vbh + 15) / 16) * nblk * (par == 2 ? 2 : 1) / 4);
}
__device__ __forceinline__ int pair_warp(int cta) { return cta * 4 + (threadIdx.x >> 5); }

template <int OPS, int PAR, class LP>
__global__ void __launch_bounds__(128, DW_MINB32)
    dirac_pair_kernel(Geom g, const float4 *__restrict__ s, const float4 *__restrict__ t, float4 *r,
                      const void *__restrict__ u, const void *__restrict__ sw, const void *__restrict__ swinv,
                      float mu_e, float mu_o, const int *__restrict__ sched, const float4 *__restrict__ sub) {
  pair_body<OPS, PAR, LP, 0>(g, DDGeom{0, 0, nullptr, nullptr}, pair_warp(blockIdx.x), s, t, r, u, sw, swinv, mu_e, mu_o,
                             sched, sub);
}
template <int OPS, int PAR, class LP>
__global__ void __launch_bounds__(128, DW_MINB32)
    dirac_pair_dd_kernel(Geom g, DDGeom dg, const float4 *__restrict__ s, const float4 *__restrict__ t, float4 *r,
                         const void *__restrict__ u, const void *__restrict__ sw, const void *__restrict__ swinv,
                         float mu_e, float mu_o, const int *__restrict__ sched) {
  pair_body<OPS, PAR, LP, 1>(g, dg, pair_warp(blockIdx.x), s, t, r, u, sw, swinv, mu_e, mu_o, sched, nullptr);
}

// The direct FP64 kernels (the DD twin takes the slab's geometry)
template <typename R, int OPS, int PAR, int RHALF = 0, int THALF = 0>
__global__ void __launch_bounds__(128, DW_MINB64)
    dirac_kernel(Geom g, const void *__restrict__ s, const void *__restrict__ t, void *r, const void *__restrict__ u,
                 const void *__restrict__ sw, const void *__restrict__ swinv, R mu_e, R mu_o,
                 const int *__restrict__ sched, const void *__restrict__ sub) {
  dirac_body<R, OPS, PAR, RHALF, THALF, 0>(g, DDGeom{0, 0, nullptr, nullptr}, blockIdx.x * blockDim.x + threadIdx.x, s,
                                           t, r, u, sw, swinv, mu_e, mu_o, sched, sub);
}
template <typename R, int OPS, int PAR>
__global__ void __launch_bounds__(128, DW_MINB64)
    dirac_dd_kernel(Geom g, DDGeom dg, const void *__restrict__ s, const void *__restrict__ t, void *r,
                    const void *__restrict__ u, const void *__restrict__ sw, const void *__restrict__ swinv, R mu_e,
                    R mu_o, const int *__restrict__ sched) {
  dirac_body<R, OPS, PAR, 0, 0, 1>(g, dg, blockIdx.x * blockDim.x + threadIdx.x, s, t, r, u, sw, swinv, mu_e, mu_o,
                                   sched, nullptr);
}

// ------------------------------------------------------------------------
// FP64 operator with the SW matrices staged in shared memory.  A CTA owns a
// tile of DWT_TS consecutive sites of one chunk.  At its start one warp
// issues bulk asynchronous copies (cp.async.bulk with the evict-first L2
// policy, completed on an mbarrier; no multicast) of the tile's 36 SW
// planes; they are needed only after the hop loop, so the copy overlaps it
// and the SW bytes (43 % of the reads) leave the warps' load chains.
// Spinors and links are read from global memory, where the compiler hoists
// the loads of later directions.  Same arithmetic as dirac_kernel
// (operators without OP_ACC).
//
// Tried and dropped (B200, 32^3x64, 4^4 blocks): staging the forward links
// too, in two rotating stages (0.81 ms against 0.72 ms direct: the barrier
// per direction stops the load hoisting); staging the block's other-parity
// spinor chunk so that in-block hops read shared memory (0.79 ms: the copy's
// latency at the CTA start is exposed and the L2 traffic hardly fell, L1
// already caught those reads); three CTAs per SM (168 registers, 0.91 ms);
// an L2 bulk prefetch (cp.async.bulk.prefetch.L2) of the tile's links and
// other-parity spinors at the CTA start (0.72 ms against 0.66 ms); 64-site
// tiles at four CTAs per SM (the same warps per SM: 0.670 against 0.667 ms,
// and the same under the power cap).
#ifndef DWT_TILE
#define DWT_TILE 128
#endif
constexpr int DWT_TS = DWT_TILE;
#ifndef DWT_MINB
#define DWT_MINB 2
#endif
constexpr size_t DWT_SMEM = (size_t)36 * DWT_TS * sizeof(double2);     // 73,728 B

__device__ __forceinline__ spinor<double> apply_sw_smem(const double2 *sm, int t, double mu,
                                                        const spinor<double> &in) {
  spinor<double> out;
  double u[36];
  cpx<double> w[6], r[6];
#pragma unroll
  for (int half = 0; half < 2; half++) {
#pragma unroll
    for (int k = 0; k < 18; k++) {
      const double2 v = sm[(18 * half + k) * DWT_TS + t];
      u[2 * k] = v.x;
      u[2 * k + 1] = v.y;
    }
    weyl_get(in, half, w);
    mul_pauli<double>(half == 0 ? mu : -mu, u, w, r);
    weyl_put(out, half, r);
  }
  return out;
}

// h += sg (A + i mu g5) in for one Weyl half (half = 0, 1) of the input,
// with the Pauli entries read from shared memory one at a time and the
// product folded into the hop sum as it is formed, so that neither the
// whole input nor the whole product is live beside h.  The products and
// their order are those of mul_pauli.  With sg = -2 and the sum scaled by
// -1/2 afterwards (or +2 and +1/2) this equals forming (A + i mu g5) in and
// -1/2 h apart and adding (subtracting) them, rounding included: the
// scalings by 2 and 1/2 are exact.
__device__ __forceinline__ void sw_fold_half(const double2 *sm, int t, double mu, int half, const cpx<double> (&w)[6],
                                             double sg, spinor<double> &h) {
  const double m = half == 0 ? mu : -mu;
  cpx<double> r[6];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double2 d = sm[(18 * half + i) * DWT_TS + t];
    r[2 * i] = mk<double>(d.x * w[2 * i].re - m * w[2 * i].im, d.x * w[2 * i].im + m * w[2 * i].re);
    r[2 * i + 1] = mk<double>(d.y * w[2 * i + 1].re - m * w[2 * i + 1].im, d.y * w[2 * i + 1].im + m * w[2 * i + 1].re);
  }
  int e = 0;
#pragma unroll
  for (int i = 0; i < 6; i++)
#pragma unroll
    for (int j = i + 1; j < 6; j++) {
      const double2 a = sm[(18 * half + 3 + e) * DWT_TS + t];
      e++;
      r[i].re += a.x * w[j].re - a.y * w[j].im;
      r[i].im += a.x * w[j].im + a.y * w[j].re;
      r[j].re += a.x * w[i].re + a.y * w[i].im;
      r[j].im += a.x * w[i].im - a.y * w[i].re;
    }
#pragma unroll
  for (int i = 0; i < 6; i++) {
    cpx<double> &hh = h.c[2 * half + i / 3].c[i % 3];
    hh.re += sg * r[i].re;
    hh.im += sg * r[i].im;
  }
}

__device__ __forceinline__ void load_weyl(const double2 *p, size_t vbh, int half, cpx<double> (&w)[6]) {
#pragma unroll
  for (int i = 0; i < 6; i++) {
    const double2 v = __ldg(p + (size_t)(6 * half + i) * vbh);
    w[i] = mk<double>(v.x, v.y);
  }
}

// Tile t of a launch: its chunk (parity p, block blk) and first site.
__device__ __forceinline__ void staged_tile(const Geom &g, int PAR_, int t, int tpc, const int *sched, int &p,
                                           int &blk, int &si0) {
  int tile;
  if (PAR_ == 2) {
    const int b = t / (2 * tpc);
    const int rr = t - b * 2 * tpc;
    p = rr / tpc;
    tile = rr - p * tpc;
    blk = sched ? __ldg(sched + b) : b;
  } else {
    p = PAR_;
    blk = t / tpc;
    tile = t - blk * tpc;
    if (sched) blk = __ldg(sched + blk);
  }
  si0 = tile * DWT_TS;
}

// The CTA runs the tiles blockIdx.x, blockIdx.x + gridDim.x, ... (one tile
// when the grid covers them all, as the launches here do).
//
// Also tried and dropped: a persistent grid (2 CTAs per SM looping over the
// tiles) in which one warp asked L2 for the next tile's links and spinors
// with bulk prefetches while the current tile was computed: 0.90 ms against
// 0.69 ms at 32^3x64, DRAM reads 4.35 GB against 3.36 GB per launch (the
// prefetched lines were partly evicted before use).
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

template <int OPS, int PAR, int DD>
__device__ __forceinline__ void staged_body(const Geom &g, const DDGeom &dg, const double2 *__restrict__ s,
                                            const double2 *__restrict__ t, double2 *r, const double2 *__restrict__ u,
                                            const double2 *__restrict__ swm, double mu_e, double mu_o,
                                            const int *__restrict__ sched, int tpc, int ntiles, int *err,
                                            double2 *sw_s, uint64_t *bar) {
  constexpr bool HAS_SW = (OPS & (OP_SW | OP_INV)) != 0;
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_fence_init();
  }
  __syncthreads();
  unsigned phase = 0;
  for (int tl = blockIdx.x; tl < ntiles; tl += gridDim.x, phase ^= 1u) {
    int p, blk, si0;
    staged_tile(g, PAR, tl, tpc, sched, p, blk, si0);
    const int nsite = min(DWT_TS, g.vbh - si0);
    const int chunk = p * g.nbl + blk;
    const unsigned pbytes = (unsigned)nsite * 16u;
    if (HAS_SW && tid < 32) {
      if (tid == 0) mbar_expect_tx(&bar[0], 36 * pbytes);
      __syncwarp();
      const uint64_t pol = l2_policy_evict_first();
      for (int k = tid; k < 36; k += 32) {
        const double2 *src = swm + ((size_t)chunk * 36 + k) * g.vbh + si0;
        if (DW_HINTS) bulk_g2s_hint(sw_s + k * DWT_TS, src, pbytes, &bar[0], pol);
        else bulk_g2s(sw_s + k * DWT_TS, src, pbytes, &bar[0]);
      }
    }
    const bool active = tid < nsite;
    const int si = si0 + tid;
    bool ok = true;
    if (active) {
      Site x;
      site_decode(g, p, blk, si, x);
      spinor<double> h;
      szero(h);
#pragma unroll
      for (int mu = 0; mu < 4; mu++) {
        int c2, s2;
        bool fwd_done = false, bwd_done = false;
        if constexpr (DD != 0) {
          // the x0-neighbours across the rank boundary come from the faces
          if (mu == 0 && x.n[0] + 1 == g.nb[0] && x.y[0] + 1 == g.bs[0]) {
            vec3<double> h0, h1;
            Half<double>::load(dg.hup, face_sites(g), face_index_of(g, x.n, x.y), h0, h1);
            const su3<double> uu = Store<double>::load_link(u, chunk, mu, si, g.vbh);
            dd_hop_fwd<double>(uu, h0, h1, h);
            fwd_done = true;
          }
          if (mu == 0 && x.n[0] == 0 && x.y[0] == 0) {
            vec3<double> c0, c1;
            Half<double>::load(dg.hdn, face_sites(g), face_index_of(g, x.n, x.y), c0, c1);
            dd_hop_bwd<double>(c0, c1, h);
            bwd_done = true;
          }
        }
        if (!fwd_done) {
          site_nbr(g, x, mu, +1, c2, s2);
          const spinor<double> sp = Store<double>::load_spinor(t, c2, s2, g.vbh);
          const su3<double> uu = Store<double>::load_link(u, chunk, mu, si, g.vbh);
          hop_fwd<double>(mu, uu, sp, h);
        }
        if (!bwd_done) {
          site_nbr(g, x, mu, -1, c2, s2);
          const spinor<double> sm = Store<double>::load_spinor(t, c2, s2, g.vbh);
          const su3<double> ub = Store<double>::load_link(u, c2, mu, s2, g.vbh);
          hop_bwd<double>(mu, ub, sm, h);
        }
      }
      const double mux = p == 0 ? mu_e : mu_o;
      spinor<double> acc;
      if constexpr ((OPS & OP_SW) && !(OPS & OP_INV) && (OPS & (OP_HOP | OP_HOPSUB))) {
        // SW term folded into the hop sum, half by half
        const double2 *ip = s + (size_t)chunk * 12 * g.vbh + si;
        const double sg = (OPS & OP_HOP) ? -2.0 : 2.0;
        cpx<double> w[6];
        load_weyl(ip, g.vbh, 0, w);
        ok &= mbar_wait_st(&bar[0], phase, err);
        sw_fold_half(sw_s, tid, mux, 0, w, sg, h);
        load_weyl(ip, g.vbh, 1, w);
        sw_fold_half(sw_s, tid, mux, 1, w, sg, h);
        sscale<double>(h, (OPS & OP_HOP) ? -0.5 : 0.5);
        acc = h;
      } else {
        sscale<double>(h, -0.5);
        if (OPS & OP_INV) {
          ok &= mbar_wait_st(&bar[0], phase, err);
          h = apply_sw_smem(sw_s, tid, 0.0, h);
        }
        if (OPS & OP_SW) {
          const spinor<double> in = Store<double>::load_spinor(s, chunk, si, g.vbh);
          ok &= mbar_wait_st(&bar[0], phase, err);
          acc = apply_sw_smem(sw_s, tid, mux, in);
        } else {
          szero(acc);
        }
        if (OPS & OP_HOP) sadd(acc, h);
        else if (OPS & OP_HOPSUB) ssub(acc, h);
      }
      // a site whose SW matrices did not arrive keeps its old output (the
      // error flag tells the host the result is invalid)
      if (ok) store_spinor_cs(r, chunk, si, g.vbh, acc);
    }
    // every thread is done with this tile's SW matrices before the next
    // tile's copies overwrite them; if a wait gave up, thread 0 waits once
    // more (bounded) for the copies still addressed to this CTA's shared
    // memory and the CTA stops (thread 0 always has a site and waits on the
    // barrier when it was armed)
    const bool all_ok = __syncthreads_and(ok);
    if (!all_ok) {
      if (HAS_SW && tid == 0) mbar_wait_st(&bar[0], phase, err);
      return;
    }
  }
}

template <int OPS, int PAR>
__global__ void __launch_bounds__(DWT_TS, DWT_MINB)
    dirac_staged_kernel(Geom g, const double2 *__restrict__ s, const double2 *__restrict__ t, double2 *r,
                        const double2 *__restrict__ u, const double2 *__restrict__ swm, double mu_e, double mu_o,
                        const int *__restrict__ sched, int tpc, int ntiles, int *err) {
  extern __shared__ __align__(128) unsigned char dwt_smem[];
  __shared__ uint64_t bar[1];
  staged_body<OPS, PAR, 0>(g, DDGeom{0, 0, nullptr, nullptr}, s, t, r, u, swm, mu_e, mu_o, sched, tpc, ntiles, err,
                           (double2 *)dwt_smem, bar);
}
template <int OPS, int PAR>
__global__ void __launch_bounds__(DWT_TS, DWT_MINB)
    dirac_staged_dd_kernel(Geom g, DDGeom dg, const double2 *__restrict__ s, const double2 *__restrict__ t,
                           double2 *r, const double2 *__restrict__ u, const double2 *__restrict__ swm, double mu_e,
                           double mu_o, const int *__restrict__ sched, int tpc, int ntiles, int *err) {
  extern __shared__ __align__(128) unsigned char dwt_smem[];
  __shared__ uint64_t bar[1];
  staged_body<OPS, PAR, 1>(g, dg, s, t, r, u, swm, mu_e, mu_o, sched, tpc, ntiles, err, (double2 *)dwt_smem, bar);
}

template <int OPS, int PAR, int DD>
static void launch_staged(const Ctx &c, const DDGeom &dg, const void *s, const void *t, void *r, double mu_e,
                          double mu_o, cudaStream_t st) {
  const Geom &g = c.g;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(DD ? (const void *)dirac_staged_dd_kernel<OPS, PAR> : (const void *)dirac_staged_kernel<OPS, PAR>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DWT_SMEM);
    attr = true;
  }
  const int tpc = (g.vbh + DWT_TS - 1) / DWT_TS;
  const int nchunk = PAR == 2 ? 2 * g.nbl : g.nbl;
  const void *swm = (OPS & OP_INV) ? (const void *)c.swd_inv : (const void *)c.swd;
  const int ntiles = nchunk * tpc;
  if (DD)
    dirac_staged_dd_kernel<OPS, PAR><<<ntiles, DWT_TS, DWT_SMEM, st>>>(
        g, dg, (const double2 *)s, (const double2 *)t, (double2 *)r, (const double2 *)c.ud, (const double2 *)swm,
        mu_e, mu_o, c.sched, tpc, ntiles, c.d_kerr);
  else
    dirac_staged_kernel<OPS, PAR><<<ntiles, DWT_TS, DWT_SMEM, st>>>(
        g, (const double2 *)s, (const double2 *)t, (double2 *)r, (const double2 *)c.ud, (const double2 *)swm, mu_e,
        mu_o, c.sched, tpc, ntiles, c.d_kerr);
}

template <int OPS, int PAR, int DD>
static void launch_plain(const Ctx &c, const DDGeom &dg, const void *s, const void *t, void *r, double mu_e,
                         double mu_o, cudaStream_t st) {
  const Geom &g = c.g;
  const int n = PAR == 2 ? g.vol : g.volh, threads = 128;
  if (DD)
    dirac_dd_kernel<double, OPS, PAR><<<(n + threads - 1) / threads, threads, 0, st>>>(g, dg, s, t, r, c.ud, c.swd,
                                                                                      c.swd_inv, mu_e, mu_o, c.sched);
  else
    dirac_kernel<double, OPS, PAR><<<(n + threads - 1) / threads, threads, 0, st>>>(g, s, t, r, c.ud, c.swd, c.swd_inv,
                                                                                   mu_e, mu_o, c.sched, nullptr);
}

// the FP32 operators on the listed blocks (all of them in the order sched),
// with the links u read by LP
template <int OPS, int PAR, class LP>
static void launch_pairs(const Ctx &c, const DDGeom *dg, const void *s, const void *t, void *r, const void *u,
                         float mu_e, float mu_o, const int *sched, int nblk, const void *sub, cudaStream_t st) {
  const unsigned nb = pair_grid(c.g, PAR, nblk);
  if constexpr (!(OPS & OP_SUB)) {
    if (dg) {
      dirac_pair_dd_kernel<OPS, PAR, LP><<<nb, 128, 0, st>>>(c.g, *dg, (const float4 *)s, (const float4 *)t, (float4 *)r,
                                                            u, c.sw32, c.sw32_inv, mu_e, mu_o, sched);
      return;
    }
  }
  dirac_pair_kernel<OPS, PAR, LP><<<nb, 128, 0, st>>>(c.g, (const float4 *)s, (const float4 *)t, (float4 *)r, u, c.sw32,
                                                     c.sw32_inv, mu_e, mu_o, sched, (const float4 *)sub);
}

// With domain decomposition the operators that hop (all but Dwee, Dwoo)
// first exchange the x0-faces of the field they hop on.
template <typename R, int OPS, int PAR>
static void launch(const Ctx &c, const void *s, const void *t, void *r, R mu_e, R mu_o, bool inv,
                   cudaStream_t st) {
  (void)inv;
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
  } else if (!(OPS & OP_ACC) && (OPS & (OP_SW | OP_INV)) && c.dw_staged && c.d_kerr) {
    if (dd) launch_staged<OPS, PAR, 1>(c, g, s, t, r, mu_e, mu_o, st);
    else launch_staged<OPS, PAR, 0>(c, g, s, t, r, mu_e, mu_o, st);
  } else {
    if (dd) launch_plain<OPS, PAR, 1>(c, g, s, t, r, mu_e, mu_o, st);
    else launch_plain<OPS, PAR, 0>(c, g, s, t, r, mu_e, mu_o, st);
  }
}

// op: 0 Dw, 1 Dwee, 2 Dwoo, 3 Dwoe, 4 Dweo, 5 Dwhat.  tmp: a scratch field
// (same precision) used by Dwhat for its odd intermediate.
template <typename R>
int dirac_op(const Ctx &c, int op, R mu, const void *s, void *r, void *tmp, cudaStream_t st) {
  R muo = c.eoflg ? (R)0 : mu;
  switch (op) {
    case 0: launch<R, OP_SW | OP_HOP, 2>(c, s, s, r, mu, muo, false, st); break;
    case 1: launch<R, OP_SW, 0>(c, s, s, r, mu, mu, false, st); break;
    case 2: launch<R, OP_SW, 1>(c, s, s, r, muo, muo, false, st); break;
    case 3: launch<R, OP_HOP, 1>(c, s, s, r, mu, mu, false, st); break;
    case 4: launch<R, OP_HOPSUB | OP_ACC, 0>(c, s, s, r, mu, mu, false, st); break;
    case 5:
      launch<R, OP_HOP | OP_INV, 1>(c, s, s, tmp, (R)0, (R)0, true, st);
      launch<R, OP_SW | OP_HOPSUB, 0>(c, s, tmp, r, mu, mu, false, st);
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
  if (sizeof(R) == 8 && c.dw_staged && c.d_kerr) {
    static bool attr = false;
    if (!attr) {
      cudaFuncSetAttribute(dirac_staged_kernel<OPS, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DWT_SMEM);
      attr = true;
    }
    const int tpc = (c.g.vbh + DWT_TS - 1) / DWT_TS;
    const int ntiles = 2 * nblk * tpc;
    dirac_staged_kernel<OPS, 2><<<ntiles, DWT_TS, DWT_SMEM, st>>>(
        c.g, (const double2 *)s, (const double2 *)s, (double2 *)r, (const double2 *)c.ud, (const double2 *)c.swd,
        (double)mu, (double)muo, blocks, tpc, ntiles, c.d_kerr);
  } else if constexpr (sizeof(R) == 4) {
    if (const void *u12 = links12(const_cast<Ctx &>(c), st))
      launch_pairs<OPS, 2, EoTwoRow>(c, nullptr, s, s, r, u12, mu, muo, blocks, nblk, nullptr, st);
    else
      launch_pairs<OPS, 2, EoFull>(c, nullptr, s, s, r, c.u32, mu, muo, blocks, nblk, nullptr, st);
  } else {
    const int threads = 128, n = nblk * c.g.vb;
    dirac_kernel<R, OPS, 2><<<(n + threads - 1) / threads, threads, 0, st>>>(c.g, s, s, r, c.ud, c.swd, nullptr, mu, muo,
                                                                            blocks, nullptr);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
template int dirac_dw_blocks<double>(const Ctx &, double, const void *, void *, const int *, int, cudaStream_t);
template int dirac_dw_blocks<float>(const Ctx &, float, const void *, void *, const int *, int, cudaStream_t);

// Dwhat_dble with the odd intermediate in a caller-provided half-field
// (odd chunks only, volh sites); used by the allocation-free entry point.
int dwhat_dble_halfscratch(const Ctx &c, double mu, const void *s, void *r, void *odd_scratch, cudaStream_t st) {
  const int threads = 128;
  const unsigned nb = (unsigned)((c.g.volh + threads - 1) / threads);
  dirac_kernel<double, OP_HOP | OP_INV, 1, 1, 0><<<nb, threads, 0, st>>>(c.g, s, s, odd_scratch, c.ud, c.swd,
                                                                          c.swd_inv, 0.0, 0.0, nullptr, nullptr);
  dirac_kernel<double, OP_SW | OP_HOPSUB, 0, 0, 1><<<nb, threads, 0, st>>>(c.g, s, odd_scratch, r, c.ud, c.swd,
                                                                           c.swd_inv, mu, mu, nullptr, nullptr);
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
