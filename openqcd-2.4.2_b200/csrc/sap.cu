// Schwarz alternating procedure (SAP) on the device, FP32.
//
// One cycle of the reference's sap() (modules/sap/sap.c:720) visits the
// blocks of colour 0 and then those of colour 1.  For every block of the
// current colour it solves the block Dirac equation with Dirichlet (zero)
// exterior by nmr minimal-residual steps, adds the block solution phi to psi,
// replaces rho on the block by the block residual, and then subtracts the hop
// of phi out of the block from rho on the neighbouring blocks
// (Dw_bnd + sap_com, modules/dirac/Dw_bnd.c:801, modules/sap/sap_com.c:465).
// Blocks of one colour never touch each other, so they run as independent
// CTAs; the exterior update is a separate gather kernel over the sites of the
// other colour.
//
// k_sap_blocks_eo restates the even-odd preconditioned block solve of the
// reference (isolv=1: Dwoo_blk, Dweo_blk, blk_eo_mres, Dwoe_blk, Dwoo_blk,
// update_flds1/2; sap.c:740-767, blk_solv.c:1153, sap.c:618-716);
// k_sap_blocks_plain the plain one (isolv=0: blk_mres, update_flds0;
// blk_solv.c:1117, sap.c:592).  One CTA owns one block: the fields that
// neighbouring sites read (the current even residual, the odd intermediate)
// live in shared memory, links and SW matrices come through the L1 cache.
// Fields that only their own site reads (the odd start vector of the eo
// solve, the solution of the plain solve) are kept in registers or in the
// output fields, so that blocks of up to 768 sites per parity (6^4 blocks
// among them) fit into shared memory.
#include "lib.h"
#include "pairs.cuh"
#include <cstring>
#include <cuda_fp16.h>

namespace qcd {

// nsys systems (SAP_MS at most) per launch, with their own fields psi,
// rho, phi and twisted masses; the CTAs of one block are adjacent (CTA x:
// block x / nsys, system x % nsys), so the block's links and SW matrices
// are read by all systems while they are in L2.
struct SapArgs {
  Geom g;
  int colour;
  int nmr;
  int eoflg;
  float4 *psi[SAP_MS], *rho[SAP_MS], *phi[SAP_MS];
  const void *u;        // links, as the storage mode's policy reads them
  const void *sw, *swinv;
  int nsys;
  float mus[SAP_MS];
};

// the fields and twisted mass of system r of a launch
struct SapSys {
  float4 *psi, *rho, *phi;
  float mu;
};
__device__ __forceinline__ SapSys sap_sys(const SapArgs &a, int r) {
  // selected without indexing the parameter arrays by a variable (which
  // would copy them to local memory)
  SapSys y;
  y.psi = a.psi[0];
  y.rho = a.rho[0];
  y.phi = a.phi[0];
  y.mu = a.mus[0];
#pragma unroll
  for (int q = 1; q < SAP_MS; q++)
    if (r == q) {
      y.psi = a.psi[q];
      y.rho = a.rho[q];
      y.phi = a.phi[q];
      y.mu = a.mus[q];
    }
  return y;
}

// block of the given colour with in-colour index h (block lex index of the
// pair 2h, 2h+1 that has the requested parity of sum(n))
__device__ __forceinline__ int block_of_colour(const Geom &g, int h, int colour) {
  int q = 2 * h;
  int n[4];
  unpack4(__ldg(g.bcoord + q), n);
  return q + (((n[0] + n[1] + n[2] + n[3]) & 1) != colour);
}

// Storage policies of the SW matrices: SapF32 reads FP32 Pauli matrices,
// SapF16 FP16 copies of them (uint2 planes of four halves), with all
// arithmetic in FP32; the links have theirs in pairs.cuh.  The plain block
// solver (SapF32) keeps its work vectors in shared memory as 6 float4 planes
// (plane j at sm[4*(j*ld + s)], the complex components 2j and 2j+1 of site s).
// (FP16 work vectors were tried: their rounding, relative to each cycle's
// input residual, is of the size of the residual reduction of five cycles
// and cost half as many GCR iterations again.)
struct SapF32 {
  using T = float;
  __device__ __forceinline__ static spinor<float> sm_load(const float *sm, int ld, int s) {
    const float4 *p = reinterpret_cast<const float4 *>(sm);
    spinor<float> r;
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const float4 v = p[j * ld + s];
      const int k = 2 * j;
      r.c[k / 3].c[k % 3] = mk<float>(v.x, v.y);
      r.c[(k + 1) / 3].c[(k + 1) % 3] = mk<float>(v.z, v.w);
    }
    return r;
  }
  __device__ __forceinline__ static void sm_store(float *sm, int ld, int s, const spinor<float> &v) {
    float4 *p = reinterpret_cast<float4 *>(sm);
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const int k = 2 * j;
      const cpx<float> a = v.c[k / 3].c[k % 3], b = v.c[(k + 1) / 3].c[(k + 1) % 3];
      p[j * ld + s] = make_float4(a.re, a.im, b.re, b.im);
    }
  }
  __device__ __forceinline__ static su3<float> link(const void *u, int chunk, int mu, int s, int vbh) {
    return Store<float>::load_link(u, chunk, mu, s, vbh);
  }
  __device__ __forceinline__ static void pauli(const void *m, int chunk, int half, int s, int vbh, float (&u)[36]) {
    Store<float>::load_pauli(m, chunk, half, s, vbh, u);
  }
};

struct SapF16 {
  __device__ __forceinline__ static void pauli(const void *m, int chunk, int half, int s, int vbh, float (&u)[36]) {
    const uint2 *p = (const uint2 *)m + ((size_t)chunk * 18 + 9 * half) * vbh + s;
#pragma unroll
    for (int j = 0; j < 9; j++) {
      uint2 v = __ldg(p + (size_t)j * vbh);
      const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
      const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
      u[4 * j] = a.x; u[4 * j + 1] = a.y; u[4 * j + 2] = b.x; u[4 * j + 3] = b.y;
    }
  }
};

// h += H restricted to the block (Dirichlet exterior): hop terms of the
// field in shared memory (parity 1-p) around site (p, s) of block blk.
template <class P>
__device__ __forceinline__ void block_hop_acc(const SapArgs &a, int p, int blk, int s, const typename P::T *src,
                                              int ld, spinor<float> &h) {
  const Geom &g = a.g;
  int y[4];
  unpack4(__ldg(g.lcoord + p * g.vbh + s), y);
  int l = y[0] * g.lstr[0] + y[1] * g.lstr[1] + y[2] * g.lstr[2] + y[3] * g.lstr[3];
  const int chunk = p * g.nbl + blk, ochunk = (1 - p) * g.nbl + blk;
#pragma unroll
  for (int mu = 0; mu < 4; mu++) {
    if (y[mu] + 1 < g.bs[mu]) {
      int s2 = (l + g.lstr[mu]) >> 1;
      spinor<float> sp = P::sm_load(src, ld, s2);
      su3<float> uu = P::link(a.u, chunk, mu, s, g.vbh);
      hop_fwd<float>(mu, uu, sp, h);
    }
    if (y[mu] > 0) {
      int s2 = (l - g.lstr[mu]) >> 1;
      spinor<float> sm = P::sm_load(src, ld, s2);
      su3<float> uu = P::link(a.u, ochunk, mu, s2, g.vbh);
      hop_bwd<float>(mu, uu, sm, h);
    }
  }
}

// -1/2 * H restricted to the block
template <class P>
__device__ __forceinline__ spinor<float> block_hop(const SapArgs &a, int p, int blk, int s,
                                                   const typename P::T *src, int ld) {
  spinor<float> h;
  szero(h);
  block_hop_acc<P>(a, p, blk, s, src, ld, h);
  sscale<float>(h, -0.5f);
  return h;
}

// v = the block's sums of the three values v, the same in every thread, with
// one barrier.  The lanes of a warp first halve the set of values they carry
// (four, one of them unused) while they halve the set of lanes, then sum
// over the remaining lanes; every warp adds the warps' sums in the same
// order.  The callers separate two reductions by other barriers, so red is
// never overwritten while a thread still reads it.
__device__ __forceinline__ double shfl_xor_d(double x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }
__device__ __forceinline__ void block_allreduce3(double (&v)[3], double *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  // lanes with bit 4 clear keep v[0], v[1], the others v[2]; then bit 3
  const double a0 = shfl_xor_d(h16 ? v[0] : v[2], 16), a1 = shfl_xor_d(h16 ? v[1] : 0.0, 16);
  const double x0 = (h16 ? v[2] : v[0]) + a0, x1 = (h16 ? 0.0 : v[1]) + a1;
  double x = (h8 ? x1 : x0) + shfl_xor_d(h8 ? x0 : x1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) x += shfl_xor_d(x, o);
  if ((lane & 7) == 0) red[(lane >> 3) * 32 + w] = x;   // value lane / 8 of warp w
  __syncthreads();
  double t = 0.0;
  for (int j = lane & 7; j < nw; j += 8) t += red[(lane >> 3) * 32 + j];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += shfl_xor_d(t, o);
#pragma unroll
  for (int k = 0; k < 3; k++) v[k] = __shfl_sync(0xffffffffu, t, 8 * k);
}

// ------------------------------------------------------------------------
// The even-odd block solver, two lanes per site (pairs.cuh).  In shared
// memory a site's spinor is 9 float4 (144 bytes, free of bank conflicts for 8
// consecutive sites; neighbours' rows are shorter, and a fifth of the load
// wavefronts are conflicts with 4^4 and with 6^4 blocks): for each colour k the
// pairs (c1 c2), (c3 c4) and (c4 c3), real parts then imaginary parts; the
// swapped copy lets both roles load their lower components in the order of
// their projector.
//
// What bounds it: the shared-memory and L1 data path (52 % busy with 4^4 blocks
// on 32^4, 39 % with 6^4 blocks on 48x24^3; issue 55 and 45 %) and the latency of
// the link and SW reads, at 8 to 16 warps per SM; HBM is far from busy.  Against one thread per site (the form this replaces) a block of 4^4
// has 8 warps instead of 4 and each works through half the chain.  One cycle
// (nmr = 4: two launches each of this and the boundary kernel): 8^4 lattice 120
// -> 66 us, 16^4 126 -> 70 us, 32^4 841 -> 760 us (4^4 blocks); 48x24^3 (6^4
// blocks) 701 -> 664 us.  Tried and dropped: the links of the block copied into
// shared memory at the start (their reads compete with the spinors' for the
// same data path: 90.8 against 81.2 us on 8^4); the two half spinors as packed
// FP32 pairs (fma.rn.f32x2 issues at half the rate: the same time within
// 2 %); three CTAs of 256 threads per SM (80 registers, 3 % slower).
constexpr int EO_SREC = 9;   // float4 of a spinor record

template <int FI, int DAG>
__device__ __forceinline__ void hop_pair(const float4 *rec, int lo_slot, const float (&u)[18], float gy,
                                         Pair3<float> &up, Pair3<float> &lo) {
  float2 hr[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float4 a = rec[3 * k], b = rec[3 * k + lo_slot];
    hop_project<FI, DAG>(mk2(a.x, a.y), mk2(a.z, a.w), mk2(b.x, b.y), mk2(b.z, b.w), gy, hr[k], hi[k]);
  }
  hop_link<FI, DAG>(hr, hi, u, gy, up, lo);
}

// own chirality of the sum of the hops around site (p, s) within the block;
// src: spinor records of parity 1-p.  Every lane of the warp takes part.
template <class LP>
__device__ __forceinline__ void eo_hop(const SapArgs &a, const EoRole &ro, int p, int blk, int s,
                                       const float4 *src, cpx<float> (&o)[6]) {
  const Geom &g = a.g;
  int y[4];
  unpack4(__ldg(g.lcoord + p * g.vbh + s), y);
  const int l = y[0] * g.lstr[0] + y[1] * g.lstr[1] + y[2] * g.lstr[2] + y[3];
  const int ya = ro.role ? y[2] : y[0], yb = ro.role ? y[1] : y[3];
  const int chunk = p * g.nbl + blk, ochunk = (1 - p) * g.nbl + blk;
  Pair3<float> up, lo;
  pair_zero(up);
  pair_zero(lo);
  // a neighbour outside the block is one of the eight zero records at index
  // vbh8 (the one in the banks of the record it replaces), with any link: no
  // branches, so that the loads of a hop overlap the arithmetic of the one
  // before
  const int slot = 1 + ro.role, vbh = g.vbh, vbh8 = (vbh + 7) & ~7;
  const bool fa = ya + 1 < ro.bsa, ba = ya > 0, fb = yb + 1 < ro.bsb, bb = yb > 0;
  int sfa = (l + ro.stra) >> 1, sba = (l - ro.stra) >> 1, sfb = (l + ro.strb) >> 1, sbb = (l - ro.strb) >> 1;
  sfa = fa ? sfa : vbh8 + (sfa & 7);
  sba = ba ? sba : vbh8 + (sba & 7);
  sfb = fb ? sfb : vbh8 + (sfb & 7);
  sbb = bb ? sbb : vbh8 + (sbb & 7);
  float r0[LP::NRAW], r1[LP::NRAW], u[18];
  LP::load(a.u, chunk, ro.mua, s, vbh, r0);
  LP::load(a.u, ochunk, ro.mua, ba ? sba : s, vbh, r1);
  LP::expand(r0, u);
  hop_pair<0, 0>(src + sfa * EO_SREC, slot, u, ro.s, up, lo);
  LP::load(a.u, chunk, ro.mub, s, vbh, r0);
  LP::expand(r1, u);
  hop_pair<0, 1>(src + sba * EO_SREC, slot, u, -ro.s, up, lo);
  LP::load(a.u, ochunk, ro.mub, bb ? sbb : s, vbh, r1);
  LP::expand(r0, u);
  hop_pair<1, 0>(src + sfb * EO_SREC, slot, u, ro.t, up, lo);
  LP::expand(r1, u);
  hop_pair<1, 1>(src + sbb * EO_SREC, slot, u, -ro.t, up, lo);
  eo_exchange(ro.role, up, lo, o);
}

// a chirality (6 components) of a spinor record and of a field
__device__ __forceinline__ void eo_get(const float4 *rec, int role, cpx<float> (&v)[6]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float4 q = rec[3 * k + role];
    v[k] = mk<float>(q.x, q.z);
    v[3 + k] = mk<float>(q.y, q.w);
  }
}
__device__ __forceinline__ void eo_put(float4 *rec, int role, const cpx<float> (&v)[6]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    rec[3 * k + role] = make_float4(v[k].re, v[3 + k].re, v[k].im, v[3 + k].im);
    if (role) rec[3 * k + 2] = make_float4(v[3 + k].re, v[k].re, v[3 + k].im, v[k].im);
  }
}
// psi += phi on one chirality
__device__ __forceinline__ void eo_add(float4 *f, int vbh, const cpx<float> (&v)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    float4 q = f[(size_t)j * vbh];
    q.x += v[2 * j].re;
    q.y += v[2 * j].im;
    q.z += v[2 * j + 1].re;
    q.w += v[2 * j + 1].im;
    f[(size_t)j * vbh] = q;
  }
}

// rho += 1/2 h on one chirality
__device__ __forceinline__ void eo_add_half(float4 *f, int vbh, const cpx<float> (&h)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    float4 q = f[(size_t)j * vbh];
    q.x = fmaf(0.5f, h[2 * j].re, q.x);
    q.y = fmaf(0.5f, h[2 * j].im, q.y);
    q.z = fmaf(0.5f, h[2 * j + 1].re, q.z);
    q.w = fmaf(0.5f, h[2 * j + 1].im, q.w);
    f[(size_t)j * vbh] = q;
  }
}

// r = (A + i m) w for one chirality of a site
template <class P>
__device__ __forceinline__ void eo_sw(const void *m, int chunk, int half, int s, int vbh, float mu,
                                      const cpx<float> (&w)[6], cpx<float> (&r)[6]) {
  float u[36];
  P::pauli(m, chunk, half, s, vbh, u);
  eo_pauli(half == 0 ? mu : -mu, u, w, r);
}

// Own chirality of the sum of the hops of phi into site (p, blk, s) across
// the faces of its block (the block-boundary hop of the reference's
// Dw_bnd/sap_com, as a gather); false if the site lies on no face of the
// role's directions.  With domain decomposition the x0-neighbours across the
// rank boundary are half spinors in the exchanged faces.
template <class LP, int DD>
__device__ __forceinline__ bool eo_cross(const SapArgs &a, const DDGeom &dg, const EoRole &ro, const float4 *phi,
                                         int p, int blk, int s, cpx<float> (&o)[6]) {
  const Geom &g = a.g;
  Site x;
  site_decode(g, p, blk, s, x);
  const int chunk = p * g.nbl + blk;
  const int ya = ro.role ? x.y[2] : x.y[0], yb = ro.role ? x.y[1] : x.y[3];
  // global time coordinate: the time links at x0 = N0-1 carry the boundary sign
  const int x0 = (DD ? dg.x0off : 0) + x.n[0] * g.bs[0] + x.y[0], xlast = (DD ? dg.N0 : g.L[0]) - 1;
  Pair3<float> up, lo;
  pair_zero(up);
  pair_zero(lo);
  // chunk and site of the neighbour in the block across the face: block
  // coordinate n of nb, step bstr, in-block stride str
  auto across = [&](int n, int nb, int bstr, int bs, int str, int dir, int &c2, int &s2) {
    int b = blk, l = x.l;
    if (dir > 0) {
      l -= (bs - 1) * str;
      b += n + 1 < nb ? bstr : -(nb - 1) * bstr;
    } else {
      l += (bs - 1) * str;
      b += n > 0 ? -bstr : (nb - 1) * bstr;
    }
    c2 = (1 - p) * g.nbl + b;
    s2 = l >> 1;
  };
  const int na = ro.role ? x.n[2] : x.n[0], nba = ro.role ? g.nb[2] : g.nb[0], bsta = ro.role ? g.bstr[2] : g.bstr[0];
  const int nb_ = ro.role ? x.n[1] : x.n[3], nbb = ro.role ? g.nb[1] : g.nb[3], bstb = ro.role ? g.bstr[1] : 1;
  const bool fa = ya + 1 == ro.bsa, ba = ya == 0, fb = yb + 1 == ro.bsb, bb = yb == 0;
  int c2, s2;
  if (fa) {
    if (DD && ro.role == 0 && na + 1 == nba) {
      eo_face_fwd<LP>(dg.hup, face_sites(g), face_index_of(g, x.n, x.y), a.u, g.vbh, chunk, s, x0 == xlast, up, lo);
    } else {
      across(na, nba, bsta, ro.bsa, ro.stra, +1, c2, s2);
      eo_field_hop<0, 0, LP>(ro, phi, a.u, g.vbh, c2, s2, chunk, ro.mua, s, ro.s, ro.role == 0 && x0 == xlast, up, lo);
    }
  }
  if (ba) {
    if (DD && ro.role == 0 && na == 0) {
      eo_face_bwd(dg.hdn, face_sites(g), face_index_of(g, x.n, x.y), up, lo);
    } else {
      across(na, nba, bsta, ro.bsa, ro.stra, -1, c2, s2);
      eo_field_hop<0, 1, LP>(ro, phi, a.u, g.vbh, c2, s2, c2, ro.mua, s2, -ro.s, ro.role == 0 && x0 == 0, up, lo);
    }
  }
  if (fb) {
    across(nb_, nbb, bstb, ro.bsb, ro.strb, +1, c2, s2);
    eo_field_hop<1, 0, LP>(ro, phi, a.u, g.vbh, c2, s2, chunk, ro.mub, s, ro.t, false, up, lo);
  }
  if (bb) {
    across(nb_, nbb, bstb, ro.bsb, ro.strb, -1, c2, s2);
    eo_field_hop<1, 1, LP>(ro, phi, a.u, g.vbh, c2, s2, c2, ro.mub, s2, -ro.t, false, up, lo);
  }
  __syncwarp();
  eo_exchange(ro.role, up, lo, o);
  const bool any = fa || ba || fb || bb;
  return __shfl_xor_sync(0xffffffffu, (int)any, 16) || any;
}

// One CTA per block and system, NS sites per lane pair.
//   step 0         : V = W = A_o^-1 rho_o ;  S1 = rho_e - D_eo W ; S0 = 0
//                    (V is kept in phi_o until the last step)
//   step 1..nmr    : W = A_o^-1 D_oe S1 ;  s2 = (A_e + i mu g5) S1 - D_eo W ;
//                    z = (s2,S1)/|s2|^2 ; S0 += z S1 ; S1 -= z s2
//   after the last : rho_e = S1 ; phi_e = S0 ; S0 takes the place of S1
//   step nmr+1     : phi_o = V - A_o^-1 D_oe S0 ; psi += phi ;
//                    rho_o = -i mu g5 phi_o (0 with the eo flag)
// S0 and s2 stay in registers with one site per lane pair; with more of them
// S0 is kept in phi_e and s2 in rho_e (whose start value is used up in step 0).
template <int NS, class LP, class P, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_sap_blocks_eo(SapArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geom &g = a.g;
  const int vbh = g.vbh;
  const int nrec = ((vbh + 7) & ~7) + 8;   // records of a field, the zero records last
  float4 *S1 = reinterpret_cast<float4 *>(smem_raw), *W = S1 + EO_SREC * nrec;
  __shared__ double red[4 * 32];
  const SapSys y = sap_sys(a, blockIdx.x % a.nsys);
  const int blk = block_of_colour(g, blockIdx.x / a.nsys, a.colour);
  const int ce = blk, co = g.nbl + blk;
  for (int i = threadIdx.x; i < 8 * EO_SREC; i += blockDim.x)
    S1[EO_SREC * (nrec - 8) + i] = W[EO_SREC * (nrec - 8) + i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const EoRole ro = eo_role(g, lane >> 4);
  // site k of a lane pair; lanes beyond the last site work on it again and
  // store nothing
  const int sa = wp * 16 + (lane & 15);
  auto site = [&](int k, bool &act) {
    const int s = sa + k * nw * 16;
    act = s < vbh;
    return act ? s : vbh - 1;
  };
  // a chirality of a field at (chunk, s): planes 3 role .. 3 role + 2
  auto fld = [&](float4 *f, int chunk, int s) { return f + ((size_t)chunk * 6 + 3 * ro.role) * vbh + s; };
  cpx<float> S0[6];
#pragma unroll
  for (int i = 0; i < 6; i++) S0[i] = mk<float>(0.0f, 0.0f);
  const int nmr = a.nmr;
  for (int step = 0; step <= nmr + 1; step++) {
    const bool last = step == nmr + 1;
    // ---- odd sites
#pragma unroll 1
    for (int k = 0; k < NS; k++) {
      bool act;
      const int s = site(k, act);
      cpx<float> h[6], t[6];
      if (step == 0) {
        eo_load(fld(y.rho, co, s), vbh, h);
      } else {
        eo_hop<LP>(a, ro, 1, blk, s, S1, h);
#pragma unroll
        for (int i = 0; i < 6; i++) h[i] = mk<float>(-0.5f * h[i].re, -0.5f * h[i].im);
      }
      eo_sw<P>(a.swinv, co, ro.role, s, vbh, 0.0f, h, t);
      if (!act) continue;
      if (!last) {
        if (step == 0) eo_store(fld(y.phi, co, s), vbh, t);
        eo_put(W + s * EO_SREC, ro.role, t);
      } else {
        cpx<float> ph[6];
        eo_load(fld(y.phi, co, s), vbh, ph);
        // rho_o = i m phi_o with m = -mu on the upper, +mu on the lower chirality
        const float m = a.eoflg ? 0.0f : (ro.role ? y.mu : -y.mu);
#pragma unroll
        for (int i = 0; i < 6; i++) {
          ph[i].re -= t[i].re;
          ph[i].im -= t[i].im;
          t[i] = a.eoflg ? mk<float>(0.0f, 0.0f) : mk<float>(-m * ph[i].im, m * ph[i].re);
        }
        eo_store(fld(y.phi, co, s), vbh, ph);
        eo_add(fld(y.psi, co, s), vbh, ph);
        eo_store(fld(y.rho, co, s), vbh, t);
      }
    }
    if (last) break;
    __syncthreads();
    // ---- even sites
    cpx<float> s2[6];
    double v[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int k = 0; k < NS; k++) {
      bool act;
      const int s = site(k, act);
      cpx<float> b[6], s1[6];
      eo_hop<LP>(a, ro, 0, blk, s, W, b);
      if (step == 0) {
        eo_load(fld(y.rho, ce, s), vbh, s1);
#pragma unroll
        for (int i = 0; i < 6; i++) s1[i] = mk<float>(s1[i].re + 0.5f * b[i].re, s1[i].im + 0.5f * b[i].im);
        if (act) {
          eo_put(S1 + s * EO_SREC, ro.role, s1);
          if (NS > 1) eo_store(fld(y.phi, ce, s), vbh, S0);
        }
        continue;
      }
      eo_get(S1 + s * EO_SREC, ro.role, s1);
      eo_sw<P>(a.sw, ce, ro.role, s, vbh, y.mu, s1, s2);
#pragma unroll
      for (int i = 0; i < 6; i++) {
        s2[i].re += 0.5f * b[i].re;
        s2[i].im += 0.5f * b[i].im;
      }
      if (act) {
        if (NS > 1) eo_store(fld(y.rho, ce, s), vbh, s2);
#pragma unroll
        for (int i = 0; i < 6; i++) {
          const double xr = s2[i].re, xi = s2[i].im, yr = s1[i].re, yi = s1[i].im;
          v[0] += xr * xr + xi * xi;
          v[1] += xr * yr + xi * yi;
          v[2] += xr * yi - xi * yr;
        }
      }
    }
    if (step == 0) {
      __syncthreads();
      continue;
    }
    // MR coefficient (blk_solv.c:1153-1188): stop if |s2|^2 < 2 FLT_MIN;
    // every thread has the same sums and computes the same coefficient
    block_allreduce3(v, red);
    const float rr = (float)v[0];
    const bool stop = rr < 2.0f * 1.17549435e-38f;
    const float ri = 1.0f / rr, zr = stop ? 0.0f : (float)v[1] * ri, zi = stop ? 0.0f : (float)v[2] * ri;
    const bool fin = stop || step == nmr;
#pragma unroll 1
    for (int k = 0; k < NS; k++) {
      bool act;
      const int s = site(k, act);
      if (!act) continue;
      cpx<float> s1[6];
      eo_get(S1 + s * EO_SREC, ro.role, s1);
      if (NS > 1) {
        eo_load(fld(y.phi, ce, s), vbh, S0);
        eo_load(fld(y.rho, ce, s), vbh, s2);
      }
      if (!stop) {
#pragma unroll
        for (int i = 0; i < 6; i++) {
          S0[i].re += zr * s1[i].re - zi * s1[i].im;
          S0[i].im += zr * s1[i].im + zi * s1[i].re;
          s1[i].re -= zr * s2[i].re - zi * s2[i].im;
          s1[i].im -= zr * s2[i].im + zi * s2[i].re;
        }
      }
      if (NS > 1 || fin) eo_store(fld(y.phi, ce, s), vbh, S0);
      if (fin) {
        eo_store(fld(y.rho, ce, s), vbh, s1);
        eo_add(fld(y.psi, ce, s), vbh, S0);
        eo_put(S1 + s * EO_SREC, ro.role, S0);
      } else {
        eo_put(S1 + s * EO_SREC, ro.role, s1);
      }
    }
    if (fin) step = nmr;   // the reconstruction step is next
    __syncthreads();
  }
}

// Plain MR on the block Dirac operator Dw_blk + i mu g5 (twisted mass off on
// odd sites with the eo flag): all sites, s0/s1 in shared memory, Dw s1 in
// registers.  Sites are handled as (parity, s) pairs.
template <int NS>
__global__ void __launch_bounds__(256) k_sap_blocks_plain(SapArgs a) {
  using P = SapF32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *smem = reinterpret_cast<float *>(smem_raw);
  const Geom &g = a.g;
  const int ld = g.vbh;
  // planes: S1 even, S1 odd; the solution S0 accumulates in phi
  float *S1[2] = {smem, smem + 24 * ld};
  __shared__ double red[4 * 32];
  const SapSys y = sap_sys(a, blockIdx.x % a.nsys);
  const int blk = block_of_colour(g, blockIdx.x / a.nsys, a.colour);
  const int T = blockDim.x;
  const float muo = a.eoflg ? 0.0f : y.mu;

  for (int p = 0; p < 2; p++)
#pragma unroll
    for (int k = 0; k < NS; k++) {
      int s = threadIdx.x + k * T;
      if (s < g.vbh) {
        P::sm_store(S1[p], ld, s, Store<float>::load_spinor_rw(y.rho, p * g.nbl + blk, s, g.vbh));
        spinor<float> z;
        szero(z);
        Store<float>::store_spinor(y.phi, p * g.nbl + blk, s, g.vbh, z);
      }
    }
  __syncthreads();

  for (int imr = 0; imr < a.nmr; imr++) {
    spinor<float> s2[2][NS];
    double v[3] = {0.0, 0.0, 0.0};
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int k = 0; k < NS; k++) {
        int s = threadIdx.x + k * T;
        if (s < g.vbh) {
          spinor<float> s1 = P::sm_load(S1[p], ld, s);
          s2[p][k] = apply_sw_site<float>(a.sw, p * g.nbl + blk, s, g.vbh, p ? muo : y.mu, s1);
          sadd(s2[p][k], block_hop<P>(a, p, blk, s, S1[1 - p], ld));
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
              const cpx<float> x2 = s2[p][k].c[c].c[j], x1 = s1.c[c].c[j];
              v[0] += (double)x2.re * x2.re + (double)x2.im * x2.im;
              v[1] += (double)x2.re * x1.re + (double)x2.im * x1.im;
              v[2] += (double)x2.re * x1.im - (double)x2.im * x1.re;
            }
        }
      }
    block_allreduce3(v, red);
    const float rr = (float)v[0];
    if (rr < 2.0f * 1.17549435e-38f) break;
    const float ri = 1.0f / rr, zr = (float)v[1] * ri, zi = (float)v[2] * ri;
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int k = 0; k < NS; k++) {
        int s = threadIdx.x + k * T;
        if (s < g.vbh) {
          const int ch = p * g.nbl + blk;
          spinor<float> s1 = P::sm_load(S1[p], ld, s), s0 = Store<float>::load_spinor_rw(y.phi, ch, s, g.vbh);
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
              cpx<float> x1 = s1.c[c].c[j], x2 = s2[p][k].c[c].c[j];
              s0.c[c].c[j].re += zr * x1.re - zi * x1.im;
              s0.c[c].c[j].im += zr * x1.im + zi * x1.re;
              s1.c[c].c[j].re -= zr * x2.re - zi * x2.im;
              s1.c[c].c[j].im -= zr * x2.im + zi * x2.re;
            }
          Store<float>::store_spinor(y.phi, ch, s, g.vbh, s0);
          P::sm_store(S1[p], ld, s, s1);
        }
      }
    __syncthreads();
  }
  for (int p = 0; p < 2; p++)
#pragma unroll
    for (int k = 0; k < NS; k++) {
      int s = threadIdx.x + k * T;
      if (s < g.vbh) {
        int ch = p * g.nbl + blk;
        spinor<float> s0 = Store<float>::load_spinor_rw(y.phi, ch, s, g.vbh);
        spinor<float> ps = Store<float>::load_spinor_rw(y.psi, ch, s, g.vbh);
        sadd(ps, s0);
        Store<float>::store_spinor(y.psi, ch, s, g.vbh, ps);
        Store<float>::store_spinor(y.rho, ch, s, g.vbh, P::sm_load(S1[p], ld, s));
      }
    }
}

// rho(y) -= D_{y,x} phi(x) for every site y of a block of colour 1-c and every
// neighbour x of y in a (colour c) block.  Two lanes per site, as in the block
// solver: against one thread per site a launch takes 4.8 instead of 9.7 us on
// 8^4 and 6 instead of 9.7 us on 16^4 (5 CTAs per SM); on large lattices, where
// the gather's bytes in flight count, 8 CTAs per SM of 64 registers are as
// fast as one thread per site was (71 against 69 us on 32^4, 47 against 44 us on
// 48x24^3 with 6^4 blocks; with 5 CTAs 76 and 54 us).
template <class LP, int DD>
__device__ __forceinline__ void sap_bnd_body(const SapArgs &a, const DDGeom &dg) {
  const Geom &g = a.g;
  const SapSys y = sap_sys(a, blockIdx.x % a.nsys);
  const int lane = threadIdx.x & 31;
  const EoRole ro = eo_role(g, lane >> 4);
  const size_t n = (size_t)(g.nbl / 2) * g.vb;
  size_t i = ((blockIdx.x / a.nsys) * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 16 + (lane & 15);
  const bool act = i < n;
  if (!act) i = n - 1;   // every lane takes part in the exchange
  const int h = (int)(i / g.vb), r = (int)(i % g.vb);
  const int p = r >= g.vbh, s = r - p * g.vbh;
  const int blk = block_of_colour(g, h, 1 - a.colour);
  cpx<float> o[6];
  const bool any = eo_cross<LP, DD>(a, dg, ro, y.phi, p, blk, s, o);
  if (act && any) eo_add_half(y.rho + ((size_t)(p * g.nbl + blk) * 6 + 3 * ro.role) * g.vbh + s, g.vbh, o);
}

// the single-GPU kernel keeps its parameter list; the DD twin takes the
// slab's geometry with the received faces
template <class LP, int MINB>
__global__ void __launch_bounds__(128, MINB) k_sap_bnd(SapArgs a) {
  sap_bnd_body<LP, 0>(a, DDGeom{0, 0, nullptr, nullptr});
}
template <class LP>
__global__ void __launch_bounds__(128, 5) k_sap_bnd_dd(SapArgs a, DDGeom dg) {
  sap_bnd_body<LP, 1>(a, dg);
}

// DD: the x0-faces of the block solutions phi (FP32 half spinors, as
// k_dd_pack in dd.cu, with the links as the boundary hops read them)
template <class LP>
__global__ void k_sap_dd_pack(SapArgs a, DDGeom dg, void *dn, void *up) {
  const Geom &g = a.g;
  const int F = face_sites(g);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * F) return;
  const int side = i >= F, f = i - side * F;
  int chunk, s, n[4], y[4];
  face_site(g, side, f, chunk, s, n, y);
  const spinor<float> v = Store<float>::load_spinor(a.phi[0], chunk, s, g.vbh);
  vec3<float> h0, h1;
  eo_face_send<LP>(side, v, a.u, g.vbh, chunk, s, dg.x0off + g.L[0] - 1 == dg.N0 - 1, h0, h1);
  Half<float>::store(side == 0 ? dn : up, F, f, h0, h1);
}

template <class LP>
static void sap_bnd_launch(Ctx &c, SapArgs a, cudaStream_t st) {
  const size_t nb_sites = (size_t)(c.g.nbl / 2) * c.g.vb;
  const unsigned nbnd = (unsigned)((nb_sites + 63) / 64);   // 64 lane pairs per CTA
  DDGeom dg = c.ddg;
  if (!dd_on(c)) {
    // one wave of the form with more registers, or the form with more CTAs
    const unsigned n = nbnd * a.nsys;
    if (n <= 5 * 148) k_sap_bnd<LP, 5><<<n, 128, 0, st>>>(a);
    else k_sap_bnd<LP, 8><<<n, 128, 0, st>>>(a);
    return;
  }
  const int F = c.g.L[1] * c.g.L[2] * c.g.L[3];
  k_sap_dd_pack<LP><<<(unsigned)((2 * F + 127) / 128), 128, 0, st>>>(a, dg, c.dd.buf[0], c.dd.buf[1]);
  if (dd_exchange(c, (size_t)F * 48, st)) return;
  dg.hup = c.dd.buf[2];
  dg.hdn = c.dd.buf[3];
  k_sap_bnd_dd<LP><<<nbnd, 128, 0, st>>>(a, dg);
}

// dynamic shared memory a block kernel may use (of 227 KB per CTA)
static const int SAP_SMEM_MAX = 224 * 1024;

// Threads of the plain block kernel: up to three sites per thread.
static int pick_threads(int vbh, int &ns) {
  for (ns = 1; ns <= 3; ns++) {
    int t = ((vbh + ns - 1) / ns + 31) / 32 * 32;
    if (t <= 256) return t;
  }
  ns = 0;
  return 0;
}

// Launch variants of the even-odd block kernel: sites per lane pair, the
// launch bound and the register budget it implies.  The autotuner below
// times every variant that fits the block on the resident fields and keeps
// the fastest per block size, storage mode and size of launch.
// Which one wins, in us per cycle of four MR steps:
//   ns maxt (registers)   8^4, 4^4 blocks  32^4, 4^4  4x4x6x4   48x24^3, 6^4  8x4x6x8
//   1   512 (128)               72            769        -              -             -
//   1   256 (230)               66            958        -              -             -
//   3   512 (128)              130            987        -             666           364
//   1   768 (80)                80            797       132            -             -
//   2   320 (96, two CTAs/SM)  111            941       379            -             -
//   2   128 (128, four CTAs/SM)  for launches of three and more CTAs per SM (below)
// Few blocks leave one CTA to an SM: what counts is a lane's chain, and
// registers shorten it; many blocks want warps.  A block shared by a cluster
// of 2, 4 or 8 CTAs, each writing its sites into the others' shared memory,
// took 86 to 95 us where one CTA takes 66.
struct EoVariant {
  int ns, maxt;
  void (*k[3])(SapArgs);   // per storage mode
};
#define EO_KERNELS(NS, MAXT, MINB)                                                                      \
  {k_sap_blocks_eo<NS, EoFull, SapF32, MAXT, MINB>, k_sap_blocks_eo<NS, EoHalf, SapF16, MAXT, MINB>,     \
   k_sap_blocks_eo<NS, EoTwoRow, SapF32, MAXT, MINB>}
static const EoVariant kEo[] = {
    {1, 512, EO_KERNELS(1, 512, 1)}, {1, 256, EO_KERNELS(1, 256, 1)}, {3, 512, EO_KERNELS(3, 512, 1)},
    {1, 768, EO_KERNELS(1, 768, 1)}, {2, 320, EO_KERNELS(2, 320, 2)}, {2, 128, EO_KERNELS(2, 128, 4)},
};
static const int kNEo = sizeof(kEo) / sizeof(kEo[0]);
static const int kEoLarge = 2;   // the variant for every block that the shared memory holds

static size_t eo_smem(int vbh) { return (size_t)(((vbh + 7) & ~7) + 8) * 2 * EO_SREC * sizeof(float4); }
// threads of a variant, 0 if it does not fit the block size
static int eo_threads(const EoVariant &v, int vbh) {
  if (eo_smem(vbh) > (size_t)SAP_SMEM_MAX) return 0;
  const int t = 32 * ((vbh + 16 * v.ns - 1) / (16 * v.ns));
  return t > v.maxt ? 0 : t;
}

// FP16 copies of the FP32 links and Pauli matrices, same plane indexing
__global__ void k_to_half2(size_t n, const float2 *__restrict__ a, __half2 *b) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = __float22half2_rn(__ldg(a + i));
}
__global__ void k_to_half4(size_t n, const float4 *__restrict__ a, uint2 *b) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) {
    const float4 v = __ldg(a + i);
    __half2 x = __floats2half2_rn(v.x, v.y), y = __floats2half2_rn(v.z, v.w);
    b[i] = make_uint2(*reinterpret_cast<unsigned *>(&x), *reinterpret_cast<unsigned *>(&y));
  }
}

static int sap_half_fields(Ctx &c, cudaStream_t st) {
  if (c.h16_valid) return 0;
  const size_t nl = (size_t)c.g.vol * 36, np = (size_t)c.g.vol * 18;
  if (!c.u16 && cudaMalloc(&c.u16, nl * sizeof(__half2)) != cudaSuccess) return fail("out of device memory (FP16 links)");
  if (!c.sw16 && cudaMalloc(&c.sw16, np * sizeof(uint2)) != cudaSuccess) return fail("out of device memory (FP16 SW)");
  if (!c.sw16_inv && cudaMalloc(&c.sw16_inv, np * sizeof(uint2)) != cudaSuccess)
    return fail("out of device memory (FP16 SW)");
  k_to_half2<<<(unsigned)((nl + 255) / 256), 256, 0, st>>>(nl, c.u32, (__half2 *)c.u16);
  k_to_half4<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(np, c.sw32, (uint2 *)c.sw16);
  k_to_half4<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(np, c.sw32_inv, (uint2 *)c.sw16_inv);
  if (cudaGetLastError() != cudaSuccess) return fail("sap: FP16 conversion failed");
  c.h16_valid = true;
  return 0;
}

// 12-real copies of the FP32 links (first two rows) and a check that every
// link satisfies row3 = conj(row1 x row2) to FP32 accuracy, with the sign
// flipped on the time links at x0 = N0-1 (the antiperiodic boundary phase
// of bc type 3); bad[0] counts links that do not.
__global__ void k_links12(Geom g, DDGeom dg, size_t nlink, const float2 *__restrict__ u32, float4 *u12, int *bad) {
  const int vbh = g.vbh;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= nlink) return;
  const size_t cm = i / vbh, s = i - cm * vbh;   // cm = chunk*4 + mu
  const int chunk = (int)(cm >> 2), mu = (int)(cm & 3);
  const int par = chunk >= g.nbl;
  Site x;
  site_decode(g, par, chunk - par * g.nbl, (int)s, x);
  const bool neg = mu == 0 && dg.x0off + x.n[0] * g.bs[0] + x.y[0] == dg.N0 - 1;
  const float2 *p = u32 + cm * 9 * vbh + s;
  float2 e[9];
#pragma unroll
  for (int k = 0; k < 9; k++) e[k] = p[(size_t)k * vbh];
  float4 *q = u12 + cm * 3 * vbh + s;
#pragma unroll
  for (int j = 0; j < 3; j++) q[(size_t)j * vbh] = make_float4(e[2 * j].x, e[2 * j].y, e[2 * j + 1].x, e[2 * j + 1].y);
  float dp = 0.0f, dm = 0.0f;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int a = (j + 1) % 3, b = (j + 2) % 3;
    const float re = e[a].x * e[3 + b].x - e[a].y * e[3 + b].y - (e[b].x * e[3 + a].x - e[b].y * e[3 + a].y);
    const float im = -(e[a].x * e[3 + b].y + e[a].y * e[3 + b].x - (e[b].x * e[3 + a].y + e[b].y * e[3 + a].x));
    dp = fmaxf(dp, fabsf(re - e[6 + j].x) + fabsf(im - e[6 + j].y));
    dm = fmaxf(dm, fabsf(re + e[6 + j].x) + fabsf(im + e[6 + j].y));
  }
  if ((neg ? dm : dp) > 1e-5f) atomicAdd(bad, 1);
}

static int sap_link12_fields(Ctx &c, cudaStream_t st) {
  if (c.u12_valid) return 0;
  const size_t nlink = (size_t)c.g.vol * 4;
  if (!c.u12 && cudaMalloc(&c.u12, nlink * 6 * sizeof(float2)) != cudaSuccess)
    return fail("out of device memory (12-real links)");
  int *bad = nullptr;
  if (cudaMallocAsync(&bad, sizeof(int), st) != cudaSuccess) return fail("out of device memory");
  cudaMemsetAsync(bad, 0, sizeof(int), st);
  k_links12<<<(unsigned)((nlink + 255) / 256), 256, 0, st>>>(c.g, c.ddg, nlink, c.u32, (float4 *)c.u12, bad);
  int h = 0;
  cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(bad, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return fail("sap: 12-real link conversion failed");
  c.u12_ok = dd_all(c, h == 0) != 0;   // the same choice on every rank
  c.u12_valid = true;
  return 0;
}

// The 12-real FP32 links when they may be read (on, and every link passed
// the check), else null: the FP32 Dirac operators read them too.
const void *links12(Ctx &c, cudaStream_t st) {
  if (!c.sap_link12 || !c.u32) return nullptr;
  if (sap_link12_fields(c, st)) return nullptr;
  return c.u12_ok ? c.u12 : nullptr;
}

// storage mode of the even-odd block solver: 0 FP32, 1 FP16, 2 FP32 with
// 12-real links (the FP32 default when all links pass the SU(3) check)
static int sap_mode(Ctx &c, int isolv, cudaStream_t st) {
  if (!isolv) return 0;
  if (c.sap_prec == 16) return 1;
  if (!c.sap_link12) return 0;
  if (sap_link12_fields(c, st)) return -1;
  return c.u12_ok ? 2 : 0;
}

// The choice for launches of nsys systems: at most one CTA per SM, at most two,
// or more.  Several systems make a larger launch, where another variant wins.
// Six GCR steps on 16^4 with 4^4 blocks, ms: one system (128 CTAs) 2.37 with one
// CTA of 230 registers per lane on an SM, 2.60 with two of 128; two systems (256
// CTAs) 4.53 and 4.09, and 4.54 with four of two sites per lane pair; four (512)
// 9.19, 8.09 and 7.74.
static Ctx::SapTuned &sap_tuned(Ctx &c, int mode, int nsys) {
  const int n = c.g.nbl / 2 * nsys;
  return c.sap_tuned[mode][n <= 148 ? 0 : n <= 2 * 148 ? 1 : 2];
}

static void launch_eo(const Ctx &c, const SapArgs &a, int variant, int mode, cudaStream_t st) {
  const EoVariant &v = kEo[variant];
  v.k[mode]<<<c.g.nbl / 2 * a.nsys, eo_threads(v, c.g.vbh), eo_smem(c.g.vbh), st>>>(a);
}

static void launch_blocks(Ctx &c, const SapArgs &a, int isolv, int mode, cudaStream_t st) {
  const int nbh = c.g.nbl / 2;
  if (isolv) {
    launch_eo(c, a, sap_tuned(c, mode, a.nsys).variant, mode, st);
  } else {
    int ns;
    int t = pick_threads(c.g.vbh, ns);
    const size_t shm = (size_t)48 * c.g.vbh * sizeof(float);
    if (ns == 1) k_sap_blocks_plain<1><<<nbh * a.nsys, t, shm, st>>>(a);
    else if (ns == 2) k_sap_blocks_plain<2><<<nbh * a.nsys, t, shm, st>>>(a);
    else k_sap_blocks_plain<3><<<nbh * a.nsys, t, shm, st>>>(a);
  }
}

static SapArgs sap_args(Ctx &c, float mu, int nmr, int mode, void *psi, void *rho, void *phi) {
  SapArgs a;
  std::memset(&a, 0, sizeof(a));   // the bytes are also a CUDA-graph key
  const bool half = mode == 1;
  a.g = c.g;
  a.colour = 0;
  a.nmr = nmr;
  a.eoflg = c.eoflg;
  a.psi[0] = (float4 *)psi;
  a.rho[0] = (float4 *)rho;
  a.phi[0] = (float4 *)phi;
  a.nsys = 1;
  a.mus[0] = mu;
  a.u = half ? (const void *)c.u16 : (mode == 2 ? (const void *)c.u12 : (const void *)c.u32);
  a.sw = half ? (const void *)c.sw16 : (const void *)c.sw32;
  a.swinv = half ? (const void *)c.sw16_inv : (const void *)c.sw32_inv;
  return a;
}

// Time every fitting variant of the even-odd block kernel (both colours, 4
// MR steps, on random residuals) and keep the fastest: on one system if that
// makes a launch of the size in question, or on nsys of them, or as many as
// there is room for.
static int sap_autotune(Ctx &c, int mode, int nsys, cudaStream_t st) {
  Ctx::SapTuned &best = sap_tuned(c, mode, nsys);
  if (best.vbh == c.g.vbh) return 0;
  bool fits = false;
  for (int i = 0; i < kNEo; i++) {
    for (int m = 0; m < 3; m++)
      cudaFuncSetAttribute(kEo[i].k[m], cudaFuncAttributeMaxDynamicSharedMemorySize, SAP_SMEM_MAX);
    fits |= eo_threads(kEo[i], c.g.vbh) != 0;
  }
  if (!fits) return fail("sap: block too large for shared memory");
  if (&best == &sap_tuned(c, mode, 1)) nsys = 1;
  const size_t nb = spinor_bytes(c, 32);
  char *fld = nullptr;   // psi, rho and phi of every system
  while (cudaMallocAsync(&fld, 3 * nb * nsys, st) != cudaSuccess) {
    cudaGetLastError();
    fld = nullptr;
    if (nsys == 1) return fail("sap: out of device memory (autotuning)");
    nsys = (nsys + 1) / 2;
  }
  cudaMemsetAsync(fld, 0, nb * nsys, st);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int win = -1;
  float win_ms = 0.0f;
  SapArgs a = sap_args(c, 0.0f, 4, mode, fld, nullptr, nullptr);
  a.nsys = nsys;
  for (int r = 0; r < nsys; r++) {
    a.psi[r] = (float4 *)(fld + nb * r);
    a.rho[r] = (float4 *)(fld + nb * (nsys + r));
    a.phi[r] = (float4 *)(fld + nb * (2 * nsys + r));
  }
  for (int i = 0; i < kNEo; i++) {
    if (!eo_threads(kEo[i], c.g.vbh)) continue;
    float tot = 0.0f;
    for (int rep = 0; rep < 4; rep++) {
      for (int r = 0; r < nsys; r++) gen_uniform_spinor32(c, a.rho[r], 977ull + rep, st);
      cudaEventRecord(e0, st);
      for (int ic = 0; ic < 2; ic++) {
        a.colour = ic;
        launch_eo(c, a, i, mode, st);
      }
      cudaEventRecord(e1, st);
      cudaEventSynchronize(e1);
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep > 0) tot += ms;   // the first run warms up
    }
    if (cudaGetLastError() != cudaSuccess) continue;   // a variant that cannot launch is skipped
    if (win < 0 || tot < win_ms) {
      win = i;
      win_ms = tot;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(fld, st);
  if (win < 0) return fail("sap: no block-kernel variant fits this block size");
  best.variant = dd_rank0(c, win);   // every rank runs rank 0's choice (the same arithmetic everywhere)
  best.vbh = c.g.vbh;
  best.ms = win_ms / 3.0f;
  return cudaStreamSynchronize(st) == cudaSuccess ? 0 : fail("sap: CUDA error while autotuning");
}

// the choice for launches of one system, null if there is none yet
const Ctx::SapTuned *sap_tuned_one(const Ctx &c, int slot, int *threads) {
  const Ctx::SapTuned &t = sap_tuned(const_cast<Ctx &>(c), slot, 1);
  if (t.vbh != c.g.vbh) return nullptr;
  *threads = eo_threads(kEo[t.variant], c.g.vbh);
  return &t;
}

// Fix the launch variant of the even-odd block kernel for the current block
// size and storage mode (-1: tune again on the next use).
int sap_set_variant(Ctx &c, int v) {
  const int mode = sap_mode(c, 1, c.stream);
  if (mode < 0) return -1;
  if (v < 0) {
    for (auto &t : c.sap_tuned[mode]) t.vbh = 0;
    return 0;
  }
  // numbers 1 to 3 have always been good for large blocks: where their own
  // form is too small, they stand for the one with three sites per lane pair
  if (v > 0 && v < 4 && !eo_threads(kEo[v], c.g.vbh)) v = kEoLarge;
  if (v >= kNEo || !eo_threads(kEo[v], c.g.vbh))
    return fail("sap: this launch variant does not fit the block size");
  cudaFuncSetAttribute(kEo[v].k[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, SAP_SMEM_MAX);
  for (auto &t : c.sap_tuned[mode]) t = {v, c.g.vbh, 0.0f};
  return 0;
}

int sap_prepare(Ctx &c, cudaStream_t st, int nsys) {
  int ns;
  if (!pick_threads(c.g.vbh, ns)) return fail("sap: block volume too large (at most 1536 sites)");
  static bool attrs = false;
  if (!attrs) {
    cudaFuncSetAttribute(k_sap_blocks_plain<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAP_SMEM_MAX);
    cudaFuncSetAttribute(k_sap_blocks_plain<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAP_SMEM_MAX);
    cudaFuncSetAttribute(k_sap_blocks_plain<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAP_SMEM_MAX);
    attrs = true;
  }
  if (c.sap_prec == 16 && sap_half_fields(c, st)) return -1;
  const int mode = sap_mode(c, 1, st);
  if (mode < 0) return -1;
  return sap_autotune(c, mode, nsys, st);
}

// storage mode in use (for reports): 0 FP32, 1 FP16, 2 FP32 with 12-real links
int sap_storage_mode(Ctx &c) { return sap_mode(c, 1, c.stream); }

// Everything a SAP cycle needs before its launches (storage mode, derived
// link/SW copies, autotuned variant), done outside any stream capture.
// Returns the storage mode or -1.
static int sap_ready(Ctx &c, int isolv, cudaStream_t st, int nsys = 1) {
  const int mode = sap_mode(c, isolv, st);
  if (mode < 0) return -1;
  if (isolv && sap_tuned(c, mode, nsys).vbh != c.g.vbh && sap_prepare(c, st, nsys)) return -1;
  if (mode == 1 && !c.h16_valid && sap_half_fields(c, st)) return -1;
  int ns;
  if (!pick_threads(c.g.vbh, ns) || (!isolv && (size_t)48 * c.g.vbh * sizeof(float) > (size_t)SAP_SMEM_MAX))
    return fail("sap: block too large");
  return mode;
}

// the launches of ncy cycles: per cycle the block solves and boundary
// updates of colour 0, then of colour 1 (sap.c:720).  (A block kernel that
// gathered the other colour's boundary hops itself before it solved its
// blocks was tried: 78 against 80 us per cycle on 16^4, but 806 against 788 us
// on 32^4 and 7 % slower with 6^4 blocks, for want of warps to hide the
// gather's latency.)
static void sap_cycles_launch(Ctx &c, SapArgs a, int isolv, int mode, int ncy, cudaStream_t st) {
  for (int n = 0; n < 2 * ncy; n++) {
    a.colour = n & 1;
    launch_blocks(c, a, isolv, mode, st);
    if (mode == 1) sap_bnd_launch<EoHalf>(c, a, st);
    else if (mode == 2) sap_bnd_launch<EoTwoRow>(c, a, st);
    else sap_bnd_launch<EoFull>(c, a, st);
  }
}

namespace {
struct SapKey {
  int tag, isolv, mode, variant, ncy, pad;
  SapArgs a;
};
}  // namespace

// ph = sap psi (+ add), ch = base - sap rho: the output step of the
// preconditioner (base = rh, or the residual the caller's preconditioner
// started from; add = the part of the solution applied before SAP)
__global__ void k_sap_out(size_t n, const float4 *__restrict__ spsi, const float4 *__restrict__ srho,
                          const float4 *base, const float4 *__restrict__ add, float4 *ph, float4 *ch) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = base[i], b = srho[i];
  float4 p = spsi[i];
  if (add) {
    const float4 q = add[i];
    p = make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
  }
  ph[i] = p;
  ch[i] = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
}

int sap_cycles(Ctx &c, float mu, int isolv, int nmr, int ncy, void *psi, void *rho, void *phi_blk,
               cudaStream_t st) {
  const int mode = sap_ready(c, isolv, st);
  if (mode < 0) return -1;
  const SapArgs a = sap_args(c, mu, nmr, mode, psi, rho, phi_blk);
  sap_cycles_launch(c, a, isolv, mode, ncy, st);
  return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
}

// ncy cycles for n systems with the same twisted mass on their own fields
// (psi[r], rho[r] in and out, phi_blk[r] scratch), up to SAP_MS systems per
// launch; with domain decomposition one system after the other
int sap_cycles_multi(Ctx &c, int n, float mu, int isolv, int nmr, int ncy, void *const *psi, void *const *rho,
                     void *const *phi_blk, cudaStream_t st) {
  if (dd_on(c)) {
    for (int r = 0; r < n; r++)
      if (sap_cycles(c, mu, isolv, nmr, ncy, psi[r], rho[r], phi_blk[r], st)) return -1;
    return 0;
  }
  int mode = 0;
  for (int r0 = 0; r0 < n; r0 += SAP_MS) {
    const int m = n - r0 < SAP_MS ? n - r0 : SAP_MS;
    if ((mode = sap_ready(c, isolv, st, m)) < 0) return -1;
    SapArgs a = sap_args(c, mu, nmr, mode, psi[r0], rho[r0], phi_blk[r0]);
    a.nsys = m;
    for (int r = 0; r < m; r++) {
      a.psi[r] = (float4 *)psi[r0 + r];
      a.rho[r] = (float4 *)rho[r0 + r];
      a.phi[r] = (float4 *)phi_blk[r0 + r];
      a.mus[r] = mu;
    }
    sap_cycles_launch(c, a, isolv, mode, ncy, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
}

// The preconditioner of sap_gcr (sap_gcr.c:126-134): psi = ncy SAP cycles
// from psi = 0 on rho = rh, then rho = rh - rho (= D psi); with base given,
// rho = base - (final residual), and psi += add (the deflated
// preconditioner of dfl_sap_gcr.c:212-241, where SAP runs on what the
// deflation part left and base is the residual it started from).  With CUDA graphs
// on, the cycles run on three library-owned fields (solution, residual,
// block scratch) whose addresses never change, so the captured sequence
// (zero the solution, ncy x [block solves, boundary updates] per colour) is
// one graph per parameter set, replayed at every GCR step: rh is copied in
// before the replay and the results copied out after it.
// The field the captured SAP sequence reads its input from (null when CUDA
// graphs are off): a caller that computes rh can write it there directly
// and pass it as rh, which saves sap_mop the copy.
void *sap_input_field(Ctx &c) {
  if (!c.use_graphs || dd_on(c)) return nullptr;
  if (!c.sap_fld[1] && cudaMalloc(&c.sap_fld[1], spinor_bytes(c, 32)) != cudaSuccess) return nullptr;
  return c.sap_fld[1];
}

int sap_mop(Ctx &c, float mu, int isolv, int nmr, int ncy, const void *rh, void *psi, void *rho, void *phi_blk,
            cudaStream_t st, const void *base, const void *add) {
  if (!base) base = rh;
  // with domain decomposition the cycles call the exchange between their
  // launches, so they are not captured
  if (!c.use_graphs || dd_on(c)) {
    la_zero(c, 32, psi, PAR_ALL, st);
    if (rho != rh) la_copy(c, 32, rh, 32, rho, PAR_ALL, st);
    if (sap_cycles(c, mu, isolv, nmr, ncy, psi, rho, phi_blk, st)) return -1;
    la_diff(c, 32, base, rho, PAR_ALL, st);
    if (add) la_axpy(c, 32, psi, 1.0, 0.0, add, PAR_ALL, st);
    return 0;
  }
  for (int k = 0; k < 3; k++)
    if (!c.sap_fld[k] && cudaMalloc(&c.sap_fld[k], spinor_bytes(c, 32)) != cudaSuccess)
      return fail("out of device memory (SAP graph fields)");
  const int mode = sap_ready(c, isolv, st);
  if (mode < 0) return -1;
  void *spsi = c.sap_fld[0], *srho = c.sap_fld[1], *sphi = c.sap_fld[2];
  SapKey key;
  std::memset(&key, 0, sizeof(key));
  key.tag = 0x5a9;
  key.isolv = isolv;
  key.mode = mode;
  key.variant = sap_tuned(c, mode, 1).variant;
  key.ncy = ncy;
  key.a = sap_args(c, mu, nmr, mode, spsi, srho, sphi);
  if (base == srho) return fail("sap_mop: an input in the SAP input field needs a separate base");
  if (rh != srho) la_copy(c, 32, rh, 32, srho, PAR_ALL, st);
  const int rc = graph_run(c, &key, sizeof(key), st, [&]() {
    la_zero(c, 32, spsi, PAR_ALL, st);
    sap_cycles_launch(c, key.a, isolv, mode, ncy, st);
    return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
  });
  if (rc) return -1;
  const size_t n = (size_t)c.g.vol * 6;
  k_sap_out<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, (const float4 *)spsi, (const float4 *)srho,
                                                           (const float4 *)base, (const float4 *)add,
                                                           (float4 *)psi, (float4 *)rho);
  return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
}

// the fields of sap_mop_multi for n systems; false (and nothing held) when
// the device has no room for them, in which case the systems run one at a
// time
static bool sap_multi_fields(Ctx &c, int n) {
  if (c.sap_mfld_n >= n) return true;
  for (int k = 0; k < 3; k++) {
    cudaFree(c.sap_mfld[k]);
    c.sap_mfld[k] = nullptr;
  }
  c.sap_mfld_n = 0;
  for (int k = 0; k < 3; k++)
    if (cudaMalloc(&c.sap_mfld[k], (size_t)n * spinor_bytes(c, 32)) != cudaSuccess) {
      cudaGetLastError();
      for (int j = 0; j < 3; j++) {
        cudaFree(c.sap_mfld[j]);
        c.sap_mfld[j] = nullptr;
      }
      return false;
    }
  c.sap_mfld_n = n;
  return true;
}

void *sap_input_field_multi(Ctx &c, int r, int n) {
  if (!c.use_graphs || dd_on(c) || r < 0 || r >= n || n > SAP_MS || !sap_multi_fields(c, n)) return nullptr;
  return (char *)c.sap_mfld[1] + (size_t)r * spinor_bytes(c, 32);
}

// Several systems: the SAP sequence of sap_mop captured once for up to
// SAP_MS systems on library-owned fields, every block-solver and boundary
// launch covering all of them.  Without graphs, or with domain
// decomposition, the systems run one after the other through sap_mop.
int sap_mop_multi(Ctx &c, int ns, const float *mu, int isolv, int nmr, int ncy, const void *const *rh,
                  void *const *psi, void *const *rho, void *phi_blk, cudaStream_t st, const void *const *base,
                  const void *const *add) {
  if (!c.use_graphs || dd_on(c) || ns == 1 || !sap_multi_fields(c, ns < SAP_MS ? ns : SAP_MS)) {
    for (int r = 0; r < ns; r++)
      if (sap_mop(c, mu[r], isolv, nmr, ncy, rh[r], psi[r], rho[r], phi_blk, st, base ? base[r] : nullptr,
                  add ? add[r] : nullptr))
        return -1;
    return 0;
  }
  const size_t fb = spinor_bytes(c, 32);
  const size_t n = (size_t)c.g.vol * 6;   // float4 of a field
  for (int r0 = 0; r0 < ns; r0 += SAP_MS) {
    const int m = ns - r0 < SAP_MS ? ns - r0 : SAP_MS;
    const int mode = sap_ready(c, isolv, st, m);
    if (mode < 0) return -1;
    SapKey key;
    std::memset(&key, 0, sizeof(key));
    key.tag = 0x5aa;
    key.isolv = isolv;
    key.mode = mode;
    key.variant = sap_tuned(c, mode, m).variant;
    key.ncy = ncy;
    key.a = sap_args(c, mu[r0], nmr, mode, c.sap_mfld[0], c.sap_mfld[1], c.sap_mfld[2]);
    key.a.nsys = m;
    for (int r = 0; r < m; r++) {
      key.a.psi[r] = (float4 *)c.sap_mfld[0] + (size_t)r * n;
      key.a.rho[r] = (float4 *)c.sap_mfld[1] + (size_t)r * n;
      key.a.phi[r] = (float4 *)c.sap_mfld[2] + (size_t)r * n;
      key.a.mus[r] = mu[r0 + r];
    }
    for (int r = 0; r < m; r++) {
      void *in = (char *)c.sap_mfld[1] + (size_t)r * fb;
      const void *b = base && base[r0 + r] ? base[r0 + r] : rh[r0 + r];
      if (b == in) return fail("sap_mop_multi: an input in the SAP input field needs a separate base");
      if (rh[r0 + r] != in) la_copy(c, 32, rh[r0 + r], 32, in, PAR_ALL, st);
    }
    const int rc = graph_run(c, &key, sizeof(key), st, [&]() {
      cudaMemsetAsync(c.sap_mfld[0], 0, (size_t)m * fb, st);
      sap_cycles_launch(c, key.a, isolv, mode, ncy, st);
      return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
    });
    if (rc) return -1;
    for (int r = 0; r < m; r++) {
      const float4 *spsi = (const float4 *)((char *)c.sap_mfld[0] + (size_t)r * fb);
      const float4 *srho = (const float4 *)((char *)c.sap_mfld[1] + (size_t)r * fb);
      const void *b = base && base[r0 + r] ? base[r0 + r] : rh[r0 + r];
      k_sap_out<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, spsi, srho, (const float4 *)b,
                                                               (const float4 *)(add ? add[r0 + r] : nullptr),
                                                               (float4 *)psi[r0 + r], (float4 *)rho[r0 + r]);
    }
  }
  (void)phi_blk;
  return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
}

// One SAP cycle sap(mu, isolv, nmr, psi, rho) on FP32 device fields.
// phi_blk is a scratch FP32 field.  The even-odd block solver (isolv = 1)
// reads the links and SW matrices in the storage mode of sap_mode(); the
// plain solver (isolv = 0) always in FP32.
int sap_cycle(Ctx &c, float mu, int isolv, int nmr, void *psi, void *rho, void *phi_blk, cudaStream_t st) {
  const int mode = sap_ready(c, isolv, st);
  if (mode < 0) return -1;
  sap_cycles_launch(c, sap_args(c, mu, nmr, mode, psi, rho, phi_blk), isolv, mode, 1, st);
  return cudaGetLastError() == cudaSuccess ? 0 : fail("sap: launch failed");
}

}  // namespace qcd
