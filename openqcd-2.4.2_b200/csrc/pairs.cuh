// Hop terms with two lanes per site (the Dirac operators, the SAP block solver
// and its boundary update).  A lane has a role:
//   role 0 takes the hops in directions 0 and 3, whose projectors couple
//          component c1 to c3 and c2 to c4, and owns the upper chirality
//          (c1, c2) of the result;
//   role 1 takes directions 2 and 1, which couple c1 to c4 and c2 to c3, and
//          owns the lower chirality (c3, c4).
// Both roles run the same code: the first direction of a role has the factor
// +-1 in its projector, the second +-i, and the sign of the second half
// spinor is an operand.  Lanes l and l + 16 of a warp hold the two roles of a
// site, so that 16 consecutive sites of a plane are read together.
#pragma once
#include "qcd.cuh"
#include <cuda_fp16.h>

namespace qcd {

// All products are written as fused multiply-adds in a fixed order, so that
// every kernel that includes this rounds alike (the ranks of a domain
// decomposition reproduce the results of one rank bit for bit).

// The types of a precision: a pair of reals, the element of a spinor plane and
// the planes of a chirality
template <typename R> struct Prec;
template <> struct Prec<float> {
  using V = float2;
  using E = float4;
  static constexpr int NP = 3;
};
template <> struct Prec<double> {
  using V = double2;
  using E = double2;
  static constexpr int NP = 6;
};
__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float fm(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fm(double a, double b, double c) { return fma(a, b, c); }

template <typename R> struct Pair3 {
  typename Prec<R>::V re[3], im[3];   // .x, .y: the two half spinors
};
template <typename R> __device__ __forceinline__ void pair_zero(Pair3<R> &a) {
#pragma unroll
  for (int k = 0; k < 3; k++) a.re[k] = a.im[k] = mk2((R)0, (R)0);
}

// One hop: h = upper + g lower (FI = 0) or upper + i g lower (FI = 1) of the
// neighbour's record, c = U h (DAG = 0) or U^dagger h, up += c, lo += g c
// (FI = 0) or -i g c.  The sign g is +1 (forward, DAG = 0) or -1 (backward)
// for the first half spinor and gy for the second.
template <int FI, int DAG, typename R, typename V>
__device__ __forceinline__ void hop_project(V ar, V ai, V br, V bi, R gy, V &hr, V &hi) {
  const R gx = DAG ? (R)-1 : (R)1;
  hr = FI ? mk2(ar.x - gx * bi.x, fm(-gy, bi.y, ar.y)) : mk2(ar.x + gx * br.x, fm(gy, br.y, ar.y));
  hi = FI ? mk2(ai.x + gx * br.x, fm(gy, br.y, ai.y)) : mk2(ai.x + gx * bi.x, fm(gy, bi.y, ai.y));
}
// up += c, lo += g c or -i g c for colour i of c
template <int FI, int DAG, typename R, typename V>
__device__ __forceinline__ void hop_add(int i, V cr, V ci, R gy, Pair3<R> &up, Pair3<R> &lo) {
  const R gx = DAG ? (R)-1 : (R)1;
  up.re[i].x += cr.x;
  up.re[i].y += cr.y;
  up.im[i].x += ci.x;
  up.im[i].y += ci.y;
  lo.re[i].x += gx * (FI ? ci.x : cr.x);
  lo.re[i].y = fm(gy, FI ? ci.y : cr.y, lo.re[i].y);
  lo.im[i].x += FI ? -gx * cr.x : gx * ci.x;
  lo.im[i].y = fm(FI ? -gy : gy, FI ? cr.y : ci.y, lo.im[i].y);
}
template <int FI, int DAG, typename R, typename V>
__device__ __forceinline__ void hop_link(const V (&hr)[3], const V (&hi)[3], const R (&u)[18], R gy, Pair3<R> &up,
                                         Pair3<R> &lo) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    V cr = mk2((R)0, (R)0), ci = cr;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int e = DAG ? 3 * j + i : 3 * i + j;
      const R x = u[2 * e], y = DAG ? -u[2 * e + 1] : u[2 * e + 1];
      cr.x = j ? fm(x, hr[j].x, cr.x) : x * hr[j].x;
      cr.y = j ? fm(x, hr[j].y, cr.y) : x * hr[j].y;
      ci.x = j ? fm(x, hi[j].x, ci.x) : x * hi[j].x;
      ci.y = j ? fm(x, hi[j].y, ci.y) : x * hi[j].y;
      cr.x = fm(-y, hi[j].x, cr.x);
      cr.y = fm(-y, hi[j].y, cr.y);
      ci.x = fm(y, hr[j].x, ci.x);
      ci.y = fm(y, hr[j].y, ci.y);
    }
    hop_add<FI, DAG>(i, cr, ci, gy, up, lo);
  }
}
// Links: how many reals are read, and the 18 made of them.  EoTwoRow reads
// the first two rows (12 reals, three float4 planes of two complex entries
// each) and rebuilds the third as the complex conjugate of their cross product,
// exact for SU(3) and negated for a link that carries the antiperiodic
// time-boundary sign (the library checks every link for this relation, with
// the sign its position implies, before it reads 12-real links); EoFull reads
// FP32 links of 18 reals, EoHalf FP16 ones, EoDouble FP64 ones.
struct EoTwoRow {
  using R = float;
  static constexpr int NRAW = 12;
  __device__ __forceinline__ static void load(const void *u, int chunk, int mu, int s, int vbh, float (&r)[NRAW]) {
    const float4 *q = (const float4 *)u + ((size_t)chunk * 4 + mu) * 3 * vbh + s;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const float4 v = __ldg(q + (size_t)j * vbh);
      r[4 * j] = v.x;
      r[4 * j + 1] = v.y;
      r[4 * j + 2] = v.z;
      r[4 * j + 3] = v.w;
    }
  }
  __device__ __forceinline__ static void expand(const float (&r)[NRAW], float (&u)[18]) {
#pragma unroll
    for (int k = 0; k < 12; k++) u[k] = r[k];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int a = 2 * ((j + 1) % 3), b = 2 * ((j + 2) % 3);
      u[12 + 2 * j] = fmaf(-r[a + 1], r[7 + b], r[a] * r[6 + b]) - fmaf(-r[b + 1], r[7 + a], r[b] * r[6 + a]);
      u[13 + 2 * j] = fmaf(r[b + 1], r[6 + a], r[b] * r[7 + a]) - fmaf(r[a + 1], r[6 + b], r[a] * r[7 + b]);
    }
  }
  // a time link that carries the boundary sign: the rebuilt row changes sign
  __device__ __forceinline__ static void sign(bool neg, float (&u)[18]) {
#pragma unroll
    for (int k = 12; k < 18; k++) u[k] = neg ? -u[k] : u[k];
  }
};
struct EoFull {
  using R = float;
  static constexpr int NRAW = 18;
  __device__ __forceinline__ static void load(const void *u, int chunk, int mu, int s, int vbh, float (&r)[NRAW]) {
    const float2 *p = (const float2 *)u + ((size_t)chunk * 4 + mu) * 9 * vbh + s;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const float2 v = __ldg(p + (size_t)k * vbh);
      r[2 * k] = v.x;
      r[2 * k + 1] = v.y;
    }
  }
  __device__ __forceinline__ static void expand(const float (&r)[NRAW], float (&u)[18]) {
#pragma unroll
    for (int k = 0; k < 18; k++) u[k] = r[k];
  }
  __device__ __forceinline__ static void sign(bool, float (&)[18]) {}   // stored with its sign
};
struct EoHalf {
  using R = float;
  static constexpr int NRAW = 9;
  __device__ __forceinline__ static void load(const void *u, int chunk, int mu, int s, int vbh, float (&r)[NRAW]) {
    const float *p = (const float *)u + ((size_t)chunk * 4 + mu) * 9 * vbh + s;   // __half2 planes
#pragma unroll
    for (int k = 0; k < 9; k++) r[k] = __ldg(p + (size_t)k * vbh);
  }
  __device__ __forceinline__ static void expand(const float (&r)[NRAW], float (&u)[18]) {
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&r[k]));
      u[2 * k] = f.x;
      u[2 * k + 1] = f.y;
    }
  }
  __device__ __forceinline__ static void sign(bool, float (&)[18]) {}
};

struct EoDouble {
  using R = double;
  static constexpr int NRAW = 18;
  __device__ __forceinline__ static void load(const void *u, int chunk, int mu, int s, int vbh, double (&r)[NRAW]) {
    const double2 *p = (const double2 *)u + ((size_t)chunk * 4 + mu) * 9 * vbh + s;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double2 v = __ldg(p + (size_t)k * vbh);
      r[2 * k] = v.x;
      r[2 * k + 1] = v.y;
    }
  }
  __device__ __forceinline__ static void expand(const double (&r)[NRAW], double (&u)[18]) {
#pragma unroll
    for (int k = 0; k < 18; k++) u[k] = r[k];
  }
  __device__ __forceinline__ static void sign(bool, double (&)[18]) {}   // stored with its sign
};

// What a lane keeps of its role: the two directions and their signs
struct EoRole {
  int role, mua, mub, stra, strb, bsa, bsb;
  float s, t;   // signs of the second half spinor
};

__device__ __forceinline__ EoRole eo_role(const Geom &g, int role) {
  EoRole ro;
  ro.role = role;
  ro.mua = role ? 2 : 0;
  ro.mub = role ? 1 : 3;
  ro.stra = role ? g.lstr[2] : g.lstr[0];
  ro.strb = role ? g.lstr[1] : 1;
  ro.bsa = role ? g.bs[2] : g.bs[0];
  ro.bsb = role ? g.bs[1] : g.bs[3];
  // signs of the two half spinors: direction 0 (+,+), 2 (+,-), 3 (+,-), 1 (+,+)
  ro.s = role ? -1.0f : 1.0f;
  ro.t = role ? 1.0f : -1.0f;
  return ro;
}

// each role sends the other one its part of the other's chirality; o: the
// sum of the own one.  Every lane of the warp takes part.
template <typename R>
__device__ __forceinline__ void eo_exchange(int role, const Pair3<R> &up, const Pair3<R> &lo, cpx<R> (&o)[6]) {
  using V = typename Prec<R>::V;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const V sr = role ? up.re[k] : lo.re[k], si = role ? up.im[k] : lo.im[k];
    const V kr = role ? mk2(lo.re[k].y, lo.re[k].x) : up.re[k];
    const V ki = role ? mk2(lo.im[k].y, lo.im[k].x) : up.im[k];
    o[k].re = kr.x + __shfl_xor_sync(0xffffffffu, sr.x, 16);
    o[3 + k].re = kr.y + __shfl_xor_sync(0xffffffffu, sr.y, 16);
    o[k].im = ki.x + __shfl_xor_sync(0xffffffffu, si.x, 16);
    o[3 + k].im = ki.y + __shfl_xor_sync(0xffffffffu, si.y, 16);
  }
}

// one chirality of a field: f points at its first plane and the site
__device__ __forceinline__ void eo_load(const float4 *f, int vbh, cpx<float> (&v)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const float4 q = f[(size_t)j * vbh];
    v[2 * j] = mk<float>(q.x, q.y);
    v[2 * j + 1] = mk<float>(q.z, q.w);
  }
}
__device__ __forceinline__ void eo_store(float4 *f, int vbh, const cpx<float> (&v)[6]) {
#pragma unroll
  for (int j = 0; j < 3; j++)
    f[(size_t)j * vbh] = make_float4(v[2 * j].re, v[2 * j].im, v[2 * j + 1].re, v[2 * j + 1].im);
}
__device__ __forceinline__ void eo_load(const double2 *f, int vbh, cpx<double> (&v)[6]) {
#pragma unroll
  for (int j = 0; j < 6; j++) {
    const double2 q = f[(size_t)j * vbh];
    v[j] = mk<double>(q.x, q.y);
  }
}
// (evict first: the operators' output is not read back by the launch; Dwhat's
// odd intermediate, which its second launch reads, goes the same way)
__device__ __forceinline__ void eo_store(double2 *f, int vbh, const cpx<double> (&v)[6]) {
#pragma unroll
  for (int j = 0; j < 6; j++) __stcs(f + (size_t)j * vbh, make_double2(v[j].re, v[j].im));
}

// r = (A + i mu) w for one chirality of a site, A packed as in mul_pauli.  The
// entries off the diagonal, which are small, are summed first and the
// diagonal's product is added to them last, so that few roundings are of the
// size of the result.
template <typename R>
__device__ __forceinline__ void eo_pauli(R mu, const R (&u)[36], const cpx<R> (&w)[6], cpx<R> (&r)[6]) {
#pragma unroll
  for (int i = 0; i < 6; i++) r[i] = mk<R>(-mu * w[i].im, mu * w[i].re);
  int k = 6;
#pragma unroll
  for (int i = 0; i < 6; i++)
#pragma unroll
    for (int j = i + 1; j < 6; j++) {
      const R x = u[k], y = u[k + 1];
      k += 2;
      r[i].re = fm(-y, w[j].im, fm(x, w[j].re, r[i].re));
      r[i].im = fm(y, w[j].re, fm(x, w[j].im, r[i].im));
      r[j].re = fm(y, w[i].im, fm(x, w[i].re, r[j].re));
      r[j].im = fm(-y, w[i].re, fm(x, w[i].im, r[j].im));
    }
#pragma unroll
  for (int i = 0; i < 6; i++) r[i] = mk<R>(fm(u[i], w[i].re, r[i].re), fm(u[i], w[i].im, r[i].im));
}

// One hop of a field in global memory: neighbour (c2, s2), link (cl, mu, sl)
__device__ __forceinline__ void eo_components(const float4 *f, int vbh, float2 (&c)[12]) {
#pragma unroll
  for (int j = 0; j < 6; j++) {
    const float4 q = __ldg(f + (size_t)j * vbh);
    c[2 * j] = make_float2(q.x, q.y);
    c[2 * j + 1] = make_float2(q.z, q.w);
  }
}
__device__ __forceinline__ void eo_components(const double2 *f, int vbh, double2 (&c)[12]) {
#pragma unroll
  for (int j = 0; j < 12; j++) c[j] = __ldg(f + (size_t)j * vbh);
}
template <int FI, int DAG, class LP, typename R = typename LP::R>
__device__ __forceinline__ void eo_field_hop(const EoRole &ro, const typename Prec<R>::E *phi, const void *links,
                                             int vbh, int c2, int s2, int cl, int mu, int sl, R gy, bool neg,
                                             Pair3<R> &up, Pair3<R> &lo) {
  R r[LP::NRAW], u[18];
  typename Prec<R>::V c[12], hr[3], hi[3];
  eo_components(phi + (size_t)c2 * 2 * Prec<R>::NP * vbh + s2, vbh, c);
  LP::load(links, cl, mu, sl, vbh, r);
  LP::expand(r, u);
  LP::sign(neg, u);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const auto l1 = ro.role ? c[9 + k] : c[6 + k], l2 = ro.role ? c[6 + k] : c[9 + k];
    hop_project<FI, DAG>(mk2(c[k].x, c[3 + k].x), mk2(c[k].y, c[3 + k].y), mk2(l1.x, l2.x), mk2(l1.y, l2.y), gy, hr[k],
                         hi[k]);
  }
  hop_link<FI, DAG>(hr, hi, u, gy, up, lo);
}

// The x0-hops across a rank boundary (domain decomposition), from the half
// spinors of the exchanged faces: the forward hop U(x,0)(1 - g0) s(x+0) needs
// the neighbour's projection h = (s1 + s3, s2 + s4), the backward hop
// U(x-0,0)^dag (1 + g0) s(x-0) the product U^dag (s1 - s3, s2 - s4), which the
// rank holding the link forms.  Role 0 only.
template <class LP, typename R = typename LP::R>
__device__ __forceinline__ void eo_face_fwd(const void *face, int F, int f, const void *links, int vbh, int chunk,
                                            int s, bool neg, Pair3<R> &up, Pair3<R> &lo) {
  vec3<R> h0, h1;
  Half<R>::load(face, F, f, h0, h1);
  R r[LP::NRAW], u[18];
  LP::load(links, chunk, 0, s, vbh, r);
  LP::expand(r, u);
  LP::sign(neg, u);
  typename Prec<R>::V hr[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    hr[k] = mk2(h0.c[k].re, h1.c[k].re);
    hi[k] = mk2(h0.c[k].im, h1.c[k].im);
  }
  hop_link<0, 0>(hr, hi, u, (R)1, up, lo);
}
template <typename R>
__device__ __forceinline__ void eo_face_bwd(const void *face, int F, int f, Pair3<R> &up, Pair3<R> &lo) {
  vec3<R> c0, c1;
  Half<R>::load(face, F, f, c0, c1);
#pragma unroll
  for (int k = 0; k < 3; k++)
    hop_add<0, 1>(k, mk2(c0.c[k].re, c1.c[k].re), mk2(c0.c[k].im, c1.c[k].im), (R)-1, up, lo);
}
// the two faces a rank sends: the projections of its first plane, and the
// products with the time links of its last one
template <class LP, typename R = typename LP::R>
__device__ __forceinline__ void eo_face_send(int side, const spinor<R> &v, const void *links, int vbh, int chunk,
                                             int s, bool neg, vec3<R> &o0, vec3<R> &o1) {
  typename Prec<R>::V hr[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const auto ar = mk2(v.c[0].c[k].re, v.c[1].c[k].re), ai = mk2(v.c[0].c[k].im, v.c[1].c[k].im);
    const auto br = mk2(v.c[2].c[k].re, v.c[3].c[k].re), bi = mk2(v.c[2].c[k].im, v.c[3].c[k].im);
    if (side == 0) hop_project<0, 0>(ar, ai, br, bi, (R)1, hr[k], hi[k]);
    else hop_project<0, 1>(ar, ai, br, bi, (R)-1, hr[k], hi[k]);
  }
  if (side != 0) {
    R r[LP::NRAW], u[18];
    LP::load(links, chunk, 0, s, vbh, r);
    LP::expand(r, u);
    LP::sign(neg, u);
    Pair3<R> up, lo;
    pair_zero(up);
    pair_zero(lo);
    hop_link<0, 1>(hr, hi, u, (R)-1, up, lo);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      hr[k] = up.re[k];
      hi[k] = up.im[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    o0.c[k] = mk<R>(hr[k].x, hi[k].x);
    o1.c[k] = mk<R>(hr[k].y, hi[k].y);
  }
}

}  // namespace qcd
