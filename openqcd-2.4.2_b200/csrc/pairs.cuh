// FP32 hop terms with two lanes per site (the FP32 Dirac operators, the SAP block
// solver and its boundary update).  A lane has a role:
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

struct Pair3 {
  float2 re[3], im[3];   // .x, .y: the two half spinors
};

// One hop: h = upper + g lower (FI = 0) or upper + i g lower (FI = 1) of the
// neighbour's record, c = U h (DAG = 0) or U^dagger h, up += c, lo += g c
// (FI = 0) or -i g c.  The sign g is +1 (forward, DAG = 0) or -1 (backward)
// for the first half spinor and gy for the second.
template <int FI, int DAG>
__device__ __forceinline__ void hop_project(const float4 &a, const float4 &b, float gy, float2 &hr, float2 &hi) {
  const float gx = DAG ? -1.0f : 1.0f;
  hr = FI ? make_float2(a.x - gx * b.z, fmaf(-gy, b.w, a.y)) : make_float2(a.x + gx * b.x, fmaf(gy, b.y, a.y));
  hi = FI ? make_float2(a.z + gx * b.x, fmaf(gy, b.y, a.w)) : make_float2(a.z + gx * b.z, fmaf(gy, b.w, a.w));
}
// up += c, lo += g c or -i g c for colour i of c
template <int FI, int DAG>
__device__ __forceinline__ void hop_add(int i, float2 cr, float2 ci, float gy, Pair3 &up, Pair3 &lo) {
  const float gx = DAG ? -1.0f : 1.0f;
  up.re[i].x += cr.x;
  up.re[i].y += cr.y;
  up.im[i].x += ci.x;
  up.im[i].y += ci.y;
  lo.re[i].x += gx * (FI ? ci.x : cr.x);
  lo.re[i].y = fmaf(gy, FI ? ci.y : cr.y, lo.re[i].y);
  lo.im[i].x += FI ? -gx * cr.x : gx * ci.x;
  lo.im[i].y = fmaf(FI ? -gy : gy, FI ? cr.y : ci.y, lo.im[i].y);
}
template <int FI, int DAG>
__device__ __forceinline__ void hop_link(const float2 (&hr)[3], const float2 (&hi)[3], const float (&u)[18], float gy,
                                         Pair3 &up, Pair3 &lo) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    float2 cr = make_float2(0.0f, 0.0f), ci = cr;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int e = DAG ? 3 * j + i : 3 * i + j;
      const float x = u[2 * e], y = DAG ? -u[2 * e + 1] : u[2 * e + 1];
      cr.x = j ? fmaf(x, hr[j].x, cr.x) : x * hr[j].x;
      cr.y = j ? fmaf(x, hr[j].y, cr.y) : x * hr[j].y;
      ci.x = j ? fmaf(x, hi[j].x, ci.x) : x * hi[j].x;
      ci.y = j ? fmaf(x, hi[j].y, ci.y) : x * hi[j].y;
      cr.x = fmaf(-y, hi[j].x, cr.x);
      cr.y = fmaf(-y, hi[j].y, cr.y);
      ci.x = fmaf(y, hr[j].x, ci.x);
      ci.y = fmaf(y, hr[j].y, ci.y);
    }
    hop_add<FI, DAG>(i, cr, ci, gy, up, lo);
  }
}
// Links: how many reals are read, and the 18 made of them.  EoTwoRow reads
// the first two rows and rebuilds the third (load_link12), EoFull FP32 links
// of 18 reals, EoHalf FP16 ones.
struct EoTwoRow {
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
__device__ __forceinline__ void eo_exchange(int role, const Pair3 &up, const Pair3 &lo, cpx<float> (&o)[6]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float2 sr = role ? up.re[k] : lo.re[k], si = role ? up.im[k] : lo.im[k];
    const float2 kr = role ? make_float2(lo.re[k].y, lo.re[k].x) : up.re[k];
    const float2 ki = role ? make_float2(lo.im[k].y, lo.im[k].x) : up.im[k];
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
// r = (A + i mu) w for one chirality of a site, A packed as in mul_pauli; the
// two products of an entry are summed before they are added (as one chain of
// multiply-adds the operator's error was a fifth larger)
__device__ __forceinline__ void eo_pauli(float mu, const float (&u)[36], const cpx<float> (&w)[6], cpx<float> (&r)[6]) {
#pragma unroll
  for (int i = 0; i < 6; i++) r[i] = mk<float>(fmaf(-mu, w[i].im, u[i] * w[i].re), fmaf(mu, w[i].re, u[i] * w[i].im));
  int k = 6;
#pragma unroll
  for (int i = 0; i < 6; i++)
#pragma unroll
    for (int j = i + 1; j < 6; j++) {
      const float x = u[k], y = u[k + 1];
      k += 2;
      r[i].re += fmaf(-y, w[j].im, x * w[j].re);
      r[i].im += fmaf(y, w[j].re, x * w[j].im);
      r[j].re += fmaf(y, w[i].im, x * w[i].re);
      r[j].im += fmaf(-y, w[i].re, x * w[i].im);
    }
}

// One hop of a field in global memory: neighbour (c2, s2), link (cl, mu, sl)
template <int FI, int DAG, class LP>
__device__ __forceinline__ void eo_field_hop(const EoRole &ro, const float4 *phi, const void *links, int vbh, int c2,
                                             int s2, int cl, int mu, int sl, float gy, bool neg, Pair3 &up, Pair3 &lo) {
  float r[LP::NRAW], u[18];
  float4 q[6];
  const float4 *f = phi + (size_t)c2 * 6 * vbh + s2;
#pragma unroll
  for (int j = 0; j < 6; j++) q[j] = __ldg(f + (size_t)j * vbh);
  LP::load(links, cl, mu, sl, vbh, r);
  LP::expand(r, u);
  LP::sign(neg, u);
  float2 hr[3], hi[3];
  auto comp = [&](int i) { return i & 1 ? make_float2(q[i / 2].z, q[i / 2].w) : make_float2(q[i / 2].x, q[i / 2].y); };
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float2 c1 = comp(k), c2_ = comp(3 + k), c3 = comp(6 + k), c4 = comp(9 + k);
    const float2 l1 = ro.role ? c4 : c3, l2 = ro.role ? c3 : c4;
    hop_project<FI, DAG>(make_float4(c1.x, c2_.x, c1.y, c2_.y), make_float4(l1.x, l2.x, l1.y, l2.y), gy, hr[k], hi[k]);
  }
  hop_link<FI, DAG>(hr, hi, u, gy, up, lo);
}

// The x0-hops across a rank boundary (domain decomposition), from the half
// spinors of the exchanged faces: the neighbour's projection times the own
// link (forward), the product the neighbour formed (backward).  Role 0 only.
template <class LP>
__device__ __forceinline__ void eo_face_fwd(const void *face, int F, int f, const void *links, int vbh, int chunk,
                                            int s, bool neg, Pair3 &up, Pair3 &lo) {
  vec3<float> h0, h1;
  Half<float>::load(face, F, f, h0, h1);
  float r[LP::NRAW], u[18];
  LP::load(links, chunk, 0, s, vbh, r);
  LP::expand(r, u);
  LP::sign(neg, u);
  float2 hr[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    hr[k] = make_float2(h0.c[k].re, h1.c[k].re);
    hi[k] = make_float2(h0.c[k].im, h1.c[k].im);
  }
  hop_link<0, 0>(hr, hi, u, 1.0f, up, lo);
}
// the two faces a rank sends: the projections of its first plane, and the
// products with the time links of its last one
template <class LP>
__device__ __forceinline__ void eo_face_send(int side, const spinor<float> &v, const void *links, int vbh, int chunk,
                                             int s, bool neg, vec3<float> &o0, vec3<float> &o1) {
  float2 hr[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float4 a = make_float4(v.c[0].c[k].re, v.c[1].c[k].re, v.c[0].c[k].im, v.c[1].c[k].im);
    const float4 b = make_float4(v.c[2].c[k].re, v.c[3].c[k].re, v.c[2].c[k].im, v.c[3].c[k].im);
    if (side == 0) hop_project<0, 0>(a, b, 1.0f, hr[k], hi[k]);
    else hop_project<0, 1>(a, b, -1.0f, hr[k], hi[k]);
  }
  if (side != 0) {
    float r[LP::NRAW], u[18];
    LP::load(links, chunk, 0, s, vbh, r);
    LP::expand(r, u);
    LP::sign(neg, u);
    Pair3 up, lo;
#pragma unroll
    for (int k = 0; k < 3; k++) up.re[k] = up.im[k] = lo.re[k] = lo.im[k] = make_float2(0.0f, 0.0f);
    hop_link<0, 1>(hr, hi, u, -1.0f, up, lo);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      hr[k] = up.re[k];
      hi[k] = up.im[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    o0.c[k] = mk<float>(hr[k].x, hi[k].x);
    o1.c[k] = mk<float>(hr[k].y, hi[k].y);
  }
}
__device__ __forceinline__ void eo_face_bwd(const void *face, int F, int f, Pair3 &up, Pair3 &lo) {
  vec3<float> c0, c1;
  Half<float>::load(face, F, f, c0, c1);
#pragma unroll
  for (int k = 0; k < 3; k++)
    hop_add<0, 1>(k, make_float2(c0.c[k].re, c1.c[k].re), make_float2(c0.c[k].im, c1.c[k].im), -1.0f, up, lo);
}

}  // namespace qcd
