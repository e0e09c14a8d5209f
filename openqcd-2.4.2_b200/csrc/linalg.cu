// BLAS-1 on spinor fields in the device layout, with the reference's
// precision rules: products of FP32 fields accumulate in double
// (modules/linalg/salg.c:1050-1078; here after summing the four products of
// a float4 in FP32), products of FP64 fields accumulate in double-double
// (modules/linalg/salg_dble.c:2319-2357 with utils/qsum.c).
//
// A parity half of a field is a contiguous range (even chunks come first), so
// everything here works on flat arrays: FP64 fields as double2 (one complex
// component), FP32 fields as float4 (two complex components).
//
// Reductions are two deterministic passes in one launch: a grid of at most
// RB blocks (fixed by the field's size) sums in double (per thread, then a
// fixed tree in the block), then the last block to finish adds the partials
// in the order of the blocks in double-double (Knuth's TwoSum) and writes the
// result to page-locked host memory, so results are bit-identical from run
// to run and a reduction costs the host one launch and one wait.
#include <cmath>
#include <cstring>
#include "lib.h"

namespace qcd {

static const int RB = LA_RB;
static const int RT = 256;

struct Range { size_t beg, n; };

static Range range(const Ctx &c, int prec, int par) {
  size_t per_site = prec == 64 ? 12 : 6;       // double2 or float4 elements per site
  size_t half = (size_t)c.g.volh * per_site;
  if (par == PAR_ALL) return {0, 2 * half};
  return {par == PAR_ODD ? half : 0, half};
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// block sum of NC values into out[NC*blockIdx.x + k]
template <int NC>
__device__ __forceinline__ void block_store(double v[NC], double *out) {
  __shared__ double sh[NC][RT / 32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NC; k++) {
    double t = warp_sum(v[k]);
    if (lane == 0) sh[k][w] = t;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < NC; k++) {
      double t = threadIdx.x < RT / 32 ? sh[k][threadIdx.x] : 0.0;
      t = warp_sum(t);
      if (threadIdx.x == 0) out[(size_t)NC * blockIdx.x + k] = t;
    }
  }
}

// (h, l) += (x, xl) in double-double (Knuth's TwoSum)
__device__ __forceinline__ void dd_acc(double &h, double &l, double x, double xl) {
  const double s = h + x, bb = s - h;
  l += (h - (s - bb)) + (x - bb) + xl;
  h = s;
}

// The second pass in the same launch: every block stores its NC partial sums
// and the block that arrives last at the counter adds them all, in the order
// of the blocks' indices whichever block that is, in double-double.  True in
// thread 0 of that block only, with the sums in (hi, lo) pairs; the counter
// is zero again for the next launch of the stream.  (As kernels of their own
// the second pass and the copy of its result to the host cost two more
// launches, about 10 us per reduction.)
struct Fin {
  double *part;
  unsigned *cnt;
};
template <int NC> __device__ __forceinline__ bool block_last(const Fin &f) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(f.cnt, 1u) == gridDim.x - 1;
    if (last) *f.cnt = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}
template <int NC> __device__ __forceinline__ bool block_finish(double v[NC], const Fin &f, double (&hi)[NC], double (&lo)[NC]) {
  __shared__ double sh[RT / 32][2 * NC];
  block_store<NC>(v, f.part);
  if (!block_last<NC>(f)) return false;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NC; k++) hi[k] = lo[k] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += RT)
#pragma unroll
    for (int k = 0; k < NC; k++) dd_acc(hi[k], lo[k], __ldcg(f.part + (size_t)NC * b + k), 0.0);
#pragma unroll
  for (int k = 0; k < NC; k++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double h2 = __shfl_down_sync(0xffffffffu, hi[k], o), l2 = __shfl_down_sync(0xffffffffu, lo[k], o);
      dd_acc(hi[k], lo[k], h2, l2);
    }
    if (lane == 0) {
      sh[w][2 * k] = hi[k];
      sh[w][2 * k + 1] = lo[k];
    }
  }
  __syncthreads();
  if (threadIdx.x) return false;
#pragma unroll
  for (int k = 0; k < NC; k++) {
    for (int j = 1; j < RT / 32; j++) dd_acc(hi[k], lo[k], sh[j][2 * k], sh[j][2 * k + 1]);
    const double s = hi[k] + lo[k];
    lo[k] -= s - hi[k];
    hi[k] = s;
  }
  return true;
}
// the sums to out[2k], out[2k+1] (page-locked host memory)
template <int NC> __device__ __forceinline__ void finish_to(double v[NC], const Fin &f, double *out) {
  double hi[NC], lo[NC];
  if (block_finish<NC>(v, f, hi, lo))
#pragma unroll
    for (int k = 0; k < NC; k++) {
      out[2 * k] = hi[k];
      out[2 * k + 1] = lo[k];
    }
}

// FP32 fields: the products of one float4 (two complex components) are
// summed in FP32 and that sum is added in double (per-product FP64
// arithmetic made these reductions FP64-throughput bound on B200, at about
// half their bandwidth-bound speed)
template <typename R>
__global__ void k_norm2(const void *__restrict__ x, Range r, Fin f, double *out) {
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < r.n; i += (size_t)gridDim.x * RT) {
    if (sizeof(R) == 8) {
      double2 a = __ldg((const double2 *)x + r.beg + i);
      v[0] += a.x * a.x + a.y * a.y;
    } else {
      float4 a = __ldg((const float4 *)x + r.beg + i);
      v[0] += (double)(a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w);
    }
  }
  finish_to<1>(v, f, out);
}

template <typename R>
__global__ void k_dot(const void *__restrict__ x, const void *__restrict__ y, Range r, Fin f, double *out) {
  double v[2] = {0.0, 0.0};
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < r.n; i += (size_t)gridDim.x * RT) {
    if (sizeof(R) == 8) {
      double2 a = __ldg((const double2 *)x + r.beg + i), b = __ldg((const double2 *)y + r.beg + i);
      v[0] += a.x * b.x + a.y * b.y;
      v[1] += a.x * b.y - a.y * b.x;
    } else {
      float4 a = __ldg((const float4 *)x + r.beg + i), b = __ldg((const float4 *)y + r.beg + i);
      v[0] += (double)(a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w);
      v[1] += (double)(a.x * b.y - a.y * b.x + a.z * b.w - a.w * b.z);
    }
  }
  finish_to<2>(v, f, out);
}

// uniform norm: max over sites of the spinor norm (sflds/unorm.c)
template <typename R>
__global__ void k_unorm(Geom g, const void *__restrict__ x, int c0, int nch, Fin f, double *out) {
  double m = 0.0;
  size_t nsite = (size_t)nch * g.vbh;
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < nsite; i += (size_t)gridDim.x * RT) {
    int chunk = c0 + (int)(i / g.vbh), s = (int)(i % g.vbh);
    spinor<R> v = Store<R>::load_spinor(x, chunk, s, g.vbh);
    double n2 = 0.0;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int k = 0; k < 3; k++) n2 += (double)v.c[a].c[k].re * v.c[a].c[k].re + (double)v.c[a].c[k].im * v.c[a].c[k].im;
    m = fmax(m, n2);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  __shared__ double sh[RT / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < RT / 32; w++) t = fmax(t, sh[w]);
    f.part[blockIdx.x] = t;
  }
  if (!block_last<1>(f) || threadIdx.x >= 32) return;
  m = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) m = fmax(m, __ldcg(f.part + b));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if (threadIdx.x == 0) {
    out[0] = sqrt(m);
    out[1] = 0.0;
  }
}

int alloc_all(std::initializer_list<Buffer> want) {
  bool ok = true;
  for (const Buffer &b : want) {
    *b.p = nullptr;
    if (!ok) continue;
    ok = (b.host ? cudaMallocHost(b.p, b.bytes) : cudaMalloc(b.p, b.bytes)) == cudaSuccess;
    if (!ok) *b.p = nullptr;
  }
  if (ok) return 0;
  for (const Buffer &b : want) {
    if (b.host) cudaFreeHost(*b.p);
    else cudaFree(*b.p);
    *b.p = nullptr;
  }
  return -1;
}

int la_buffers(Ctx &c) {
  if (c.red) return 0;
  if (alloc_all({dev_buf(c.red, (size_t)RB * 4), dev_buf(c.red_out, 8), dev_buf(c.red_cnt, 1), host_buf(c.h_red, 8)}))
    return fail("out of memory (reduction buffers)");
  cudaMemsetAsync(c.red_cnt, 0, sizeof(unsigned), c.stream);
  return 0;
}
static Fin fin(const Ctx &c) { return Fin{c.red, c.red_cnt}; }
// blocks of a reduction over n elements: at most RB, none without work
static unsigned rgrid(size_t n) {
  const size_t b = (n + RT - 1) / RT;
  return (unsigned)(b < 1 ? 1 : (b < (size_t)RB ? b : (size_t)RB));
}

// the nc (hi, lo) results of this rank, which the kernel wrote to h_red,
// then (domain decomposition) their sum or maximum over the ranks, the same
// on every rank
static int finish(Ctx &c, int nc, double *res, bool is_max = false) {
  if (cudaStreamSynchronize(c.stream) != cudaSuccess) return fail("reduction: CUDA error");
  for (int k = 0; k < 2 * nc; k++) res[k] = c.h_red[k];
  return dd_on(c) ? dd_global(c, res, nc, is_max) : 0;
}

int la_norm2(Ctx &c, int prec, const void *x, int par, double *res) {
  if (la_buffers(c)) return -1;
  Range r = range(c, prec, par);
  if (prec == 64) k_norm2<double><<<rgrid(r.n), RT, 0, c.stream>>>(x, r, fin(c), c.h_red);
  else k_norm2<float><<<rgrid(r.n), RT, 0, c.stream>>>(x, r, fin(c), c.h_red);
  return finish(c, 1, res);
}

int la_dot(Ctx &c, int prec, const void *x, const void *y, int par, double *res) {
  if (la_buffers(c)) return -1;
  Range r = range(c, prec, par);
  if (prec == 64) k_dot<double><<<rgrid(r.n), RT, 0, c.stream>>>(x, y, r, fin(c), c.h_red);
  else k_dot<float><<<rgrid(r.n), RT, 0, c.stream>>>(x, y, r, fin(c), c.h_red);
  return finish(c, 2, res);
}

// x += a p ; r -= a ap ; then |r|^2 -- the FP64 CG update of the
// multi-shift solver (modules/linsolv/mscg.c:242-275, cg_step2 with the norm
// of cg_step3) in one pass
__global__ void k_xr_norm2(Range rg, double2 *__restrict__ x, double2 *__restrict__ r,
                           const double2 *__restrict__ p, const double2 *__restrict__ ap, double a, Fin f,
                           double *out) {
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < rg.n; i += (size_t)gridDim.x * RT) {
    const size_t j = rg.beg + i;
    const double2 pp = __ldg(p + j), aa = __ldg(ap + j);
    double2 xx = x[j], rr = r[j];
    xx.x += a * pp.x;
    xx.y += a * pp.y;
    rr.x -= a * aa.x;
    rr.y -= a * aa.y;
    x[j] = xx;
    r[j] = rr;
    v[0] += rr.x * rr.x + rr.y * rr.y;
  }
  finish_to<1>(v, f, out);
}

int la_xr_norm2(Ctx &c, void *x, void *r, const void *p, const void *ap, double a, int par, double *res) {
  if (la_buffers(c)) return -1;
  Range rg = range(c, 64, par);
  k_xr_norm2<<<rgrid(rg.n), RT, 0, c.stream>>>(rg, (double2 *)x, (double2 *)r, (const double2 *)p, (const double2 *)ap, a,
                                               fin(c), c.h_red);
  return finish(c, 1, res);
}

// x -> gamma5 x on a parity range of an FP64 field (spin components 2, 3 of
// every site change sign: double2 planes 6..11 of a chunk), then |x|^2
__global__ void k_mulg5_norm2(Range rg, double2 *__restrict__ x, int vbh, Fin f, double *out) {
  double v[1] = {0.0};
  const size_t per = (size_t)12 * vbh;
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < rg.n; i += (size_t)gridDim.x * RT) {
    const size_t j = rg.beg + i;
    double2 xx = x[j];
    if ((j % per) / vbh >= 6) {
      xx.x = -xx.x;
      xx.y = -xx.y;
      x[j] = xx;
    }
    v[0] += xx.x * xx.x + xx.y * xx.y;
  }
  finish_to<1>(v, f, out);
}

int la_mulg5_norm2(Ctx &c, void *x, int par, double *res) {
  if (la_buffers(c)) return -1;
  Range rg = range(c, 64, par);
  k_mulg5_norm2<<<rgrid(rg.n), RT, 0, c.stream>>>(rg, (double2 *)x, c.g.vbh, fin(c), c.h_red);
  return finish(c, 1, res);
}

int la_unorm(Ctx &c, int prec, const void *x, int par, double *res) {
  if (la_buffers(c)) return -1;
  int c0 = par == PAR_ODD ? c.g.nbl : 0;
  int nch = par == PAR_ALL ? 2 * c.g.nbl : c.g.nbl;
  const unsigned nb = rgrid((size_t)nch * c.g.vbh);
  if (prec == 64) k_unorm<double><<<nb, RT, 0, c.stream>>>(c.g, x, c0, nch, fin(c), c.h_red);
  else k_unorm<float><<<nb, RT, 0, c.stream>>>(c.g, x, c0, nch, fin(c), c.h_red);
  return finish(c, 1, res, true);
}

// ---------------------------------------------- one step of the flexible GCR
// gcr_step of modules/linsolv/fgcr.c:157 (modified Gram-Schmidt of chi_k
// against chi_0..chi_{k-1}, normalisation, update of the residual rho) with
// its coefficients kept on the device: pass l subtracts the product of pass
// l-1 and forms the next one, so the step is k + 3 launches and one wait of
// the host, where launches, a wait and an update per product took k + 3 waits
// of about 25 us: sap_gcr on 8^4 2.86 -> 2.35 ms, on 32x16^3 13.7 -> 11.3 ms.  The arithmetic is that of
// la_dot, la_norm2, la_axpy and la_scale with the host's roundings between.
// rec[l] (l < k) = (chi_l, chi_k), rec[k] = |chi_k|^2, rec[k+1] = (chi_k,
// rho), rec[k+2] = |rho|^2, on the device and in page-locked memory.
enum { GS_DOT, GS_NORM, GS_SCALE };
// y -= z xp (z = *zp rounded to FP32) or, with GS_SCALE, y /= |y| (|y|^2 =
// *zp); then (xn, y), |y|^2 (GS_NORM) or (y, xn) (GS_SCALE)
template <int MODE>
__global__ void __launch_bounds__(RT) k_gcr_pass(size_t n, float4 *y, const float4 *__restrict__ xp,
                                                 const double2 *zp, const float4 *__restrict__ xn, Fin f, double2 *rec,
                                                 double2 *hrec) {
  constexpr int NC = MODE == GS_NORM ? 1 : 2;
  float zr = 0.0f, zi = 0.0f;
  bool upd = xp != nullptr;
  if (MODE == GS_SCALE) {
    const float nn = (float)sqrt((double)(float)zp->x);
    upd = nn != 0.0f;
    zr = upd ? 1.0f / nn : 1.0f;
  } else if (upd) {
    zr = -(float)zp->x;
    zi = -(float)zp->y;
  }
  double v[NC];
#pragma unroll
  for (int k = 0; k < NC; k++) v[k] = 0.0;
  for (size_t i = blockIdx.x * (size_t)RT + threadIdx.x; i < n; i += (size_t)gridDim.x * RT) {
    float4 b = y[i];
    if (MODE == GS_SCALE) {
      b = make_float4(zr * b.x, zr * b.y, zr * b.z, zr * b.w);
    } else if (upd) {
      const float4 a = __ldg(xp + i);
      b.x += zr * a.x - zi * a.y;
      b.y += zr * a.y + zi * a.x;
      b.z += zr * a.z - zi * a.w;
      b.w += zr * a.w + zi * a.z;
    }
    if (upd) y[i] = b;
    if (MODE == GS_NORM) {
      v[0] += (double)(b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w);
    } else {
      const float4 x = __ldg(xn + i);
      v[0] += (double)(x.x * b.x + x.y * b.y + x.z * b.z + x.w * b.w);
      const double im = (double)(x.x * b.y - x.y * b.x + x.z * b.w - x.w * b.z);
      v[NC - 1] += MODE == GS_SCALE ? -im : im;   // (xn, y) or (y, xn)
    }
  }
  double hi[NC], lo[NC];
  if (block_finish<NC>(v, f, hi, lo)) {
    const double2 r = make_double2(hi[0] + lo[0], NC == 2 ? hi[NC - 1] + lo[NC - 1] : 0.0);
    *rec = r;
    *hrec = r;
  }
}

// chi[0..k], rho: FP32 fields.  On return chi[k] is normalised and rho
// reduced; a[l], b, cc and rn are those of gcr_step.
int la_gcr_step(Ctx &c, int k, void *const *chi, void *rho, cplxf *a, float *b, cplxf *cc, double *rn) {
  if (la_buffers(c)) return -1;
  if (c.gcr_n < k + 3) {
    cudaFree(c.gcr_rec);
    cudaFreeHost(c.h_gcr_rec);
    c.gcr_rec = c.h_gcr_rec = nullptr;
    c.gcr_n = 0;
    const int m = k + 3 < 64 ? 64 : k + 3 + 64;
    if (cudaMalloc(&c.gcr_rec, m * sizeof(double2)) != cudaSuccess ||
        cudaMallocHost(&c.h_gcr_rec, m * sizeof(double2)) != cudaSuccess)
      return fail("out of memory (GCR record)");
    c.gcr_n = m;
  }
  const size_t n = range(c, 32, PAR_ALL).n;
  const unsigned nb = rgrid(n);
  const Fin f = fin(c);
  double2 *r = c.gcr_rec, *h = c.h_gcr_rec;
  float4 *y = (float4 *)chi[k], *rh = (float4 *)rho;
  for (int l = 0; l < k; l++)
    k_gcr_pass<GS_DOT><<<nb, RT, 0, c.stream>>>(n, y, l ? (const float4 *)chi[l - 1] : nullptr, l ? r + l - 1 : nullptr,
                                                (const float4 *)chi[l], f, r + l, h + l);
  k_gcr_pass<GS_NORM><<<nb, RT, 0, c.stream>>>(n, y, k ? (const float4 *)chi[k - 1] : nullptr, k ? r + k - 1 : nullptr,
                                               nullptr, f, r + k, h + k);
  k_gcr_pass<GS_SCALE><<<nb, RT, 0, c.stream>>>(n, y, nullptr, r + k, rh, f, r + k + 1, h + k + 1);
  k_gcr_pass<GS_NORM><<<nb, RT, 0, c.stream>>>(n, rh, y, r + k + 1, nullptr, f, r + k + 2, h + k + 2);
  if (cudaStreamSynchronize(c.stream) != cudaSuccess) return fail("gcr step: CUDA error");
  for (int l = 0; l < k; l++) a[l] = cplxf{(float)h[l].x, (float)h[l].y};
  *b = (float)std::sqrt((double)(float)h[k].x);
  *cc = cplxf{(float)h[k + 1].x, (float)h[k + 1].y};
  *rn = std::sqrt((double)(float)h[k + 2].x);
  return 0;
}

// ------------------------------------------------------------- elementwise
static unsigned nblk(size_t n) { return (unsigned)((n + 255) / 256); }

__global__ void k_copy_dd(Range r, const double2 *x, double2 *y) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) y[r.beg + i] = x[r.beg + i];
}
__global__ void k_copy_ff(Range r, const float4 *x, float4 *y) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) y[r.beg + i] = x[r.beg + i];
}
// Precision conversion works per site: plane j (float4) of an FP32 chunk
// holds components 2j, 2j+1, while an FP64 chunk has one double2 plane per
// component, so the two layouts do not line up element by element.
template <typename A, typename B>
__global__ void k_convert(Geom g, int c0, int nch, const void *x, void *y) {
  size_t i = blockIdx.x * (size_t)128 + threadIdx.x;
  if (i >= (size_t)nch * g.vbh) return;
  int chunk = c0 + (int)(i / g.vbh), s = (int)(i % g.vbh);
  spinor<A> a = Store<A>::load_spinor_rw(x, chunk, s, g.vbh);
  spinor<B> b;
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int j = 0; j < 3; j++) b.c[k].c[j] = mk<B>((B)a.c[k].c[j].re, (B)a.c[k].c[j].im);
  Store<B>::store_spinor(y, chunk, s, g.vbh, b);
}

void la_copy(const Ctx &c, int pin, const void *x, int pout, void *y, int par, cudaStream_t st) {
  if (pin == pout) {
    Range r = range(c, pin, par);
    if (pin == 64) k_copy_dd<<<nblk(r.n), 256, 0, st>>>(r, (const double2 *)x, (double2 *)y);
    else k_copy_ff<<<nblk(r.n), 256, 0, st>>>(r, (const float4 *)x, (float4 *)y);
    return;
  }
  int c0 = par == PAR_ODD ? c.g.nbl : 0;
  int nch = par == PAR_ALL ? 2 * c.g.nbl : c.g.nbl;
  size_t n = (size_t)nch * c.g.vbh;
  unsigned nb = (unsigned)((n + 127) / 128);
  if (pin == 64) k_convert<double, float><<<nb, 128, 0, st>>>(c.g, c0, nch, x, y);
  else k_convert<float, double><<<nb, 128, 0, st>>>(c.g, c0, nch, x, y);
}

void la_zero(const Ctx &c, int prec, void *x, int par, cudaStream_t st) {
  Range r = range(c, prec, par);
  size_t es = prec == 64 ? sizeof(double2) : sizeof(float4);
  cudaMemsetAsync((char *)x + r.beg * es, 0, r.n * es, st);
}

__global__ void k_scale_d(Range r, double2 *x, double a) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) { double2 v = x[r.beg + i]; x[r.beg + i] = make_double2(a * v.x, a * v.y); }
}
__global__ void k_scale_f(Range r, float4 *x, float a) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) { float4 v = x[r.beg + i]; x[r.beg + i] = make_float4(a * v.x, a * v.y, a * v.z, a * v.w); }
}
void la_scale(const Ctx &c, int prec, void *x, double a, int par, cudaStream_t st) {
  Range r = range(c, prec, par);
  if (prec == 64) k_scale_d<<<nblk(r.n), 256, 0, st>>>(r, (double2 *)x, a);
  else k_scale_f<<<nblk(r.n), 256, 0, st>>>(r, (float4 *)x, (float)a);
}

// y += a x  (mulc_spinor_add, salg.c:1319 / salg_dble.c)
__global__ void k_axpy_d(Range r, double2 *y, double ar, double ai, const double2 *x) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) {
    double2 a = x[r.beg + i], b = y[r.beg + i];
    b.x += ar * a.x - ai * a.y;
    b.y += ar * a.y + ai * a.x;
    y[r.beg + i] = b;
  }
}
__global__ void k_axpy_f(Range r, float4 *y, float ar, float ai, const float4 *x) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) {
    float4 a = x[r.beg + i], b = y[r.beg + i];
    b.x += ar * a.x - ai * a.y;
    b.y += ar * a.y + ai * a.x;
    b.z += ar * a.z - ai * a.w;
    b.w += ar * a.w + ai * a.z;
    y[r.beg + i] = b;
  }
}
void la_axpy(const Ctx &c, int prec, void *y, double ar, double ai, const void *x, int par, cudaStream_t st) {
  Range r = range(c, prec, par);
  if (prec == 64) k_axpy_d<<<nblk(r.n), 256, 0, st>>>(r, (double2 *)y, ar, ai, (const double2 *)x);
  else k_axpy_f<<<nblk(r.n), 256, 0, st>>>(r, (float4 *)y, (float)ar, (float)ai, (const float4 *)x);
}

// y (+)= sum of c_l x_l over up to 16 terms, applied in the given order with
// the arithmetic of k_axpy_f: the solution update of fgcr (update_psi,
// fgcr.c:181) in one pass over the fields instead of one axpy per term
struct LcTerms {
  const float4 *x[16];
  float2 c[16];
};
__global__ void k_lincomb_f(Range r, float4 *y, int nt, int acc, LcTerms t) {
  const size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i >= r.n) return;
  float4 b = acc ? y[r.beg + i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int l = 0; l < nt; l++) {
    const float4 a = t.x[l][r.beg + i];
    const float ar = t.c[l].x, ai = t.c[l].y;
    b.x += ar * a.x - ai * a.y;
    b.y += ar * a.y + ai * a.x;
    b.z += ar * a.z - ai * a.w;
    b.w += ar * a.w + ai * a.z;
  }
  y[r.beg + i] = b;
}
void la_lincomb32(const Ctx &c, void *y, int n, const float *cre, const float *cim, void *const *x,
                  cudaStream_t st) {
  const Range r = range(c, 32, PAR_ALL);
  if (n <= 0) {
    la_zero(c, 32, y, PAR_ALL, st);
    return;
  }
  for (int l0 = 0; l0 < n; l0 += 16) {
    LcTerms t;
    std::memset(&t, 0, sizeof(t));
    const int nt = n - l0 < 16 ? n - l0 : 16;
    for (int l = 0; l < nt; l++) {
      t.x[l] = (const float4 *)x[l0 + l];
      t.c[l] = make_float2(cre[l0 + l], cim[l0 + l]);
    }
    k_lincomb_f<<<nblk(r.n), 256, 0, st>>>(r, (float4 *)y, nt, l0 > 0, t);
  }
}

// y = x - y
__global__ void k_diff_f(Range r, const float4 *x, float4 *y) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) {
    float4 a = x[r.beg + i], b = y[r.beg + i];
    y[r.beg + i] = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
  }
}
__global__ void k_diff_d(Range r, const double2 *x, double2 *y) {
  size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i < r.n) {
    double2 a = x[r.beg + i], b = y[r.beg + i];
    y[r.beg + i] = make_double2(a.x - b.x, a.y - b.y);
  }
}
void la_diff(const Ctx &c, int prec, const void *x, void *y, int par, cudaStream_t st) {
  Range r = range(c, prec, par);
  if (prec == 64) k_diff_d<<<nblk(r.n), 256, 0, st>>>(r, (const double2 *)x, (double2 *)y);
  else k_diff_f<<<nblk(r.n), 256, 0, st>>>(r, (const float4 *)x, (float4 *)y);
}

// sd += s (add_s2sd, sflds.c:1356) and r = a - b rounded to FP32 (diff_sd2s, sflds.c:1390)
template <int MODE>
__global__ void k_mixed(Geom g, int c0, int nch, const void *a, const void *b, void *out) {
  size_t i = blockIdx.x * (size_t)128 + threadIdx.x;
  if (i >= (size_t)nch * g.vbh) return;
  int chunk = c0 + (int)(i / g.vbh), s = (int)(i % g.vbh);
  if (MODE == 0) {   // out(FP64) += a(FP32)
    spinor<float> x = Store<float>::load_spinor_rw(a, chunk, s, g.vbh);
    spinor<double> y = Store<double>::load_spinor_rw(out, chunk, s, g.vbh);
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 3; j++) { y.c[k].c[j].re += x.c[k].c[j].re; y.c[k].c[j].im += x.c[k].c[j].im; }
    Store<double>::store_spinor(out, chunk, s, g.vbh, y);
  } else {           // out(FP32) = a(FP64) - b(FP64)
    spinor<double> x = Store<double>::load_spinor_rw(a, chunk, s, g.vbh);
    spinor<double> y = Store<double>::load_spinor_rw(b, chunk, s, g.vbh);
    spinor<float> z;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 3; j++)
        z.c[k].c[j] = mk<float>((float)(x.c[k].c[j].re - y.c[k].c[j].re), (float)(x.c[k].c[j].im - y.c[k].c[j].im));
    Store<float>::store_spinor(out, chunk, s, g.vbh, z);
  }
}

void la_add_s2sd(const Ctx &c, const void *s32, void *sd, int par, cudaStream_t st) {
  int c0 = par == PAR_ODD ? c.g.nbl : 0, nch = par == PAR_ALL ? 2 * c.g.nbl : c.g.nbl;
  size_t n = (size_t)nch * c.g.vbh;
  k_mixed<0><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(c.g, c0, nch, s32, nullptr, sd);
}

void la_diff_sd2s(const Ctx &c, const void *ad, const void *bd, void *r32, int par, cudaStream_t st) {
  int c0 = par == PAR_ODD ? c.g.nbl : 0, nch = par == PAR_ALL ? 2 * c.g.nbl : c.g.nbl;
  size_t n = (size_t)nch * c.g.vbh;
  k_mixed<1><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(c.g, c0, nch, ad, bd, r32);
}

}  // namespace qcd
