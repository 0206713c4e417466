// kdiag.cu -- FP64 diagnostics on the device: norms, chemical potential sums, damping integral, error
// vs a double-precision reference.  One launch each: blocks write partial sums, the last block to
// finish adds them in a fixed order, so a result never depends on what else runs on the GPU.
//
// The FP64 pipe would bound these sums, not memory (a DFMA of a warp takes 19 cycles of its SM, a
// conversion 16; 8 bytes a lane arrive in 12).  The complex64 forms of the norm and the chemical
// potential therefore add up groups of 16 nodes in single precision without loss -- a product of floats
// is exact as a pair, and the group's sum is kept in three floats, whose additions leave 2^-66 of the
// sum of its terms' sizes -- and add the groups in FP64: one rounding to a double's last place a group,
// where FP64 sums round for every node.  (Two floats a group lost 2^-48 an addition: 8e-15 of the norm of
// a nearly uniform state, against 2.5e-15 for FP64 sums and below 1e-15 here; 2048^2, the caches cold: norm
// 21 us with two floats and 24 with three, chemical potential 56 and 64.)  Small grids and groups with
// values outside single precision's range (non-finite, squares near its ends) are added in FP64 node by
// node.
#include <algorithm>

#include "kernels.h"
#include "nls_common.cuh"

namespace nlsg {

static constexpr int kDiagBlocks = 1216;  // 8 x 152 SMs
static constexpr int kDiagThreads = 256;
static constexpr int kDiagMaxNV = kDiagStatus;
static constexpr int kGroup = 16;         // nodes added up in single precision
// Grids from which groups are added up so.  Smaller grids are added up in FP64, one node a thread: what
// counts there is the length of a thread's chain.
static constexpr long long kPairsFrom = 65536;

size_t diag_partials_bytes(long long) { return (size_t)kDiagBlocks * kDiagMaxNV * sizeof(double) + 256; }

__device__ __forceinline__ double weight(int mode, long long i, double dx) {
  return mode == 1 ? (double)i * dx : 1.0;
}

// Block sums to part; the last block of the launch adds all blocks' and writes out, and after the sums
// the context's status word, so that the host learns with them whether the state can be trusted.  The
// word after the partials counts finished blocks; it starts at zero and is left at zero.
template <int NV>
__device__ __forceinline__ void diag_finish(double (&v)[NV], const DiagOut& d) {
  double* const part = d.partials;
  __shared__ double sm[32 * NV];
  __shared__ bool last;
  block_sum<NV>(v, sm);
  unsigned* const ticket = reinterpret_cast<unsigned*>(part + kDiagBlocks * kDiagMaxNV);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) part[blockIdx.x * NV + k] = v[k];
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += __ldcg(part + b * NV + k);
  block_sum<NV>(v, sm);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) d.out[k] = v[k];
    d.out[kDiagStatus] = (double)*reinterpret_cast<const volatile int*>(d.wait_flag);
  }
}

// A sum held as h + m + l.
struct F3 {
  float h, m, l;
};
// acc += t: exact but for the additions to l, which is about 2^-48 of the terms.
__device__ __forceinline__ void sum_add(F3& acc, F2 t) {
  const F2 s = f2_sum(acc.h, t.h);
  const F2 a = f2_sum(acc.m, t.l), b = f2_sum(a.h, s.l);
  acc.h = s.h;
  acc.m = b.h;
  acc.l = fadd(acc.l, fadd(a.l, b.l));
}
__device__ __forceinline__ F2 pair_prod(float a, float b) {
  F2 r;
  r.h = fmul(a, b);
  r.l = ffma(a, b, -r.h);
  return r;
}
// A group's sum of squares of which what products of floats lose (2^-149 each) is below 2^-60, and no
// square overflowed (false for NaN).
__device__ __forceinline__ bool sum_range(float sum_sq) { return sum_sq >= 0x1p-80f && sum_sq < 0x1p100f; }
// v + the sum, rounded to a double's last place; what that leaves goes to rest.
__device__ __forceinline__ double sum_to(double v, F3 a, float& rest) {
  const F2 s = f2_sum(a.h, a.m), q = f2_sum(s.l, a.l);
  rest = fadd(rest, q.l);
  if (fabsf(s.h) < 0x1p-64f) return v + ((double)s.h + (double)q.h);   // f2_join would drop q.h
  return v + f2_join(f2_quick(s.h, q.h));
}

__global__ void __launch_bounds__(kDiagThreads) k_norm_c64(long long n, const float2* __restrict__ u,
                                                           DiagOut out) {
  double v[2] = {0.0, 0.0};
  float rest = 0.f;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kGroup * stride) {
    float2 a[kGroup];
#pragma unroll
    for (int k = 0; k < kGroup; ++k) a[k] = i0 + k * stride < n ? u[i0 + k * stride] : make_float2(0.f, 0.f);
    F3 s = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kGroup; ++k) {
      sum_add(s, pair_prod(a[k].x, a[k].x));
      sum_add(s, pair_prod(a[k].y, a[k].y));
    }
    if (sum_range(s.h)) {
      v[0] = sum_to(v[0], s, rest);
    } else {
#pragma unroll 1
      for (int k = 0; k < kGroup; ++k) {
        if (i0 + k * stride >= n) break;
        const float2 b = u[i0 + k * stride];
        const double x = b.x, y = b.y;
        v[0] += x * x + y * y;
        v[1] += (isfinite(b.x) && isfinite(b.y)) ? 0.0 : 1.0;
      }
    }
  }
  v[0] += (double)rest;
  diag_finish<2>(v, out);
}

template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_norm(long long n, const typename C2<T>::type* __restrict__ u,
                                                       DiagOut out) {
  double v[2] = {0.0, 0.0};
  int bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double2 a = make_double2(u[i].x, u[i].y);
    v[0] = dfma(a.x, a.x, dfma(a.y, a.y, v[0]));
    // exponent all ones: infinite or NaN
    bad += ((dhi(a.x) & 0x7ff00000u) == 0x7ff00000u || (dhi(a.y) & 0x7ff00000u) == 0x7ff00000u) ? 1 : 0;
  }
  v[1] = (double)bad;
  diag_finish<2>(v, out);
}

// Sums of conj(u) H(u) and |u|^2 over one array pair (the radial grids, weighted by r).
template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_mu(long long n, const void* __restrict__ u_,
                                                     const void* __restrict__ h_, int mode, double dx,
                                                     DiagOut out) {
  typedef typename C2<T>::type C;
  const C* u = reinterpret_cast<const C*>(u_);
  const C* hv = reinterpret_cast<const C*>(h_);
  double v[3] = {0.0, 0.0, 0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const C a = u[i], b = hv[i];
    const double w = weight(mode, i, dx);
    const double ax = a.x, ay = a.y, bx = b.x, by = b.y;
    // conj(a) * b
    v[0] += w * (ax * bx + ay * by);
    v[1] += w * (ax * by - ay * bx);
    v[2] += w * (ax * ax + ay * ay);
  }
  diag_finish<3>(v, out);
}

// The same on a square grid with H(u) (order 5) formed on the way: a warp walks G rows of 32 columns
// with the five rows of its column in registers (G = kGroup, or 1 without pairs).  complex64: H in single
// precision as before, the sums without loss as above; complex128: the coefficients in plain FP64 (a step's
// float pairs, f64_node.cuh, would leave 2^-45 of them in the result) and FP64 sums.  Before, H was
// written and read back by launches of their own and every term added in FP64.
template <int G>
__global__ void __launch_bounds__(kDiagThreads) k_mu_2d_c64(int n, const float2* __restrict__ u,
                                                            const float* __restrict__ P, Params<float> prm,
                                                            DiagOut out) {
  double v[3] = {0.0, 0.0, 0.0};
  float rest[3] = {0.f, 0.f, 0.f};
  const Phys<float> ph = phys_of<float>(prm);
  const int lane = threadIdx.x & 31;
  const int cols = (n + 31) / 32;
  const long long tiles = (long long)cols * ((n + G - 1) / G);
  const int warps = blockDim.x >> 5;
  for (long long t = (long long)blockIdx.x * warps + (threadIdx.x >> 5); t < tiles; t += (long long)gridDim.x * warps) {
    const int x = (int)(t % cols) * 32 + lane, y0 = (int)(t / cols) * G;
    if (x >= n) continue;
    auto at = [&](int xx, int y) -> float2 {
      return xx >= 0 && xx < n && y >= 0 && y < n ? u[(size_t)y * n + xx] : make_float2(0.f, 0.f);
    };
    auto slope = [&](float2 c, float2 s1, float2 s2, float p) -> float2 {
      const float2 lu = f2(prm.wc * c.x + prm.w1 * s1.x + prm.w2 * s2.x, prm.wc * c.y + prm.w1 * s1.y + prm.w2 * s2.y);
      return rhs<float>(c, p, lu, ph);
    };
    auto sum4 = [](float2 a, float2 b, float2 c, float2 d) -> float2 {
      return f2((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y));
    };
    float2 w[5];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = at(x, y0 - 2 + k);
    F3 re = {0.f, 0.f, 0.f}, im = re, m = re;
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int y = y0 + j;
      w[(j + 4) % 5] = at(x, y + 2);
      const float2 c = w[(j + 2) % 5];
      const float p = y < n ? P[(size_t)y * n + x] : 0.f;
      const float2 h = slope(c, sum4(at(x - 1, y), at(x + 1, y), w[(j + 1) % 5], w[(j + 3) % 5]),
                             sum4(at(x - 2, y), at(x + 2, y), w[j % 5], w[(j + 4) % 5]), p);
      if (y < n) {
        sum_add(re, pair_prod(c.x, h.x));
        sum_add(re, pair_prod(c.y, h.y));
        sum_add(im, pair_prod(c.x, h.y));
        sum_add(im, pair_prod(-c.y, h.x));
        sum_add(m, pair_prod(c.x, c.x));
        sum_add(m, pair_prod(c.y, c.y));
      }
    }
    if (G > 1 && sum_range(m.h) && fabsf(re.h) < 0x1p100f && fabsf(im.h) < 0x1p100f) {
      v[0] = sum_to(v[0], re, rest[0]);
      v[1] = sum_to(v[1], im, rest[1]);
      v[2] = sum_to(v[2], m, rest[2]);
    } else {
#pragma unroll 1
      for (int y = y0; y < y0 + G && y < n; ++y) {
        const float2 c = at(x, y);
        const float2 h = slope(c, sum4(at(x - 1, y), at(x + 1, y), at(x, y - 1), at(x, y + 1)),
                               sum4(at(x - 2, y), at(x + 2, y), at(x, y - 2), at(x, y + 2)), P[(size_t)y * n + x]);
        const double ax = c.x, ay = c.y, bx = h.x, by = h.y;
        v[0] += ax * bx + ay * by;
        v[1] += ax * by - ay * bx;
        v[2] += ax * ax + ay * ay;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] += (double)rest[k];
  diag_finish<3>(v, out);
}

__global__ void __launch_bounds__(kDiagThreads) k_mu_2d_c128(int n, const double2* __restrict__ u,
                                                             const double* __restrict__ P, F64Consts c,
                                                             DiagOut out) {
  double v[3] = {0.0, 0.0, 0.0};
  const int cols = (n + 31) / 32, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const long long tiles = (long long)cols * n;
  for (long long t = (long long)blockIdx.x * warps + (threadIdx.x >> 5); t < tiles; t += (long long)gridDim.x * warps) {
    const int x = (int)(t % cols) * 32 + lane, y = (int)(t / cols);
    if (x >= n) continue;
    double vx[8], vy[8];
    auto get = [&](int i, int xx, int yy) {
      const bool in = xx >= 0 && xx < n && yy >= 0 && yy < n;
      const double2 a = in ? u[(size_t)yy * n + xx] : make_double2(0.0, 0.0);
      vx[i] = a.x;
      vy[i] = a.y;
    };
#pragma unroll
    for (int d = 1; d <= 2; ++d) {
      get(4 * d - 4, x - d, y);
      get(4 * d - 3, x + d, y);
      get(4 * d - 2, x, y - d);
      get(4 * d - 1, x, y + d);
    }
    const double2 a = u[(size_t)y * n + x];
    const double p = P[(size_t)y * n + x];
    double hx, hy;
    double A, B;
    f64_coeffs_plain(a.x, a.y, p, c, A, B);
    f64_slope_2d<2>(a.x, a.y, vx, vy, A, dadd(B, -c.centre), c, hx, hy);
    v[0] = dfma(a.x, hx, dfma(a.y, hy, v[0]));
    v[1] = dfma(a.x, hy, dfma(-a.y, hx, v[1]));
    v[2] = dfma(a.x, a.x, dfma(a.y, a.y, v[2]));
  }
  diag_finish<3>(v, out);
}

template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_relerr(long long n, const void* __restrict__ a_,
                                                         const double2* __restrict__ b,
                                                         const double* __restrict__ P, double c12,
                                                         double c13, double c14,
                                                         DiagOut out) {
  typedef typename C2<T>::type C;
  const C* a = reinterpret_cast<const C*>(a_);
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const C x = a[i];
    const double2 y = b[i];
    const double da = (double)x.x * (double)x.x + (double)x.y * (double)x.y;
    const double db = y.x * y.x + y.y * y.y;
    const double na = c12 * P[i] / (c13 + c14 * da);
    const double nb = c12 * P[i] / (c13 + c14 * db);
    v[0] += (da - db) * (da - db);
    v[1] += db * db;
    v[2] += (na - nb) * (na - nb);
    v[3] += nb * nb;
  }
  diag_finish<4>(v, out);
}

// Damping integral of Solution.getDampingIntegral (nls/model.py:350-365): the rectangle rule of
// (n_res - 1) |u|^2 with n_res = c12 P / (c13 + c14 |u|^2), weighted by w_i = 2 pi r_i dx on the
// radial grid r_i = i * r_step (r_step = n dx / (n - 1), the spacing of linspace(0, n dx, n)) when
// radial, else by dx^2.
template <typename T>
__device__ __forceinline__ double damping_term(typename C2<T>::type a, T P, double c12, double c13, double c14) {
  const double d = (double)a.x * (double)a.x + (double)a.y * (double)a.y;
  return (c12 * (double)P / (c13 + c14 * d) - 1.0) * d;
}
template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_damping(long long n, const void* __restrict__ u_,
                                                          const void* __restrict__ P_, int radial,
                                                          double r_step, double dx, double c12, double c13,
                                                          double c14, DiagOut out) {
  typedef typename C2<T>::type C;
  const C* u = reinterpret_cast<const C*>(u_);
  const T* P = reinterpret_cast<const T*>(P_);
  const double two_pi = 6.283185307179586476925286766559;
  double v[1] = {0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double w = radial ? two_pi * ((double)i * r_step) * dx : dx * dx;
    v[0] += damping_term<T>(u[i], P[i], c12, c13, c14) * w;
  }
  diag_finish<1>(v, out);
}
// A float as a double by integer operations (a conversion takes 16 cycles of its SM); ok is cleared for
// denormal, infinite and NaN values.
__device__ __forceinline__ double widen(float f, bool& ok) {
  const uint32_t b = bitsf(f), mag = b & 0x7fffffffu;
  ok = ok && (mag == 0u || mag - 0x00800000u < 0x7f000000u);
  return mag == 0u ? 0.0 : dbits((mag >> 3) + (896u << 20) | (b & 0x80000000u), b << 29);
}
// complex64 on a square grid, every term in FP64: near balance of gain and loss, the usual state of a
// condensate, n_res - 1 is small beside n_res, so it is formed as (c12 P - D) / D with D = c13 + c14 |u|^2,
// the difference first.  The quotient is t = t0 + y (N - t0 D), t0 = N y, y = 1/D by one Newton step in
// single precision (2^-45), so t is good to a double's last place.  Eight FP64 instructions a node bound
// it: 2048^2 takes 70 us, the caches cold.  Float pairs for the whole term took 29 us, but lost 2^-45 of
// n_res: 4e-13 of the sum of the terms' sizes at n_res within 1e-3 of 1, against 1e-15 in FP64.
__global__ void __launch_bounds__(kDiagThreads) k_damping_2d_c64(long long n, const float2* __restrict__ u,
                                                                 const float* __restrict__ P, double dx, double c12,
                                                                 double c13, double c14, DiagOut out) {
  double v[1] = {0.0};
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 2
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float2 a = u[i];
    const float p = P[i];
    bool ok = true;
    const double x = widen(a.x, ok), y = widen(a.y, ok), pd = widen(p, ok);
    const double d = dfma(x, x, dmul(y, y));
    const double den = dfma(c14, d, c13), num = dfma(c12, pd, -den);
    // |den| in [2^-58, 2^58)
    ok = ok && (dhi(den) & 0x7fffffffu) - ((1023u - 58u) << 20) < (116u << 20);
    const F2 s = f2_split(den);
    const float yr = frcp(s.h);
    const double inv = f2_join(f2_quick(yr, fmul(yr, ffma(-s.l, yr, ffma(-s.h, yr, 1.f)))));
    const double t0 = dmul(num, inv);
    const double t = dfma(dfma(-t0, den, num), inv, t0);
    if (ok) v[0] = dfma(t, d, v[0]);
    else v[0] += damping_term<float>(a, p, c12, c13, c14);
  }
  v[0] *= dx * dx;
  diag_finish<1>(v, out);
}

static int blocks_for(long long n) {
  const long long b = (n + kDiagThreads - 1) / kDiagThreads;
  return (int)std::max<long long>(1, std::min<long long>(b, kDiagBlocks));
}

cudaError_t diag_norm(int dtype, long long n, const void* u, const DiagOut& out, cudaStream_t st) {
  if (dtype == NLS_C128) k_norm<double><<<blocks_for(n), kDiagThreads, 0, st>>>(n, (const double2*)u, out);
  else if (n < kPairsFrom) k_norm<float><<<blocks_for(n), kDiagThreads, 0, st>>>(n, (const float2*)u, out);
  else k_norm_c64<<<blocks_for((n + kGroup - 1) / kGroup), kDiagThreads, 0, st>>>(n, (const float2*)u, out);
  return cudaGetLastError();
}

cudaError_t diag_mu(int dtype, long long n, const void* u, const void* v, int mode, double dx,
                    const DiagOut& out, cudaStream_t st) {
  const int nb = blocks_for(n);
  if (dtype == NLS_C128) k_mu<double><<<nb, kDiagThreads, 0, st>>>(n, u, v, mode, dx, out);
  else k_mu<float><<<nb, kDiagThreads, 0, st>>>(n, u, v, mode, dx, out);
  return cudaGetLastError();
}

cudaError_t diag_mu_2d(int dtype, int n, const void* u, const void* P, const PhysD& ph, const Stencil2D& op,
                       const DiagOut& out, cudaStream_t st) {
  const int rows = dtype == NLS_C128 || (long long)n * n < kPairsFrom ? 1 : kGroup;   // of a warp at a time
  const int nb = blocks_for((long long)((n + rows - 1) / rows) * ((n + 31) / 32) * 32);
  if (dtype == NLS_C128)
    k_mu_2d_c128<<<nb, kDiagThreads, 0, st>>>(n, (const double2*)u, (const double*)P, make_f64(ph, 0.0, op), out);
  else
    (rows == 1 ? k_mu_2d_c64<1> : k_mu_2d_c64<kGroup>)<<<nb, kDiagThreads, 0, st>>>(
        n, (const float2*)u, (const float*)P, make_params<float>(ph, 0.0, op.center, op.w[0], op.w[1]), out);
  return cudaGetLastError();
}

cudaError_t diag_damping(int dtype, long long n, const void* u, const void* P, int radial, double r_step,
                         double dx, double c12, double c13, double c14, const DiagOut& out, cudaStream_t st) {
  const int nb = blocks_for(n);
  if (dtype == NLS_C128) {
    k_damping<double><<<nb, kDiagThreads, 0, st>>>(n, u, P, radial, r_step, dx, c12, c13, c14, out);
  } else if (radial) {
    k_damping<float><<<nb, kDiagThreads, 0, st>>>(n, u, P, radial, r_step, dx, c12, c13, c14, out);
  } else {
    k_damping_2d_c64<<<nb, kDiagThreads, 0, st>>>(n, (const float2*)u, (const float*)P, dx, c12, c13, c14, out);
  }
  return cudaGetLastError();
}

cudaError_t diag_relerr(int dtype_a, long long n, const void* a, const void* b, const double* P,
                        double c12, double c13, double c14, const DiagOut& out, cudaStream_t st) {
  const int nb = blocks_for(n);
  const double2* bb = reinterpret_cast<const double2*>(b);
  if (dtype_a == NLS_C128) k_relerr<double><<<nb, kDiagThreads, 0, st>>>(n, a, bb, P, c12, c13, c14, out);
  else k_relerr<float><<<nb, kDiagThreads, 0, st>>>(n, a, bb, P, c12, c13, c14, out);
  return cudaGetLastError();
}

}  // namespace nlsg
