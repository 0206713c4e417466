// k1d_wide.cuh -- one radial grid spread over the whole GPU (sm_103a).
//
// A single solve on one CTA or one cluster leaves most SMs idle: the step is a chain of four
// dependent stages whose length grows with the nodes an SM holds.  Here the grid is cut into
// segments, one per CTA of a cooperative launch, as many as it takes to hold one warp's worth of
// work per SM sub-partition.  A CTA evaluates its segment and H = 4K S halo nodes on either side, so
// S whole RK4 steps need only CTA barriers (after each stage the values within K more nodes of the
// region's ends are wrong, after S steps the segment itself is still exact); then the CTAs exchange
// the H values at either end of their segments through tagged slots (exchange.cuh).  Every launch
// starts with an exchange, so a CTA reads and writes only its own segment of the state in global
// memory and the update in place is safe.
//
// What bounds it: complex64, the latency of four dependent stages (about 350 cycles each at order 5)
// and the exchange, 540-950 cycles over S steps; complex128, the chain of a stage and the FP64
// instructions of one warp per sub-partition (f64_node.cuh) -- so there two lanes share a node, one
// for the real and one for the imaginary part, which halves them: 218 warp instructions and 1250
// cycles a stage at order 5, the FP64 pipe 50 % busy.
//
// Measured, us a step, one CTA or cluster before and this kernel: complex64 order 5, 4096 nodes 4.64
// and 0.67; complex128 order 5, 1000 nodes 5.3 and 2.5; order 7, 2501 nodes 8.5 and 3.0.
#pragma once

namespace nlsg {

// Geometry of a launch: segment length, steps per exchange.
struct Wide1D {
  int seg, S;
};

// reg1d_halo and reg1d_stage in one: a warp alone on its sub-partition evaluates what its nodes need
// alone between publishing its ends and the CTA barrier, where the two calls leave it to wait (order 5,
// 4096 nodes: 0.86 -> 0.70 us a step; orders 3 and 7 the same).  Waiting for the neighbouring warps
// alone, through tagged slots of shared memory, took 1.1: the polls cost more than the barrier.
template <int K, int NPT, int S>
__device__ __forceinline__ void wide_1d_stage(float2 (&t)[NPT], float2 (&acc)[NPT], float2 (&u)[NPT],
                                              const float (&pc)[NPT], const float (&ir)[NPT], int p0, bool near, int n,
                                              const Reg1DConst<K>& c, const Reg1DEx& e, int lane) {
  const int off = (S & 1) ? e.parity : 0;
  const bool first = lane == 0, lastl = lane == 31;
  if (first || lastl) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      e.mine[off + k] = f2(lastl ? t[NPT - K + k].x : t[k].x, lastl ? t[NPT - K + k].y : t[k].y);
  }
  float2 L[K], R[K], ab[NPT];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    L[k] = f2(__shfl_up_sync(0xffffffffu, t[NPT - K + k].x, 1), __shfl_up_sync(0xffffffffu, t[NPT - K + k].y, 1));
    R[k] = f2(__shfl_down_sync(0xffffffffu, t[k].x, 1), __shfl_down_sync(0xffffffffu, t[k].y, 1));
  }
#pragma unroll
  for (int i = 0; i < NPT; ++i) ab[i] = reg1d_point<K>(t[i], pc[i], c);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float2 v = e.nb[off + k];
    L[k] = f2(first ? v.x : L[k].x, first ? v.y : L[k].y);
    R[k] = f2(lastl ? v.x : R[k].x, lastl ? v.y : R[k].y);
  }
  reg1d_stage<K, NPT, S>(t, acc, u, pc, ir, L, R, p0, near, n, c, ab);
}

template <int K, int NPT>
__global__ void __launch_bounds__(256) rk4_1d_wide(const __grid_constant__ Inst1D I, Wide1D g, uint4* xbuf,
                                                   uint32_t tag, int* wait_flag) {
  static_assert(NPT >= K, "a thread's neighbours must lie within the adjacent lanes");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int n = I.n, H = 4 * K * g.S;
  const int q0 = blockIdx.x * g.seg, q1 = min(n, q0 + g.seg);
  const int lo = max(0, q0 - H), hi = min(n, q1 + H);
  const int p0 = lo + tid * NPT;
  const bool near = warp == 0 && lo == 0;
  const Reg1DEx e = reg1d_exchange<K>(reinterpret_cast<float2*>(smem_raw), warp, lane, nw);
  const Reg1DConst<K> c = reg1d_const<K>(I);
  const float h = (float)I.op.h;
  const float c12 = I.pf.c12;
  float2* __restrict__ Ug = reinterpret_cast<float2*>(I.u);
  const float* __restrict__ Pg = reinterpret_cast<const float*>(I.P);
  float2 u[NPT], t[NPT], acc[NPT];
  float pc[NPT], ir[NPT];
  bool halo[NPT], edge[NPT];
  bool any_halo = false;
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    const bool own = p >= q0 && p < q1;
    u[i] = own ? Ug[p] : f2(0.f, 0.f);
    pc[i] = p < hi ? c12 * Pg[p] : 0.f;
    ir[i] = p >= K ? 1.f / ((float)p * h) : 0.f;
    acc[i] = f2(0.f, 0.f);
    halo[i] = (p >= lo && p < q0) || (p >= q1 && p < hi);
    edge[i] = own && ((q0 > 0 && p < q0 + H) || (q1 < n && p >= q1 - H));
    any_halo = any_halo || halo[i];
  }
  bool dead = false;
  const uint32_t extra = g_exchange_tag_extra;
  int set = 0;
  for (int64_t left = I.steps; left > 0; ++tag, set ^= 1) {
    uint4* const slots = xbuf + (size_t)set * n;
#pragma unroll
    for (int i = 0; i < NPT; ++i)
      if (edge[i]) x_put(slots + p0 + i, x_pack(u[i]), tag);
    __syncwarp();   // no lane waits before every lane of its warp has published
    if (any_halo) {
      const uint4* want[NPT];
      uint64_t got[NPT];
#pragma unroll
      for (int i = 0; i < NPT; ++i) want[i] = halo[i] ? slots + p0 + i : nullptr;
      x_wait<NPT>(want, tag + extra, got, wait_flag, dead);
#pragma unroll
      for (int i = 0; i < NPT; ++i)
        if (halo[i]) u[i] = x_c64(got[i]);
    }
    const int run = left < g.S ? (int)left : g.S;
    left -= run;
    for (int k = 0; k < run; ++k) {
#pragma unroll
      for (int i = 0; i < NPT; ++i) t[i] = u[i];
      wide_1d_stage<K, NPT, 1>(t, acc, u, pc, ir, p0, near, hi, c, e, lane);
      wide_1d_stage<K, NPT, 2>(t, acc, u, pc, ir, p0, near, hi, c, e, lane);
      wide_1d_stage<K, NPT, 3>(t, acc, u, pc, ir, p0, near, hi, c, e, lane);
      wide_1d_stage<K, NPT, 4>(t, acc, u, pc, ir, p0, near, hi, c, e, lane);
    }
  }
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    if (p >= q0 && p < q1) Ug[p] = u[i];
  }
}

// complex128: thread 2i of a CTA holds the real part of the region's node i, thread 2i + 1 its
// imaginary part; stage inputs pass through shared memory.  Each thread evaluates the operator on
// the other part, which is what its slope needs (k_re = A u_re + (B - w_c) u_im - (L u)_im), with
// the operations of f64_slope_1d in their order.
template <int K>
__global__ void __launch_bounds__(512) rk4_1d_wide_f64(const __grid_constant__ Inst1D I, Wide1D g, uint4* xbuf,
                                                       uint32_t tag, int* wait_flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, part = tid & 1, li = (tid >> 1) + K;
  const int nodes = blockDim.x >> 1, W = nodes + 2 * K;
  double2* const buf0 = reinterpret_cast<double2*>(smem_raw);
  double2* const buf1 = buf0 + W;
  const int n = I.n, H = 4 * K * g.S;
  const int q0 = blockIdx.x * g.seg, q1 = min(n, q0 + g.seg);
  const int p = q0 - H + (tid >> 1);
  const bool in = p >= 0 && p < n && p < q1 + H;
  const bool own = in && p >= q0 && p < q1;
  const bool halo = in && !own;
  const bool edge = own && ((q0 > 0 && p < q0 + H) || (q1 < n && p >= q1 - H));
  for (int i = tid; i < 4 * W; i += blockDim.x) reinterpret_cast<double*>(buf0)[i] = 0.0;
  double* __restrict__ Ug = reinterpret_cast<double*>(I.u);
  const Node64<K> nd = node64<K>(I.op, p, reinterpret_cast<const double*>(I.P), in);
  double u = own ? Ug[2 * (size_t)p + part] : 0.0, acc = 0.0;
  bool dead = false;
  const uint32_t extra = g_exchange_tag_extra;
  const F64Lane lane = f64_lane(part, I.f64);
  // reads of a stage: both parts of the node, the other part of its neighbours
  auto slope = [&](const double2* buf, auto&& between) -> double {
    const double* o = reinterpret_cast<const double*>(buf + li) + (1 - part);
    double other[2 * K + 1];
#pragma unroll
    for (int d = 0; d < 2 * K + 1; ++d) other[d] = o[2 * (d - K)];
    return f64_slope_1d_lanes<K>(buf[li], other, nd.row, nd.p, nd.P, nd.p_ok, lane, I.f64, between);
  };
  // acc += 2 q of the stage before, while the next stage waits for its exchanges
  auto twice = [&](double q) { asm volatile("fma.rn.f64 %0, %1, %2, %0;" : "+d"(acc) : "d"(2.0), "d"(q)); };
  auto put = [&](double2* buf, double v) {
    if (in) reinterpret_cast<double*>(buf + li)[part] = v;
    __syncthreads();
  };
  __syncthreads();   // the zeroed buffers
  int set = 0;
  for (int64_t left = I.steps; left > 0; ++tag, set ^= 1) {
    uint4* const slots = xbuf + (size_t)set * 2 * n;
    if (edge) x_put(slots + 2 * (size_t)p + part, x_pack(u), tag);
    __syncwarp();   // no lane waits before every lane of its warp has published
    if (halo) {
      const uint4* want[1] = {slots + 2 * (size_t)p + part};
      uint64_t got[1];
      x_wait<1>(want, tag + extra, got, wait_flag, dead);
      u = x_f64(got[0]);
    }
    put(buf0, u);
    const int run = left < g.S ? (int)left : g.S;
    left -= run;
    for (int k = 0; k < run; ++k) {
      const double q1 = slope(buf0, [] {});
      acc = q1;
      put(buf1, dfma(I.f64.half_dt, q1, u));
      const double q2 = slope(buf1, [] {});
      put(buf0, dfma(I.f64.half_dt, q2, u));
      const double q3 = slope(buf0, [&] { twice(q2); });
      put(buf1, dfma(I.f64.dt, q3, u));
      const double q = slope(buf1, [&] { twice(q3); });
      u = dfma(I.f64.dt6, dadd(acc, q), u);
      if (k + 1 < run) put(buf0, u);
      else __syncthreads();   // buf1 is read until here, buf0 is written after the next exchange
    }
  }
  if (own) Ug[2 * (size_t)p + part] = u;
}

}  // namespace nlsg
