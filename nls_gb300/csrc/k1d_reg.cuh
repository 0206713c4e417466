// k1d_reg.cuh -- register-resident single-CTA RK4 kernel for complex64 radial grids (sm_103a).
//
// Same contract as rk4_1d_resident on one CTA (all steps of one grid per launch, the state read
// and written once), with the grid held in registers instead of shared memory: thread t owns the
// NPT consecutive nodes t*NPT .. t*NPT+NPT-1, so a node's stencil neighbours are the thread's own
// registers except the K nodes beyond either end, which come from the adjacent lanes by warp
// shuffle and, at a warp boundary, from the adjacent warp through a few bytes of shared memory.
// Every node's state, RK4 accumulator, stage value, pump and 1/r stay in registers for the whole
// launch; the radial operator (D2 + D1 / r, make_laplacian, nls/nls.f90:132-295) and the stage
// updates run on the packed FP32x2 pipe over (re, im) pairs.  As in the 2-D register tile, the
// stage slopes are carried pre-multiplied by dt/2 (q = dt/2 k, constants scaled on the fly).
#pragma once

namespace nlsg {

// Weights of one launch in the working form: scaled by dt/2, as broadcast (w, w) pairs.
template <int K>
struct Reg1DConst {
  float2 w2[2 * K + 1], w1[2 * K + 1];  // D2 and D1 taps (index d + K weights u_{p+d})
  float2 near[K][2 * K + 1];            // the full near-axis rows p < K
  float c3, nc4, c5, c6, c13, c14;      // c3, c4, c5, c6 scaled by dt/2
};

template <int K>
__device__ __forceinline__ Reg1DConst<K> reg1d_const(const Inst1D& I) {
  Reg1DConst<K> c;
  const Params<float>& p = I.pf;
  const float h = p.half_dt;
#pragma unroll
  for (int i = 0; i < 2 * K + 1; ++i) {
    c.w2[i] = f2(h * I.op.w2f[i], h * I.op.w2f[i]);
    c.w1[i] = f2(h * I.op.w1f[i], h * I.op.w1f[i]);
#pragma unroll
    for (int r = 0; r < K; ++r) c.near[r][i] = f2(h * I.op.nearf[r][i], h * I.op.nearf[r][i]);
  }
  c.c3 = h * p.c3; c.nc4 = -(h * p.c4); c.c5 = h * p.c5; c.c6 = h * p.c6;
  c.c13 = p.c13; c.c14 = p.c14;
  return c;
}

// The part of a node's slope that needs no neighbour: a and b of q = (a - i b) u + i L u, with
// r = c12 P / (c13 + c14 |u|^2), a = c3 r - c4, b = c5 |u|^2 + c6 r.
template <int K>
__device__ __forceinline__ float2 reg1d_point(float2 v, float pc, const Reg1DConst<K>& c) {
  const float sq = __fmaf_rn(v.x, v.x, v.y * v.y);
  const float r = pc * rcp_approx(__fmaf_rn(c.c14, sq, c.c13));
  return f2(__fmaf_rn(c.c3, r, c.nc4), __fmaf_rn(c.c5, sq, c.c6 * r));
}

// One RK4 stage S over the thread's NPT nodes.  t holds the stage input (re, im per node); on
// return it holds the next stage's input (S < 4), or u the new state (S = 4).  L / R: the K nodes
// before the thread's first and after its last node.  Nodes at or beyond n stay zero.  NEAR: the
// warp holds the nodes at the axis (a warp-uniform choice; within it every lane evaluates both
// forms of its first K nodes and thread 0 takes the near-axis rows).  ab: the nodes' reg1d_point, or
// null to evaluate it here.
template <int K, int NPT, int S, bool NEAR>
__device__ __forceinline__ void reg1d_stage_form(float2 (&t)[NPT], float2 (&acc)[NPT], float2 (&u)[NPT],
                                                 const float (&pc)[NPT], const float (&ir)[NPT],
                                                 const float2 (&L)[K], const float2 (&R)[K], int p0, int n,
                                                 const Reg1DConst<K>& c, const float2* ab) {
  auto at = [&](int idx) -> float2 { return idx < 0 ? L[K + idx] : (idx >= NPT ? R[idx - NPT] : t[idx]); };
  float2 nt[NPT];
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    // D2 u + (1/r) D1 u, the centre tap of D1 being zero
    float2 d2 = mul2(c.w2[K], at(i));
    float2 d1 = mul2(c.w1[0], at(i - K));
#pragma unroll
    for (int d = 1; d <= K; ++d) {
      d2 = fma2(c.w2[K - d], at(i - d), d2);
      d2 = fma2(c.w2[K + d], at(i + d), d2);
      if (d < K) d1 = fma2(c.w1[K - d], at(i - d), d1);
      d1 = fma2(c.w1[K + d], at(i + d), d1);
    }
    float2 lu = fma2(f2(ir[i], ir[i]), d1, d2);
    if (NEAR && i < K) {
      // near-axis rows (only thread 0 holds nodes p = i < K, as NPT >= K) carry the mirror folds
      // at r = 0; the weights of nodes before 0 are zero
      float2 ln = mul2(c.near[i < K ? i : 0][0], at(i - K));
#pragma unroll
      for (int d = 1; d <= 2 * K; ++d) ln = fma2(c.near[i < K ? i : 0][d], at(i - K + d), ln);
      lu = f2(p0 == 0 ? ln.x : lu.x, p0 == 0 ? ln.y : lu.y);
    }
    // q = (a - i b) u + i L u
    const float2 v = t[i];
    const float2 w_ab = ab ? ab[i] : reg1d_point<K>(v, pc[i], c);
    const float a = w_ab.x, b = w_ab.y;
    const float2 q = f2(__fmaf_rn(a, v.x, __fmaf_rn(b, v.y, -lu.y)), __fmaf_rn(a, v.y, __fmaf_rn(-b, v.x, lu.x)));
    if (S == 1) acc[i] = q;
    else if (S == 4) acc[i] = add2(acc[i], q);
    else acc[i] = fma2(f2(2.f, 2.f), q, acc[i]);
    if (S < 4) {
      const float2 w = S == 3 ? fma2(f2(2.f, 2.f), q, u[i]) : add2(u[i], q);
      nt[i] = f2(p < n ? w.x : 0.f, p < n ? w.y : 0.f);
    } else {
      // the state stays in registers across steps: nodes beyond the grid must stay zero
      const float2 w = fma2(f2(1.f / 3.f, 1.f / 3.f), acc[i], u[i]);
      u[i] = f2(p < n ? w.x : 0.f, p < n ? w.y : 0.f);
    }
  }
  if (S < 4) {
#pragma unroll
    for (int i = 0; i < NPT; ++i) t[i] = nt[i];
  }
}
template <int K, int NPT, int S>
__device__ __forceinline__ void reg1d_stage(float2 (&t)[NPT], float2 (&acc)[NPT], float2 (&u)[NPT],
                                            const float (&pc)[NPT], const float (&ir)[NPT],
                                            const float2 (&L)[K], const float2 (&R)[K], int p0, bool near, int n,
                                            const Reg1DConst<K>& c, const float2* ab = nullptr) {
  if (near) reg1d_stage_form<K, NPT, S, true>(t, acc, u, pc, ir, L, R, p0, n, c, ab);
  else reg1d_stage_form<K, NPT, S, false>(t, acc, u, pc, ir, L, R, p0, n, c, ab);
}

// Exchange of warp-end nodes within a CTA: [2 parities][nw + 2 warps][2 ends][K] values in shared
// memory, the first and the last warp's entries (beyond the CTA) zero.  Returns bytes.
__host__ __device__ inline size_t reg1d_exchange_bytes(int K, int nw) {
  return (size_t)2 * (nw + 2) * 2 * K * sizeof(float2);
}
struct Reg1DEx {
  float2 *mine, *nb;   // this lane's end of its warp (lanes 0 and 31), and the neighbour's end it reads
  int parity;          // values between the two parities
};
template <int K>
__device__ __forceinline__ Reg1DEx reg1d_exchange(float2* ex, int warp, int lane, int nw) {
  for (int i = threadIdx.x; i < 2 * (nw + 2) * 2 * K; i += blockDim.x) ex[i] = f2(0.f, 0.f);
  Reg1DEx e;
  e.mine = ex + ((warp + 1) * 2 + (lane == 31 ? 1 : 0)) * K;
  e.nb = lane == 31 ? ex + ((warp + 2) * 2 + 0) * K : ex + (warp * 2 + 1) * K;
  e.parity = (nw + 2) * 2 * K;
  __syncthreads();
  return e;
}

// The K nodes before the thread's first node (L) and after its last (R): from the adjacent lanes
// by shuffle, across a warp boundary from the neighbouring warp's published end nodes (stage
// parity double-buffers them, so one CTA barrier per stage suffices), zero beyond the CTA.  Without
// branches: every lane reads a neighbour's end and selects (branches cost a lone warp a quarter of a
// stage: 4096 nodes on one CTA ran at 930 cycles a stage, 250 of them resolving).
template <int K, int NPT, int S>
__device__ __forceinline__ void reg1d_halo(const float2 (&t)[NPT], float2 (&L)[K], float2 (&R)[K], const Reg1DEx& e,
                                           int lane) {
  const int off = (S & 1) ? e.parity : 0;
  const bool first = lane == 0, lastl = lane == 31;
  if (first || lastl) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      e.mine[off + k] = f2(lastl ? t[NPT - K + k].x : t[k].x, lastl ? t[NPT - K + k].y : t[k].y);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float2 v = e.nb[off + k];
    const float lx = __shfl_up_sync(0xffffffffu, t[NPT - K + k].x, 1), ly = __shfl_up_sync(0xffffffffu, t[NPT - K + k].y, 1);
    const float rx = __shfl_down_sync(0xffffffffu, t[k].x, 1), ry = __shfl_down_sync(0xffffffffu, t[k].y, 1);
    L[k] = f2(first ? v.x : lx, first ? v.y : ly);
    R[k] = f2(lastl ? v.x : rx, lastl ? v.y : ry);
  }
}

template <int K, int NPT>
__global__ void __launch_bounds__(512) rk4_1d_reg(const Inst1D* __restrict__ insts) {
  static_assert(NPT >= K, "a thread's neighbours must lie within the adjacent lanes");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const Inst1D& I = insts[blockIdx.x];
  const int n = I.n;
  const int p0 = tid * NPT;
  const bool near = warp == 0;
  const Reg1DEx e = reg1d_exchange<K>(reinterpret_cast<float2*>(smem_raw), warp, lane, nw);
  const Reg1DConst<K> c = reg1d_const<K>(I);
  const float h = (float)I.op.h;
  const float c12 = I.pf.c12;
  const float2* __restrict__ Ug = reinterpret_cast<const float2*>(I.u);
  const float* __restrict__ Pg = reinterpret_cast<const float*>(I.P);
  float2 u[NPT], t[NPT], acc[NPT];
  float pc[NPT], ir[NPT];
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    const bool in = p < n;
    u[i] = in ? Ug[p] : f2(0.f, 0.f);
    pc[i] = in ? c12 * Pg[p] : 0.f;
    ir[i] = p >= K ? 1.f / ((float)p * h) : 0.f;
    acc[i] = f2(0.f, 0.f);
  }
  float2 L[K], R[K];
  const int64_t steps = I.steps;
  for (int64_t step = 0; step < steps; ++step) {
#pragma unroll
    for (int i = 0; i < NPT; ++i) t[i] = u[i];
    reg1d_halo<K, NPT, 1>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 1>(t, acc, u, pc, ir, L, R, p0, near, n, c);
    reg1d_halo<K, NPT, 2>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 2>(t, acc, u, pc, ir, L, R, p0, near, n, c);
    reg1d_halo<K, NPT, 3>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 3>(t, acc, u, pc, ir, L, R, p0, near, n, c);
    reg1d_halo<K, NPT, 4>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 4>(t, acc, u, pc, ir, L, R, p0, near, n, c);
  }
  float2* __restrict__ Uo = reinterpret_cast<float2*>(I.u);
#pragma unroll
  for (int i = 0; i < NPT; ++i)
    if (p0 + i < n) Uo[p0 + i] = u[i];
}

// Cluster form (grids too long for one CTA): the grid is cut into cl segments [q0, q1), one per
// CTA of a thread-block cluster.  Each CTA holds its segment and up to H = 4K halo nodes on either
// side, [lo, hi), in registers with the single-CTA layout above, and runs the four stages over all
// of them with CTA-local barriers only; a node within K of [lo, hi)'s ends reads zeros past them,
// so after stage s the values within sK of those ends are wrong, and after the four stages exactly
// the segment itself is exact.  At the end of each step every CTA pushes the H new values at
// either end of its segment into its neighbours' halo buffers (distributed shared memory, double
// buffered by step parity: a buffer written at step s is read at the start of step s + 1 and
// written again only after the cluster's next meeting) and the cluster meets once; the next step
// starts by taking its halo nodes from those buffers.  Every CTA runs the same loop with no early
// exit, so the cluster's barriers always match.
template <int K, int NPT>
__global__ void __launch_bounds__(512) rk4_1d_reg_cl(const Inst1D* __restrict__ insts, int cl) {
  static_assert(NPT >= K, "a thread's neighbours must lie within the adjacent lanes");
  constexpr int H = 4 * K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  float2* ex = reinterpret_cast<float2*>(smem_raw);
  float2* halo = ex + reg1d_exchange_bytes(K, nw) / sizeof(float2);   // [2 parities][2 sides: left, right][H]
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int inst = blockIdx.x / cl, rank = blockIdx.x % cl;
  const Inst1D& I = insts[inst];
  const int n = I.n;
  const int seg = (n + cl - 1) / cl;
  const int q0 = min(n, rank * seg), q1 = min(n, q0 + seg);
  const int lo = max(0, q0 - H), hi = min(n, q1 + H);
  const int p0 = lo + tid * NPT;
  const bool near = warp == 0 && lo == 0;
  const Reg1DEx e = reg1d_exchange<K>(ex, warp, lane, nw);
  const Reg1DConst<K> c = reg1d_const<K>(I);
  const float h = (float)I.op.h;
  const float c12 = I.pf.c12;
  const float2* __restrict__ Ug = reinterpret_cast<const float2*>(I.u);
  const float* __restrict__ Pg = reinterpret_cast<const float*>(I.P);
  float2 u[NPT], t[NPT], acc[NPT];
  float pc[NPT], ir[NPT];
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    const bool in = p < hi;
    u[i] = in ? Ug[p] : f2(0.f, 0.f);
    pc[i] = in ? c12 * Pg[p] : 0.f;
    ir[i] = p >= K ? 1.f / ((float)p * h) : 0.f;
    acc[i] = f2(0.f, 0.f);
  }
  // the neighbours' halo buffers (their right side takes this segment's first H nodes, their
  // left side its last H)
  float2* const lnb = rank > 0 ? cluster.map_shared_rank(halo, rank - 1) : nullptr;
  float2* const rnb = rank < cl - 1 ? cluster.map_shared_rank(halo, rank + 1) : nullptr;
  cluster.sync();   // every CTA of the cluster is running before the first push
  float2 L[K], R[K];
  const int64_t steps = I.steps;
  for (int64_t step = 0; step < steps; ++step) {
    const int par = (int)(step & 1);
    if (step > 0) {
      const float2* hb = halo + (par ^ 1) * 2 * H;
#pragma unroll
      for (int i = 0; i < NPT; ++i) {
        const int p = p0 + i;
        if (p >= lo && p < q0) u[i] = hb[p - (q0 - H)];
        if (p >= q1 && p < hi) u[i] = hb[H + (p - q1)];
      }
    }
#pragma unroll
    for (int i = 0; i < NPT; ++i) t[i] = u[i];
    reg1d_halo<K, NPT, 1>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 1>(t, acc, u, pc, ir, L, R, p0, near, hi, c);
    reg1d_halo<K, NPT, 2>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 2>(t, acc, u, pc, ir, L, R, p0, near, hi, c);
    reg1d_halo<K, NPT, 3>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 3>(t, acc, u, pc, ir, L, R, p0, near, hi, c);
    reg1d_halo<K, NPT, 4>(t, L, R, e, lane);
    reg1d_stage<K, NPT, 4>(t, acc, u, pc, ir, L, R, p0, near, hi, c);
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int p = p0 + i;
      if (lnb && p >= q0 && p < q0 + H) lnb[(par * 2 + 1) * H + (p - q0)] = u[i];
      if (rnb && p >= q1 - H && p < q1) rnb[(par * 2 + 0) * H + (p - (q1 - H))] = u[i];
    }
    cluster.sync();
  }
  float2* __restrict__ Uo = reinterpret_cast<float2*>(I.u);
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int p = p0 + i;
    if (p >= q0 && p < q1) Uo[p] = u[i];
  }
}

}  // namespace nlsg
