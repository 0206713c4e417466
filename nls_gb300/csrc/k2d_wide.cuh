// k2d_wide.cuh -- one complex128 square grid held on chip by all SMs for a whole launch (sm_103a).
//
// The stage kernels run four launches a step, each reading the state, the pump and the RK4 sum from
// L2: about 2 us a launch whatever the grid's size, and idle FP64 pipes in between.  Here the grid
// is cut into one tile per CTA of a cooperative launch; state, stage inputs, RK4 sum and pump stay
// in shared memory for all steps of the launch (72 bytes a node and two halo frames), and after each
// stage the K outermost rows and columns of every tile pass to its neighbours through tagged slots
// (exchange.cuh).  FP64 instructions bound the step (f64_node.cuh), so no halo is recomputed; the
// exchange (540-950 cycles one way) hides behind arithmetic: the first warps of a CTA fetch the
// neighbours' values, the next own the tile's edge nodes -- they evaluate what their nodes need alone
// (the reservoir and the coefficients) meanwhile, then the rest, and publish -- and the other warps
// evaluate the nodes that need no neighbour's value.  One CTA barrier a stage.
// Measured, order 3, us a step, stage kernels and this one: 40^2 8.5 and 4.9-5.2, 128^2 9.2 and 5.7, 256^2
// 13.7 and 9.6 (530 warp instructions a stage and warp, FP64 pipe 40 % busy, integer pipe 46 %).
// LANES: two adjacent lanes share a node, one for each part, which shortens the chain of a node but
// repeats the reservoir's quotient and the loop around it; for tiles of few warps, where the chain
// bounds the stage.
#pragma once

namespace nlsg {

// Tiles along each axis, warps that fetch the halo (0: a single tile) and warps that own edge nodes.
struct Wide2D {
  int gx, gy, halo_warps, edge_warps;
};

template <int K>
struct Wide2DTile {
  int x0, y0, w, h, pitch, ring, inner, halo;
  __host__ __device__ Wide2DTile(int n, int gx, int gy, int bx, int by) {
    // tiles of near-equal size
    x0 = (int)((int64_t)bx * n / gx);
    y0 = (int)((int64_t)by * n / gy);
    w = (int)((int64_t)(bx + 1) * n / gx) - x0;
    h = (int)((int64_t)(by + 1) * n / gy) - y0;
    pitch = w + 2 * K;
    inner = w > 2 * K && h > 2 * K ? (w - 2 * K) * (h - 2 * K) : 0;
    ring = w * h - inner;
    halo = 2 * K * (w + h);
  }
  // Node k of the tile, ring nodes first: offset in a frame of pitch w + 2K.
  __device__ int node(int k) const {
    int x, y;
    if (inner == 0) {
      x = k % w;
      y = k / w;
    } else if (k < 2 * K * w) {
      x = k % w;
      y = k / w;
      if (y >= K) y += h - 2 * K;
    } else if (k < ring) {
      const int j = k - 2 * K * w, c = j % (2 * K);
      y = K + j / (2 * K);
      x = c < K ? c : w - 2 * K + c;
    } else {
      const int j = k - ring;
      x = K + j % (w - 2 * K);
      y = K + j / (w - 2 * K);
    }
    return (y + K) * pitch + x + K;
  }
  // Halo node k: rows above and below, columns left and right.
  __device__ int halo_node(int k) const {
    int x, y;
    if (k < 2 * K * w) {
      x = k % w;
      y = k / w;
      y = y < K ? y - K : h + y - K;
    } else {
      const int j = k - 2 * K * w;
      y = j % h;
      x = j / h;
      x = x < K ? x - K : w + x - K;
    }
    return (y + K) * pitch + x + K;
  }
};

// Shared memory of a tile: three frames, then the RK4 sum, the pump and the node lists.
inline __host__ __device__ size_t wide_2d_smem(int K, int w, int h) {
  const size_t frame = (size_t)(w + 2 * K) * (h + 2 * K) * 16, nodes = (size_t)w * h;
  return 3 * frame + nodes * (16 + 8 + 4) + (size_t)2 * K * (w + h) * 8;
}

template <int K, bool LANES>
__global__ void __launch_bounds__(LANES ? 1024 : 768) rk4_2d_wide_f64(const __grid_constant__ Inst2D I, Wide2D g,
                                                                      uint4* xbuf, uint32_t tag, int* wait_flag) {
  constexpr int SH = LANES ? 1 : 0;   // a node takes 1 << SH adjacent threads
  constexpr int PARTS = LANES ? 1 : 2;   // parts a thread holds: `part` or both
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int n = I.n;
  const Wide2DTile<K> T(n, g.gx, g.gy, blockIdx.x % g.gx, blockIdx.x / g.gx);
  const int nodes = T.w * T.h, frame = T.pitch * (T.h + 2 * K);
  // frames and sums as separate values: element 2 k + part of an array of nodes
  double* const U = reinterpret_cast<double*>(smem_raw);
  double* const T1 = U + 2 * frame;
  double* const T2 = T1 + 2 * frame;
  double* const acc = T2 + 2 * frame;
  F2* const P = reinterpret_cast<F2*>(acc + 2 * nodes);       // the pump as pairs
  int2* const hlist = reinterpret_cast<int2*>(P + nodes);     // frame offset, node in the grid (-1: none)
  int* const list = reinterpret_cast<int*>(hlist + T.halo);
  const int halo_threads = 32 * g.halo_warps, edge_threads = 32 * g.edge_warps;
  const int tid = (int)threadIdx.x - halo_threads;   // negative: a fetching thread
  const bool edge = tid >= 0 && tid < edge_threads;
  const int part = LANES ? threadIdx.x & 1 : 0;
  const F64Lane lane = f64_lane(part, I.f64);
  double* __restrict__ Ug = reinterpret_cast<double*>(I.u[0]);
  const double* __restrict__ Pg = reinterpret_cast<const double*>(I.P);
  auto grid_node = [&](int off) -> int {
    return (T.y0 + off / T.pitch - K) * n + T.x0 + off % T.pitch - K;
  };
  for (int i = threadIdx.x; i < 6 * frame; i += blockDim.x) U[i] = 0.0;
  for (int k = threadIdx.x; k < T.halo; k += blockDim.x) {
    const int off = T.halo_node(k);
    const int y = T.y0 + off / T.pitch - K, x = T.x0 + off % T.pitch - K;
    hlist[k] = make_int2(off, x >= 0 && x < n && y >= 0 && y < n ? y * n + x : -1);
  }
  __syncthreads();   // zeroed frames, halo list
  // this thread's (pair's) nodes: list entries first, first + stride, .. below last
  const int mine = tid >> SH, owners = edge_threads >> SH;
  const int first = edge ? mine : T.ring + mine - owners;
  const int stride = edge ? owners : ((int)blockDim.x - halo_threads >> SH) - owners;
  const int last = tid < 0 ? 0 : (edge ? T.ring : nodes);   // a fetching thread owns none
  for (int k = first; k < last && tid >= 0; k += stride) {
    const int off = T.node(k);
    list[k] = off;
    const size_t q = (size_t)grid_node(off);
    if (part == 0) P[k] = f2_pump(Pg[q]);
#pragma unroll
    for (int c = 0; c < PARTS; ++c) {
      const double v = Ug[2 * q + part + c];
      U[2 * off + part + c] = v;
      if (edge) x_put(xbuf + 2 * q + part + c, x_pack(v), tag);
    }
  }
  __syncthreads();
  bool dead = false;
  const uint32_t extra = g_exchange_tag_extra;
  const size_t set_slots = 2 * (size_t)n * n;
  const int64_t steps = I.steps;
  // exchange number 4 step + s - 1 brings the halo of stage s's input, from the set of its parity
  if (tid < 0) {
    for (int64_t step = 0; step < steps; ++step) {
#pragma unroll 1
      for (int s = 1; s <= 4; ++s, ++tag) {
        double* const in = s == 1 ? U : (s == 3 ? T2 : T1);
        const uint4* const from = xbuf + (size_t)((s - 1) & 1) * set_slots;
        // element 2 k + part of the halo list
        for (int k0 = threadIdx.x; k0 < 2 * T.halo; k0 += 4 * halo_threads) {
          const uint4* want[4];
          uint64_t got[4];
          int at[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = k0 + i * halo_threads;
            const int2 h = k < 2 * T.halo ? hlist[k >> 1] : make_int2(0, -1);
            at[i] = 2 * h.x + (k & 1);
            want[i] = h.y >= 0 ? from + 2 * (size_t)h.y + (k & 1) : nullptr;
          }
          x_wait<4, false>(want, tag + extra, got, wait_flag, dead);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (want[i]) in[at[i]] = x_f64(dead ? kExchangeNaN : got[i]);
        }
        __syncwarp();
        asm volatile("barrier.arrive 1, %0;" ::"r"(halo_threads + edge_threads) : "memory");
        __syncthreads();
      }
    }
    return;
  }
  for (int64_t step = 0; step < steps; ++step) {
#pragma unroll 1
    for (int s = 1; s <= 4; ++s, ++tag) {
      double* const in = s == 1 ? U : (s == 3 ? T2 : T1);
      double* const out = s == 4 ? U : (s == 2 ? T2 : T1);
      uint4* const to = xbuf + (size_t)(s & 1) * set_slots;
      // the coefficients of this thread's first node, which need no neighbour (idle lanes repeat one)
      const bool any = LANES ? first - (mine & 15) < last : first < last;
      const int k1 = first < last ? first : last - 1;
      double A1 = 0.0, bw1 = 0.0;
      auto coeffs = [&](int k, double& A, double& bw) {
        const int off = list[k];
        const double2 v = reinterpret_cast<const double2*>(in)[off];
        const F2 p = P[k];
        const double* const pg = Pg + grid_node(off);
        if constexpr (LANES) f64_coeffs_2d_lanes(v, p, f2_pump_ok(p), pg, lane, I.f64, A, bw);
        else f64_coeffs_2d(v.x, v.y, p, f2_pump_ok(p), pg, I.f64, A, bw);
      };
      if (any) coeffs(k1, A1, bw1);
      if (edge && halo_threads) {
        __syncwarp();
        asm volatile("barrier.sync 1, %0;" ::"r"(halo_threads + edge_threads) : "memory");
      }
      const bool publish = edge && (s < 4 || step + 1 < steps);
      if constexpr (LANES) {
        // walked by whole warps (the lanes of a pair exchange values): a warp's first entry decides
        // whether it goes on, entries past the end repeat the last one
        for (int k = first; k - (mine & 15) < last; k += stride) {
          const bool live = k < last;
          const int kk = live ? k : last - 1, off = list[kk];
          const double* const o = in + 2 * off + (1 - part);
          double other[4 * K];
#pragma unroll
          for (int d = 1; d <= K; ++d) {
            other[4 * d - 4] = o[-2 * d];
            other[4 * d - 3] = o[2 * d];
            other[4 * d - 2] = o[-2 * d * T.pitch];
            other[4 * d - 1] = o[2 * d * T.pitch];
          }
          const double2 v = *reinterpret_cast<const double2*>(in + 2 * off);
          if (k != first) coeffs(kk, A1, bw1);
          double a = s > 1 ? acc[2 * kk + part] : 0.0;
          const double q = f64_slope_2d_lanes<K>(v, other, A1, bw1, lane, I.f64);
          const double t = f64_stage_lane(s, U[2 * off + part], a, q, I.f64);
          if (live) {
            if (s < 4) acc[2 * kk + part] = a;
            out[2 * off + part] = t;
            if (publish) x_put(to + 2 * (size_t)grid_node(off) + part, x_pack(t), tag + 1);
          }
        }
      } else {
        for (int k = first; k < last; k += stride) {
          const int off = list[k];
          const double2* const c = reinterpret_cast<const double2*>(in) + off;
          const double2 v = c[0];
          double vx[4 * K], vy[4 * K];
#pragma unroll
          for (int d = 1; d <= K; ++d) {
            const double2 n0 = c[-d], n1 = c[d], n2 = c[-d * T.pitch], n3 = c[d * T.pitch];
            vx[4 * d - 4] = n0.x; vx[4 * d - 3] = n1.x; vx[4 * d - 2] = n2.x; vx[4 * d - 1] = n3.x;
            vy[4 * d - 4] = n0.y; vy[4 * d - 3] = n1.y; vy[4 * d - 2] = n2.y; vy[4 * d - 1] = n3.y;
          }
          double2 q, a = s > 1 ? reinterpret_cast<double2*>(acc)[k] : make_double2(0.0, 0.0);
          if (k != first) coeffs(k, A1, bw1);
          f64_slope_2d<K>(v.x, v.y, vx, vy, A1, bw1, I.f64, q.x, q.y);
          const double2 t = f64_stage(s, reinterpret_cast<double2*>(U)[off], a, q, I.f64);
          if (s < 4) reinterpret_cast<double2*>(acc)[k] = a;
          reinterpret_cast<double2*>(out)[off] = t;
          if (publish) {
            uint4* const slot = to + 2 * (size_t)grid_node(off);
            x_put(slot, x_pack(t.x), tag + 1);
            x_put(slot + 1, x_pack(t.y), tag + 1);
          }
        }
      }
      __syncthreads();
    }
  }
  for (int k = first; k < last; k += stride) {
    const int off = list[k];
#pragma unroll
    for (int c = 0; c < PARTS; ++c) Ug[2 * (size_t)grid_node(off) + part + c] = U[2 * off + part + c];
  }
}

}  // namespace nlsg
