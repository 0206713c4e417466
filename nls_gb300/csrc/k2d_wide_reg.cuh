// k2d_wide_reg.cuh -- one complex64 square grid held in registers by all SMs (sm_103a).
//
// The streaming step walks each strip of a grid row by row: a chain of rows that a small or middling
// grid has too few strips to hide (777^2: 12.1 us a step, a quarter of the rate of 4096^2; 128^2: 9.2 us),
// and one launch a step.  Here every CTA of a cooperative launch keeps one register tile
// (k2d_reg.cuh) for all steps of the launch.  It evaluates its output tile and a halo of H = 4K nodes
// around it, so the four stages of a step need CTA barriers only; then the tiles exchange the frames
// of H nodes at their edges through tagged slots (exchange.cuh), every thread fetching a share of
// the halo, and pass them to the owning threads through shared memory.  Every launch starts with an
// exchange, so a CTA reads and writes only its own output tile of the state in global memory.
//
// The arithmetic is reg_stage's, which agrees bit for bit with the streaming kernel's.  What bounds it:
// the stages' arithmetic over the region (latency at 2-4 warps a scheduler), then one exchange
// (540-950 cycles one way) a step.  Measured, order 3: 128^2 2.1 us a step, 777^2 6.0 (1361 warp
// instructions a step, issue slots 44 % busy).
#pragma once

#include "k2d_reg_stage.cuh"

namespace nlsg {

template <int K, int NW, int NJ>
struct WideRegCfg {
  typedef RegCfg<K, NW, NJ> G;
  static constexpr int H = G::H;
  static constexpr int HALO = G::RX * G::RY - G::TX * G::TY;   // halo nodes of a region
  static constexpr size_t SMEM = G::EXCH + (size_t)HALO * 8;
  // Index of region node (x, y) in the halo buffer: rows above, rows below, columns at the sides.
  static __device__ __forceinline__ int index(int x, int y) {
    if (y < H) return y * G::RX + x;
    if (y >= G::RY - H) return (H + y - (G::RY - H)) * G::RX + x;
    return 2 * H * G::RX + (y - H) * 2 * H + (x < H ? x : x - (G::RX - 2 * H));
  }
  static __device__ __forceinline__ void node(int k, int& x, int& y) {
    if (k < 2 * H * G::RX) {
      x = k % G::RX;
      y = k / G::RX;
      if (y >= H) y += G::RY - 2 * H;
    } else {
      const int j = k - 2 * H * G::RX;
      x = j % (2 * H);
      y = H + j / (2 * H);
      if (x >= H) x += G::RX - 2 * H;
    }
  }
};

template <int K, int NW, int NJ>
__global__ void __launch_bounds__(NW * 32, 1)
rk4_2d_wide_reg(const __grid_constant__ Inst2D I, uint4* xbuf, uint32_t tag, int* wait_flag) {
  typedef WideRegCfg<K, NW, NJ> C;
  typedef RegCfg<K, NW, NJ> G;
  constexpr int H = G::H, NH = (C::HALO + G::NT - 1) / G::NT;   // halo nodes a thread fetches
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float4* const exch = reinterpret_cast<float4*>(smem_raw);
  float2* const hbuf = reinterpret_cast<float2*>(smem_raw + G::EXCH);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = 2 * lane, y0 = warp * NJ;     // region position of the thread's first node
  const int n = I.n;
  const int tyi = blockIdx.x / I.tiles_x, txi = blockIdx.x - tyi * I.tiles_x;
  const int rx0 = txi * G::TX - H, ry0 = tyi * G::TY - H;   // grid position of region node (0, 0)
  const int gx = rx0 + x0, gy0 = ry0 + y0;
  const bool edge = rx0 < 0 || ry0 < 0 || rx0 + G::RX > n || ry0 + G::RY > n;
  const RegConst c = reg_const<K>(I.pf);
  const float2 c12 = f2(I.pf.c12, I.pf.c12);
  float2* __restrict__ Ug = reinterpret_cast<float2*>(I.u[0]);
  const float* __restrict__ Pg = reinterpret_cast<const float*>(I.P);
  const bool xout = x0 >= H && x0 < G::RX - H;
  // rows whose pair lies in the grid (per node), in the output tile, in its frame
  unsigned dom0 = 0, dom1 = 0, out = 0, frame = 0;
  float2 uX[NJ], uY[NJ], pc[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int y = y0 + j, gy = gy0 + j;
    const bool yin = gy >= 0 && gy < n;
    const bool i0 = yin && gx >= 0 && gx < n, i1 = yin && gx + 1 >= 0 && gx + 1 < n;
    const bool o = xout && y >= H && y < G::RY - H;
    const size_t q = (size_t)gy * n + gx;
    const float2 a = o && i0 ? Ug[q] : f2(0.f, 0.f), b = o && i1 ? Ug[q + 1] : f2(0.f, 0.f);
    uX[j] = f2(a.x, b.x);
    uY[j] = f2(a.y, b.y);
    pc[j] = mul2(c12, f2(i0 ? Pg[q] : 0.f, i1 ? Pg[q + 1] : 0.f));
    dom0 |= (unsigned)i0 << j;
    dom1 |= (unsigned)i1 << j;
    out |= (unsigned)o << j;
    frame |= (unsigned)(o && (x0 < 2 * H || x0 >= G::RX - 2 * H || y < 2 * H || y >= G::RY - 2 * H)) << j;
  }
  // the nodes this thread fetches (-1: none, or outside the grid)
  int fetch[NH];
#pragma unroll
  for (int i = 0; i < NH; ++i) {
    const int k = threadIdx.x + i * G::NT;
    int x = 0, y = 0;
    C::node(k < C::HALO ? k : 0, x, y);
    x += rx0;
    y += ry0;
    fetch[i] = k < C::HALO && x >= 0 && x < n && y >= 0 && y < n ? y * n + x : -1;
  }
  bool dead = false;
  const uint32_t extra = g_exchange_tag_extra;
  const size_t set_slots = (size_t)n * n;
  const int64_t steps = I.steps;
  for (int64_t step = 0; step < steps; ++step, ++tag) {
    uint4* const slots = xbuf + (size_t)(step & 1) * set_slots;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      if ((frame >> j) & 1u) {
        uint4* const s = slots + (size_t)(gy0 + j) * n + gx;
        if ((dom0 >> j) & 1u) x_put(s, x_pack(f2(uX[j].x, uY[j].x)), tag);
        if ((dom1 >> j) & 1u) x_put(s + 1, x_pack(f2(uX[j].y, uY[j].y)), tag);
      }
    __syncwarp();   // no lane waits before every lane of its warp has published
    const uint4* want[NH];
    uint64_t got[NH];
#pragma unroll
    for (int i = 0; i < NH; ++i) {
      want[i] = fetch[i] >= 0 ? slots + fetch[i] : nullptr;
      got[i] = 0;   // outside the grid: zero
    }
    x_wait<NH>(want, tag + extra, got, wait_flag, dead);
#pragma unroll
    for (int i = 0; i < NH; ++i) {
      const int k = threadIdx.x + i * G::NT;
      if (k < C::HALO) hbuf[k] = x_c64(got[i]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      if (!((out >> j) & 1u)) {
        const float2* const h = hbuf + C::index(x0, y0 + j);   // the pair's entries are adjacent
        uX[j] = f2(h[0].x, h[1].x);
        uY[j] = f2(h[0].y, h[1].y);
      }
    if (edge) {
      reg_step<K, NW, NJ, true>(uX, uY, pc, dom0, dom1, exch, warp, lane, c, [] {});
      // nodes beyond the grid stay zero
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const bool i0 = (dom0 >> j) & 1u, i1 = (dom1 >> j) & 1u;
        uX[j] = f2(i0 ? uX[j].x : 0.f, i1 ? uX[j].y : 0.f);
        uY[j] = f2(i0 ? uY[j].x : 0.f, i1 ? uY[j].y : 0.f);
      }
    } else {
      reg_step<K, NW, NJ, false>(uX, uY, pc, dom0, dom1, exch, warp, lane, c, [] {});
    }
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    if ((out >> j) & 1u) {
      const size_t q = (size_t)(gy0 + j) * n + gx;
      if ((dom0 >> j) & 1u) Ug[q] = f2(uX[j].x, uY[j].x);
      if ((dom1 >> j) & 1u) Ug[q + 1] = f2(uX[j].y, uY[j].y);
    }
}

}  // namespace nlsg
