// k2d_wide.cu -- single square grids spread over the whole GPU by cooperative launches (sm_103a):
// rk4_2d_wide_f64 (complex128, k2d_wide.cuh) and rk4_2d_wide_reg (complex64, k2d_wide_reg.cuh).
#include <algorithm>

#include "kernels.h"
#include "nls_common.cuh"
#include "exchange.cuh"
#include "k2d_wide.cuh"
#include "k2d_wide_reg.cuh"

namespace nlsg {

// ---- one complex128 grid over the whole GPU (k2d_wide.cuh)

static constexpr size_t kWideSmem = 227 * 1024;

// The tiling with the shortest stage by a model in cycles fitted to measured stages (order 3): one
// lane a node 3240 at one warp a CTA (40^2), 3830 at 4 (128^2), 4960 at 14 (256^2), 14 230 at 54
// (512^2); two lanes a node 2900 at 1, 3120 at 8, 6600 at 28 warps (the same grids).  So two lanes
// up to about 300 nodes a CTA, one beyond, and above 1800 nodes a CTA the stage kernels, whose
// launches amortise there (600^2: 40.2 us a step against 41.1 here; 512^2: 30.3 against 27.8).  The
// stages above are those of warps that fetched their own halo; with fetching warps 40^2 takes 5.2 us a
// step, 128^2 5.7, 256^2 9.6 (stage kernels 8.5, 9.2 and 13.7).
Wide2DPlan wide_2d_plan(int K, int n, int sms) {
  Wide2DPlan best;
  double best_cost = 1e300;
  for (int gx = 1; gx <= std::min(sms, n); ++gx)
    for (int gy = 1; gx * gy <= sms && gy <= n; ++gy) {
      const int w = (n + gx - 1) / gx, h = (n + gy - 1) / gy;
      if (w * h > 1800 || wide_2d_smem(K, w, h) > kWideSmem) continue;
      const int inner = w > 2 * K && h > 2 * K ? (w - 2 * K) * (h - 2 * K) : 0, ring = w * h - inner;
      for (int lanes = 0; lanes < 2; ++lanes) {
        const int per = lanes ? 16 : 32;
        const int ew = (ring + per - 1) / per, iw = (inner + per - 1) / per, total = ew + iw;
        // warps beyond what a CTA gives the edge take their turn twice; the halo's size stands for
        // publishing and fetching it
        const int passes = (ew + (lanes ? 12 : 8) - 1) / (lanes ? 12 : 8);
        const double cost = (lanes ? std::max(2600.0 + 40.0 * total + 1500.0 * (passes - 1), 236.0 * total)
                                   : std::max(2900.0 + 140.0 * total + 2500.0 * (passes - 1), 263.0 * total)) +
                            (gx * gy > 1 ? 100.0 : 0.0) + 3.0 * 2 * K * (w + h) + 0.1 * gx * gy;
        if (cost >= best_cost) continue;
        best_cost = cost;
        best.gx = gx;
        best.gy = gy;
        best.lanes = lanes != 0;
        // fetching warps: up to four values a lane at a time
        best.halo_warps = gx * gy > 1 ? std::min(4, (4 * K * (w + h) + 95) / 96) : 0;
        best.edge_warps = std::min(ew, lanes ? 12 : 8);
        best.threads = 32 * (best.halo_warps + best.edge_warps +
                             std::min(iw, (lanes ? 32 : 24) - best.halo_warps - best.edge_warps));
        best.smem = wide_2d_smem(K, w, h);
      }
    }
  return best;
}

size_t wide_2d_slot_bytes(int n) { return (size_t)2 * 2 * n * n * sizeof(uint4); }

cudaError_t launch_2d_wide(int K, const Inst2D& I, const Wide2DPlan& p, void* xbuf, uint32_t tag, int* wait_flag,
                           cudaStream_t s) {
  const Wide2D g{p.gx, p.gy, p.halo_warps, p.edge_warps};
  auto go = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmem);
    if (e != cudaSuccess) return e;
    return launch_coop(kern, dim3(p.gx * p.gy), dim3(p.threads), p.smem, s, I, g, (uint4*)xbuf, tag, wait_flag);
  };
  if (K == 1) return p.lanes ? go(rk4_2d_wide_f64<1, true>) : go(rk4_2d_wide_f64<1, false>);
  if (K == 2) return p.lanes ? go(rk4_2d_wide_f64<2, true>) : go(rk4_2d_wide_f64<2, false>);
  return cudaErrorInvalidValue;
}

// ---- one complex64 grid over the whole GPU (k2d_wide_reg.cuh)

// Calls f(kernel, config) for region shape number `shape`, lowest regions first; false past the last.
template <int K, typename F>
static bool wide_reg_shape_k(int shape, F&& f) {
  switch (shape) {
#define NLSG_WIDE_REG(I, NW, NJ) \
  case I: f(rk4_2d_wide_reg<K, NW, NJ>, WideRegCfg<K, NW, NJ>()); return true;
    case 0: if constexpr (K == 1) f(rk4_2d_wide_reg<K, 8, 2>, WideRegCfg<K, 8, 2>()); return true;
    NLSG_WIDE_REG(1, 8, 3)
    NLSG_WIDE_REG(2, 8, 4)
    NLSG_WIDE_REG(3, 12, 4)
    NLSG_WIDE_REG(4, 16, 4)
    NLSG_WIDE_REG(5, 16, 5)
    NLSG_WIDE_REG(6, 16, 6)
#undef NLSG_WIDE_REG
  }
  return false;
}
template <typename F>
static bool wide_reg_shape(int K, int shape, F&& f) {
  return K == 1 ? wide_reg_shape_k<1>(shape, f) : (K == 2 ? wide_reg_shape_k<2>(shape, f) : false);
}

// The lowest region whose tiles all fit: fewer rows a warp, shorter stages (a warp's rows, not the
// region's, make its length: 72 rows as 9 warps of 8 took as long as 96 as 12 of 8, 6.0 us a step at
// order 3; 96 as 16 of 6 takes 5.7).  us a step, order 3, by rows of the region (16 / 24 / 32): 64^2
// 1.99 / 2.09 / 2.32, 128^2 2.07 / 2.28 / 2.58; 512^2 3.14 with 48 rows, 3.78 with 64; streaming 8.7 to
// 9.3.  Beyond one tile an SM (840 a side at order 3, 720 at order 5) the streaming and tile kernels;
// the largest here against those: 840^2 5.5 and 11.1, order 5 700^2 7.5 and 9.5.  Sixteen warps leave 128
// registers a thread, and the largest regions spill a little (bytes a thread: 6 rows a warp 68 at order 3 and
// 124 at order 5, 5 rows 24 and 4 rows 16 at order 5); the times are with the spills.
WideReg2DPlan wide_reg_2d_plan(int K, int n, int sms) {
  WideReg2DPlan best;
  bool more = true;
  for (int shape = 0; more && !best.tiles; ++shape) {
    more = wide_reg_shape(K, shape, [&](auto, auto cfg) {
      typedef typename decltype(cfg)::G G;
      const int tx = (n + G::TX - 1) / G::TX, ty = (n + G::TY - 1) / G::TY;
      if (tx * ty > sms) return;
      best.shape = shape;
      best.tiles_x = tx;
      best.tiles = tx * ty;
    });
  }
  return best;
}

size_t wide_reg_2d_slot_bytes(int n) { return (size_t)2 * n * n * sizeof(uint4); }

cudaError_t launch_2d_wide_reg(int K, const Inst2D& I, const WideReg2DPlan& p, void* xbuf, uint32_t tag, int* wait_flag,
                               cudaStream_t s) {
  cudaError_t e = cudaErrorInvalidValue;
  wide_reg_shape(K, p.shape, [&](auto kern, auto cfg) {
    typedef decltype(cfg) C;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e == cudaSuccess)
      e = launch_coop(kern, dim3(p.tiles), dim3(C::G::NT), C::SMEM, s, I, (uint4*)xbuf, tag, wait_flag);
  });
  return e;
}

cudaError_t exchange_tag_extra_set_2d(unsigned extra) {
  return cudaMemcpyToSymbol(g_exchange_tag_extra, &extra, sizeof(extra));
}

}  // namespace nlsg
