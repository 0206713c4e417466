// k2d_reg_stage.cuh -- the register tile's layout and its RK4 stages (complex64, sm_103a), shared by
// rk4_2d_reg (k2d_reg.cuh, one step a launch) and rk4_2d_wide_reg (k2d_wide_reg.cuh, many).
#pragma once

#include "nls_common.cuh"

namespace nlsg {

template <int K, int NW, int NJ>
struct RegCfg {
  static constexpr int RX = 64;
  static constexpr int RY = NW * NJ;
  static constexpr int NT = NW * 32;
  static constexpr int H = 4 * K;
  static constexpr int TX = RX - 2 * H;
  static constexpr int TY = RY - 2 * H;
  static constexpr size_t STAGE_U = (size_t)RX * RY * 8;            // complex64 state box
  static constexpr size_t STAGE_P = (size_t)RX * RY * 4;            // pump box
  static constexpr size_t EXCH = (size_t)2 * NW * 2 * K * RX * 8;   // strip-end rows, 2 parities
  static constexpr size_t DESC = sizeof(Inst2D);                   // descriptor copy (TMA path)
  static constexpr size_t OFF_DESC = STAGE_U + STAGE_P + EXCH;      // two descriptor slots
  static constexpr size_t OFF_CTRL = OFF_DESC + 2 * DESC;
  static constexpr size_t SMEM = OFF_CTRL + 128;                    // + control block
  static_assert(NJ >= K && NJ <= 32 && TY > 0, "tile layout");
  static_assert(DESC % 16 == 0, "a descriptor bulk copy moves a multiple of 16 bytes");
};

// Per-tile constants as broadcast pairs (both halves equal) for the packed pipe.  Slopes are carried
// in units of the stencil's outermost weight w (1/h^2 at K = 1, 1/(12 h^2) at K = 2), in which the
// stencil's weights are whole numbers, q = k / w:
//   q = a u - i (b + C) u + i S,   a = c3 r - c4,  b = c5 |u|^2 + c6 r  (c3 .. c6 divided by w),
//   K = 1: C = 4, S = s1;  K = 2: C = 60, S = 16 s1 - s2  (s_d: sum of the four neighbours at distance d)
// and RK4 reads t2 = u + w dt/2 q1, t3 = u + w dt/2 q2, t4 = u + w dt q3,
// u' = u + w dt/6 (q1 + 2 q2 + 2 q3 + q4): no multiplication by a stencil weight is left.
struct RegConst {
  float2 cw, c16, n16, c3, nc4, c5, c6, c13, c14, two, m1, hw, dtw, dw6;
};

template <int K>
__device__ __forceinline__ RegConst reg_const(const Params<float>& p) {
  RegConst c;
  auto both = [](float v) { return f2(v, v); };
  c.cw = both(K == 1 ? 4.f : 60.f);
  c.c16 = both(16.f); c.n16 = both(-16.f);
  c.c3 = both(p.u3); c.nc4 = both(-p.u4); c.c5 = both(p.u5); c.c6 = both(p.u6);
  c.c13 = both(p.c13); c.c14 = both(p.c14);
  c.two = both(2.f); c.m1 = both(-1.f);
  c.hw = both(p.hw); c.dtw = both(p.dtw); c.dw6 = both(p.dw6);
  return c;
}

// One RK4 stage S over the warp's strip.  tX/tY hold the stage input of the NJ rows (planar node
// pairs); on return they hold the next stage's input (S < 4), or u holds the new state (S = 4).
// Every node of the region is evaluated; values near the region edge are wrong (their stencils
// reach outside the region) but the valid part shrinks by K per stage and the output tile is what
// remains after four.  EDGE: the region reaches outside the grid, whose nodes must read as zero
// (the reference's truncated operator), so stage outputs there are reset to zero.
template <int K, int NW, int NJ, int S, bool EDGE>
__device__ __forceinline__ void reg_stage(float2 (&tX)[NJ], float2 (&tY)[NJ], float2 (&aX)[NJ],
                                          float2 (&aY)[NJ], float2 (&uX)[NJ], float2 (&uY)[NJ],
                                          const float2 (&pc)[NJ], unsigned dom0, unsigned dom1,
                                          float4* __restrict__ exch, int warp, int lane,
                                          const RegConst& c) {
  float4* ex = exch + (S & 1) * (NW * 2 * K * 32);
  // publish the strip's first and last K rows of the stage input, then read the neighbours'
#pragma unroll
  for (int k = 0; k < K; ++k) {
    ex[((warp * 2 + 0) * K + k) * 32 + lane] = make_float4(tX[k].x, tX[k].y, tY[k].x, tY[k].y);
    ex[((warp * 2 + 1) * K + k) * 32 + lane] =
        make_float4(tX[NJ - K + k].x, tX[NJ - K + k].y, tY[NJ - K + k].x, tY[NJ - K + k].y);
  }
  __syncthreads();
  float2 upX[K], upY[K], dnX[K], dnY[K];  // rows y0 - K + k and y0 + NJ + k
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (warp > 0) a = ex[(((warp - 1) * 2 + 1) * K + k) * 32 + lane];
    if (warp < NW - 1) b = ex[(((warp + 1) * 2 + 0) * K + k) * 32 + lane];
    upX[k] = f2(a.x, a.y); upY[k] = f2(a.z, a.w);
    dnX[k] = f2(b.x, b.y); dnY[k] = f2(b.z, b.w);
  }
  auto rowX = [&](int r) -> float2 { return r < 0 ? upX[K + r] : (r >= NJ ? dnX[r - NJ] : tX[r]); };
  auto rowY = [&](int r) -> float2 { return r < 0 ? upY[K + r] : (r >= NJ ? dnY[r - NJ] : tY[r]); };

  float2 oX[NJ], oY[NJ];   // next stage's input
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const float2 X = tX[j], Y = tY[j];
    float2 sX, nY;  // S of the real plane, -S of the imaginary one
    if (K == 1) {
      // left neighbour of the pair's first node, right neighbour of its second
      const float lx = __shfl_up_sync(0xffffffffu, X.y, 1), ly = __shfl_up_sync(0xffffffffu, Y.y, 1);
      const float rx = __shfl_down_sync(0xffffffffu, X.x, 1), ry = __shfl_down_sync(0xffffffffu, Y.x, 1);
      sX = add2(add2(f2(lx + X.y, X.x + rx), rowX(j - 1)), rowX(j + 1));
      nY = fma2(c.m1, rowY(j + 1), fma2(c.m1, rowY(j - 1), f2(-ly - Y.y, -Y.x - ry)));
    } else {
      // both nodes of the pairs to the left (L) and right (R)
      const float2 LX = f2(__shfl_up_sync(0xffffffffu, X.x, 1), __shfl_up_sync(0xffffffffu, X.y, 1));
      const float2 LY = f2(__shfl_up_sync(0xffffffffu, Y.x, 1), __shfl_up_sync(0xffffffffu, Y.y, 1));
      const float2 RX = f2(__shfl_down_sync(0xffffffffu, X.x, 1), __shfl_down_sync(0xffffffffu, X.y, 1));
      const float2 RY = f2(__shfl_down_sync(0xffffffffu, Y.x, 1), __shfl_down_sync(0xffffffffu, Y.y, 1));
      const float2 s1X = add2(add2(f2(LX.y + X.y, X.x + RX.x), rowX(j - 1)), rowX(j + 1));
      const float2 s1Y = add2(add2(f2(LY.y + Y.y, Y.x + RY.x), rowY(j - 1)), rowY(j + 1));
      const float2 n2X = fma2(c.m1, rowX(j + 2), fma2(c.m1, rowX(j - 2), f2(-LX.x - RX.x, -LX.y - RX.y)));
      const float2 s2Y = add2(add2(add2(LY, RY), rowY(j - 2)), rowY(j + 2));
      sX = fma2(c.c16, s1X, n2X);
      nY = fma2(c.n16, s1Y, s2Y);
    }
    // r = c12 P / (c13 + c14 |u|^2), |u|^2 per node in scalar arithmetic (a packed square of a
    // register pair with itself costs extra register moves)
    const float2 sq = f2(__fmaf_rn(X.x, X.x, Y.x * Y.x), __fmaf_rn(X.y, X.y, Y.y * Y.y));
    const float2 den = fma2(c.c14, sq, c.c13);
    const float2 r = mul2(pc[j], f2(rcp_approx(den.x), rcp_approx(den.y)));
    const float2 a = fma2(c.c3, r, c.nc4);
    const float2 bw = fma2(c.c5, sq, fma2(c.c6, r, c.cw));
    const float2 kX = fma2(a, X, fma2(bw, Y, nY));
    const float2 kY = fma2(a, Y, fma2(neg2(bw), X, sX));
    if (S == 1) {
      aX[j] = kX;
      aY[j] = kY;
    } else if (S == 4) {
      aX[j] = add2(aX[j], kX);
      aY[j] = add2(aY[j], kY);
    } else {
      aX[j] = fma2(c.two, kX, aX[j]);
      aY[j] = fma2(c.two, kY, aY[j]);
    }
    if (S < 4) {
      float2 vX, vY;
      // Next stage input.  Packed or scalar by tile shape, as measured on the GB300: scalar is
      // faster for strips of up to 10 rows and at order 5, packed for 12-row strips at order 3 (the
      // register allocation differs, not the work).
      constexpr bool kScalarUpdate = NJ <= 10 || K == 2;
      const float2 w = S == 3 ? c.dtw : c.hw;
      if (kScalarUpdate) {
        vX = f2(__fmaf_rn(w.x, kX.x, uX[j].x), __fmaf_rn(w.x, kX.y, uX[j].y));
        vY = f2(__fmaf_rn(w.x, kY.x, uY[j].x), __fmaf_rn(w.x, kY.y, uY[j].y));
      } else {
        vX = fma2(w, kX, uX[j]);
        vY = fma2(w, kY, uY[j]);
      }
      if (EDGE) {
        const bool i0 = (dom0 >> j) & 1u, i1 = (dom1 >> j) & 1u;
        vX = f2(i0 ? vX.x : 0.f, i1 ? vX.y : 0.f);
        vY = f2(i0 ? vY.x : 0.f, i1 ? vY.y : 0.f);
      }
      oX[j] = vX;
      oY[j] = vY;
    } else {
      if (NJ <= 10 || K == 2) {  // scalar for the same shapes as the stage-input update
        const float th = c.dw6.x;
        uX[j] = f2(__fmaf_rn(th, aX[j].x, uX[j].x), __fmaf_rn(th, aX[j].y, uX[j].y));
        uY[j] = f2(__fmaf_rn(th, aY[j].x, uY[j].x), __fmaf_rn(th, aY[j].y, uY[j].y));
      } else {
        uX[j] = fma2(c.dw6, aX[j], uX[j]);
        uY[j] = fma2(c.dw6, aY[j], uY[j]);
      }
    }
  }
  if (S < 4) {
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      tX[j] = oX[j];
      tY[j] = oY[j];
    }
  }
}

// The four stages of a step; mid() runs between the second and the third.
template <int K, int NW, int NJ, bool EDGE, typename Mid>
__device__ __forceinline__ void reg_step(float2 (&uX)[NJ], float2 (&uY)[NJ], const float2 (&pc)[NJ],
                                         unsigned dom0, unsigned dom1, float4* __restrict__ exch,
                                         int warp, int lane, const RegConst& c, Mid&& mid) {
  float2 tX[NJ], tY[NJ], aX[NJ], aY[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    tX[j] = uX[j];
    tY[j] = uY[j];
  }
  reg_stage<K, NW, NJ, 1, EDGE>(tX, tY, aX, aY, uX, uY, pc, dom0, dom1, exch, warp, lane, c);
  reg_stage<K, NW, NJ, 2, EDGE>(tX, tY, aX, aY, uX, uY, pc, dom0, dom1, exch, warp, lane, c);
  mid();
  reg_stage<K, NW, NJ, 3, EDGE>(tX, tY, aX, aY, uX, uY, pc, dom0, dom1, exch, warp, lane, c);
  reg_stage<K, NW, NJ, 4, EDGE>(tX, tY, aX, aY, uX, uY, pc, dom0, dom1, exch, warp, lane, c);
}

}  // namespace nlsg
