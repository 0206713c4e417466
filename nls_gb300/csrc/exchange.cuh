// exchange.cuh -- tagged exchange of node values between the CTAs of one cooperative launch.
//
// A slot is 16 bytes of global memory: 8 bytes of payload and a 32-bit tag, written and read as one
// 128-bit access, so a reader that sees the tag has the payload with it: no fence, no flag and no
// second round trip.  Measured between two SMs: 540 cycles one way on the same side of the L2, 950
// across, against about 2000 for data, fence, flag and the reader's loads one after the other.
// Tags only grow over the life of a buffer (the host keeps the next one), so a slot never has to be
// cleared between launches; the tag sits in the last word of a slot in every layout that uses the
// buffer.  A buffer holds two sets of slots used in turn: a CTA writes a set again only after it
// has read, from every CTA it exchanges with, the set after it, which that CTA published after it
// had read the set before -- so nobody still reads what is overwritten (who reads from whom is
// symmetric: two CTAs exchange when one's nodes lie within the halo width of the other's).
//
// All CTAs of the launch are resident together (cooperative launch), so every wait ends; each is
// bounded all the same, by two to three seconds.  CTAs do not wait for one another to start: beside
// a kernel of another stream that held 24 SMs for longer than that bound, grids that need those SMs
// started when it had ended (144 and 150 CTAs; a grid that fits beside it ran at once), and no wait of
// two contexts' grids that need most SMs, solved at the same time, has expired.
// A wait that expires sets the context's status word; waits that see it set, or that belong to a
// thread that has given up, end at once.  The values a thread gave up on are NaN from then on, and
// NaN spreads with the stencil as the values would have, so a node of the final state is either
// right or NaN, and the host reports the timeout.
#pragma once

#include <stdint.h>

namespace nlsg {

// Added to every tag a thread waits for (a test control: makes the waits expire).
static __device__ unsigned g_exchange_tag_extra = 0;

__device__ __forceinline__ void x_put(uint4* slot, uint64_t data, uint32_t tag) {
  const uint64_t top = (uint64_t)tag << 32;
  asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }"
               ::"l"(slot), "l"(data), "l"(top) : "memory");
}
__device__ __forceinline__ void x_get(const uint4* slot, uint64_t& data, uint32_t& tag) {
  uint64_t top;
  asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }"
               : "=l"(data), "=l"(top) : "l"(slot) : "memory");
  tag = (uint32_t)(top >> 32);
}

// Bound of a wait: polls of about 600 cycles each.
constexpr unsigned kExchangePolls = 1u << 23;

// A NaN as a double and in both parts of a complex64 payload.
constexpr uint64_t kExchangeNaN = ~0ull;

// Waits for the N slots (null: none) to carry `tag` and reads their payloads.  dead: given up, now
// or earlier; the payloads are then NaN, or with FILL = false undefined and the caller takes NaN (the
// fetching warps of rk4_2d_wide_f64: 40^2 takes 4.83 us a step so and 5.41 filled here; the register
// kernels are 2-3 % faster filled here).
template <int N, bool FILL = true>
__device__ __forceinline__ void x_wait(const uint4* const (&slot)[N], uint32_t tag, uint64_t (&data)[N],
                                       int* wait_flag, bool& dead) {
  for (unsigned polls = 0; !dead; ++polls) {
    uint32_t got[N];
    bool all = true;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (slot[i]) x_get(slot[i], data[i], got[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) all = all && (!slot[i] || got[i] == tag);
    if (all) return;
    if (polls >= kExchangePolls) {
      atomicExch(wait_flag, 1);
      dead = true;
    } else if ((polls & 255u) == 255u && *reinterpret_cast<volatile int*>(wait_flag) != 0) {
      dead = true;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (FILL && slot[i]) data[i] = kExchangeNaN;
}

__device__ __forceinline__ uint64_t x_pack(float2 v) {
  return ((uint64_t)__float_as_uint(v.y) << 32) | __float_as_uint(v.x);
}
__device__ __forceinline__ float2 x_c64(uint64_t d) {
  return make_float2(__uint_as_float((uint32_t)d), __uint_as_float((uint32_t)(d >> 32)));
}
__device__ __forceinline__ uint64_t x_pack(double v) { return (uint64_t)__double_as_longlong(v); }
__device__ __forceinline__ double x_f64(uint64_t d) { return __longlong_as_double((long long)d); }

// Cooperative launch.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_coop(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

}  // namespace nlsg
