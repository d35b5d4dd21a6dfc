// 32-bit numbers as sums of 16-bit ones for the tensor cores.
//
// A row is scaled by a power of two s so that |x / s| < 4096, and cut into h (a multiple of 2), l (a multiple of 2^-10, |l| <= 1) and m (the rest,
// |m| <= 2^-11), each exact in 16 bits but for the last bits of m (2^-34 of the scale).  Products h h are multiples of 4 below 2^24, so that their sums
// stay exact in a 32-bit accumulator up to 2^26; h l, l h, l l, h m and m h go to an accumulator of their own, 2^11 times smaller, and what is left
// out is 2^-34 of a product of scales.
#pragma once
#include "common.cuh"

namespace split16 {

using namespace packed;
using namespace umma_lo;

// the largest magnitude of three; a value that is no number stays one
__device__ __forceinline__ float max_abs(float a, float b, float c) {
  float d;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max_abs(float a, pair_t p) {
  const float2 x = unpack(p);
  return max_abs(a, x.x, x.y);
}

// power of two s with |x| / s < 4096 for all |x| <= mx, and 1 / s (clamped to 2^-99 .. 2^88); huge: beyond 2^100, or no number
struct Scale {
  float s, inv;
  bool huge;
};
__device__ __forceinline__ Scale scale_of(float mx) {
  int e = (int)((__float_as_uint(mx) & 0x7fffffffu) >> 23);
  Scale r;
  r.huge = e >= 227;
  e = min(max(e, 39), 226);
  r.s = __int_as_float((e - 11) << 23);
  r.inv = __int_as_float((265 - e) << 23);
  return r;
}
__device__ __forceinline__ uint32_t half2_bits(pair_t v) {
  const float2 x = unpack(v);
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(x.y), "f"(x.x));
  return r;
}
constexpr uint64_t kGrid1 = 0x4bc000004bc00000ull;       // 1.5 * 2^24, twice: adding and subtracting rounds to multiples of 2
constexpr uint64_t kGrid2 = 0x4640000046400000ull;       // 1.5 * 2^13, twice: multiples of 2^-10
// two scaled numbers
__device__ __forceinline__ void split3(pair_t y, uint32_t& h, uint32_t& l, uint32_t& m) {
  const pair_t a = psub(padd(y, kGrid1), kGrid1), r = psub(y, a), b = psub(padd(r, kGrid2), kGrid2);
  h = half2_bits(a);
  l = half2_bits(b);
  m = half2_bits(psub(r, b));
}
// ---- the instructions around tensor memory that these products use
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
               "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
constexpr uint32_t idesc(int N, int mn) { return umma_idesc_f16(0, 128, N) | ((uint32_t)mn << 16); }

// mbar_wait for kernels that end by themselves: a wait of more than LLMSS_SPIN_TIMEOUT_NS sets *quit (shared memory), and waits that find it set
// end.  What the block has computed since is worth nothing: the kernel leaves its state as it was and its work to another one
static __device__ __noinline__ void wait_bar_loop(uint32_t bar, uint32_t parity, volatile int* quit) {
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
    uint32_t n = 0, ok;
    do {
      asm volatile(
          "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    } while (!ok && ++n < 4096);
    if (ok || *quit) return;
    if (globaltimer_ns() - t0 > LLMSS_SPIN_TIMEOUT_NS) *quit = 1;
  }
}
__device__ __forceinline__ void wait_bar(uint64_t* bar, uint32_t parity, int* quit) {
  if (!mbar_try_wait(bar, parity & 1)) wait_bar_loop(smem_u32(bar), parity & 1, quit);
}
// arrival of a warp whose lanes have written shared memory or read or written tensor memory
__device__ __forceinline__ void arrive_warp(uint64_t* bar) {
  tcgen05_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
__device__ __forceinline__ float ld_nc(const float* p) {       // (volatile: stays in front of the waits that follow it)
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_nc4(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

}  // namespace split16
