// K6 norm_residual: (x [+ x2] [+ residual]) -> new residual, LayerNorm / RMSNorm of it.
//
// Replaces the reference's separate ATen add + layer_norm launches (gptj_modeling.py:296,310,496; gpt_bigcode_modeling.py:367,379,404,407) and provides the
// capability of the never-instantiated FastLayerNorm wrapper (layers.py:217-256).
// One CTA per row, row held in registers (16-byte vector loads), fp32 statistics,
// two-pass variance.  Memory-bound: reads x(+res) once, writes normed(+res) once.
#include "common.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kMaxVec = 4;  // 256 thr * 4 vec * 8 elem = H <= 8192

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < kThreads / 32) ? red[l] : 0.f;
  return warp_sum(t);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) norm_residual_kernel(
    const T* __restrict__ x, const T* __restrict__ x2, const T* residual_in, T* residual_out,
    const T* __restrict__ weight, const T* __restrict__ bias, T* __restrict__ out, int H, int64_t ldx,
    int64_t ldx2, int64_t ldr, int64_t ldo, float eps, int kind) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[kThreads / 32];
  const int row = blockIdx.x;
  const int nvec = H >> 3;
  float v[kMaxVec][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i) {
    const int c = threadIdx.x + i * kThreads;
    if (c < nvec) {
      uint4 raw = *reinterpret_cast<const uint4*>(x + row * ldx + c * 8);
      unpack8<T>(raw, v[i]);
      if (x2 != nullptr) {
        float t[8];
        raw = *reinterpret_cast<const uint4*>(x2 + row * ldx2 + c * 8);
        unpack8<T>(raw, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += t[j];
      }
      if (residual_in != nullptr) {
        float t[8];
        raw = *reinterpret_cast<const uint4*>(residual_in + row * ldr + c * 8);
        unpack8<T>(raw, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += t[j];
      }
      if (residual_out != nullptr) {
        *reinterpret_cast<uint4*>(residual_out + row * ldr + c * 8) = pack8<T>(v[i]);
        // the normalisation sees the value as stored (same rounding as the unfused path)
        unpack8<T>(pack8<T>(v[i]), v[i]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += (kind == LLMSS_NORM_RMS) ? v[i][j] * v[i][j] : v[i][j];
    }
  }
  float mean = 0.f, rstd;
  if (kind == LLMSS_NORM_RMS) {
    float ss = block_sum(sum, red);
    rstd = rsqrtf(ss / (float)H + eps);
  } else {
    mean = block_sum(sum, red) / (float)H;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxVec; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float d = v[i][j] - mean;
          sq += d * d;
        }
      }
    }
    float var = block_sum(sq, red) / (float)H;
    rstd = rsqrtf(var + eps);
  }
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i) {
    const int c = threadIdx.x + i * kThreads;
    if (c < nvec) {
      float w[8], b[8], o[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(weight + c * 8), w);
      if (bias != nullptr) unpack8<T>(*reinterpret_cast<const uint4*>(bias + c * 8), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float y = (v[i][j] - mean) * rstd * w[j];
        o[j] = (bias != nullptr) ? y + b[j] : y;
      }
      *reinterpret_cast<uint4*>(out + row * ldo + c * 8) = pack8<T>(o);
    }
  }
}

__device__ __forceinline__ uint4 ld_in_order(const void* p) {
  uint4 r;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

// The same at prompt sizes: WPR warps per row (8 16-byte vectors per lane: rows up to 2048 numbers per warp), four warps a block.  A
// block per row spends its time in barriers and in the tail of its few loads: here a lane has all of its loads in flight at once
// and a row of up to 2048 numbers needs no barrier.  The sums are those of the block-per-row kernel, in its order (a warp stands for
// NP of its eight warps): a row's result does not depend on how many rows the batch has.  4004 x 2048, three inputs and two outputs (82 MB)
// on B200: 21.3 us with a block per row, 16.8 us (sums in an order of their own took as long).
template <typename T, int WPR>
__global__ void __launch_bounds__(128) norm_rows_kernel(
    const T* __restrict__ x, const T* __restrict__ x2, const T* residual_in, T* residual_out,
    const T* __restrict__ weight, const T* __restrict__ bias, T* __restrict__ out, int M, int H, int64_t ldx,
    int64_t ldx2, int64_t ldr, int64_t ldo, float eps, int kind) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int V = 8, NP = V / WPR;      // a lane's vectors i, i + NP, ... are those of one thread of the block-per-row kernel
  __shared__ float red[2][4 / WPR][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % WPR;
  const int row = blockIdx.x * (4 / WPR) + warp / WPR;
  const int nvec = row < M ? H >> 3 : 0, c0 = part * 32 + lane;      // (past the last row nothing is read or written)
  uint4 rx[V], ry[V], rr[V];
  // no branch between the loads (a predicated load is not moved past another): past the row's end the row's first vector, not counted
  const int64_t r0 = min(row, M - 1);
  auto fetch = [&](uint4 (&r)[V], const T* p) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = c0 + i * 32 * WPR;
      r[i] = ld_in_order(p + (c < nvec ? c * 8 : 0));
    }
  };
  fetch(rx, x + r0 * ldx);
  if (residual_in != nullptr) fetch(rr, residual_in + r0 * ldr);
  if (x2 != nullptr) fetch(ry, x2 + r0 * ldx2);
  float v[V][8];
  float sums[NP];
#pragma unroll
  for (int m = 0; m < NP; ++m) sums[m] = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = c0 + i * 32 * WPR;
    float t[8];
    unpack8<T>(rx[i], v[i]);
    if (x2 != nullptr) {
      unpack8<T>(ry[i], t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] += t[j];
    }
    if (residual_in != nullptr) {
      unpack8<T>(rr[i], t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] += t[j];
    }
    if (residual_out != nullptr) {
      const uint4 r = pack8<T>(v[i]);
      if (c < nvec) *reinterpret_cast<uint4*>(residual_out + row * ldr + c * 8) = r;
      unpack8<T>(r, v[i]);      // the normalisation sees the value as stored
    }
    if (c < nvec) {
#pragma unroll
      for (int j = 0; j < 8; ++j) sums[i % NP] += (kind == LLMSS_NORM_RMS) ? v[i][j] * v[i][j] : v[i][j];
    }
  }
  // One number per virtual warp: the exchanges that leave NP sums in lane groups pair lanes as warp_sum does (16, 8, 4, 2, 1 apart), and
  // the eight warps' numbers meet as block_sum pairs them (4, 2, 1 apart)
  auto over_row = [&](float (&s)[NP], int slot) {
    int o = 16;
#pragma unroll
    for (int w = NP / 2; w > 0; w >>= 1, o >>= 1) {
      const bool hi = lane & o;
#pragma unroll
      for (int m = 0; m < w; ++m) s[m] = (hi ? s[m + w] : s[m]) + __shfl_xor_sync(0xffffffffu, hi ? s[m] : s[m + w], o);
    }
    float t = s[0];                     // of virtual warp part + WPR * (lane * NP / 32)
#pragma unroll
    for (; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (WPR == 1) {
#pragma unroll
      for (int b = 16; b > 2; b >>= 1) t += __shfl_xor_sync(0xffffffffu, t, b);
      return t;
    }
    if (lane % (32 / NP) == 0) red[slot][warp / WPR][part + WPR * (lane * NP / 32)] = t;
    __syncthreads();
    const float* r = red[slot][warp / WPR];
    return ((r[0] + r[4]) + (r[2] + r[6])) + ((r[1] + r[5]) + (r[3] + r[7]));
  };
  float mean = 0.f, rstd;
  if (kind == LLMSS_NORM_RMS) {
    rstd = rsqrtf(over_row(sums, 0) / (float)H + eps);
  } else {
    mean = over_row(sums, 0) / (float)H;
    float sq[NP];
#pragma unroll
    for (int m = 0; m < NP; ++m) sq[m] = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if (c0 + i * 32 * WPR >= nvec) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) { const float d = v[i][j] - mean; sq[i % NP] += d * d; }
    }
    rstd = rsqrtf(over_row(sq, 1) / (float)H + eps);
  }
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = c0 + i * 32 * WPR;
    if (c >= nvec) continue;
    float w[8], b[8], o[8];
    unpack8<T>(*reinterpret_cast<const uint4*>(weight + c * 8), w);
    if (bias != nullptr) unpack8<T>(*reinterpret_cast<const uint4*>(bias + c * 8), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float y = (v[i][j] - mean) * rstd * w[j];
      o[j] = bias != nullptr ? y + b[j] : y;
    }
    *reinterpret_cast<uint4*>(out + row * ldo + c * 8) = pack8<T>(o);
  }
}

template <typename T>
int launch_norm(const void* x, const void* x2, const void* residual_in, void* residual_out, const void* weight, const void* bias, void* out,
                int M, int H, int64_t ldx, int64_t ldx2, int64_t ldr, int64_t ldo, float eps, int kind, cudaStream_t stream) {
#define LLMSS_NORM(KERN, GRID, THREADS, ...)                                                                                              \
  LLMSS_CHECK_CUDA(launch_pdl(KERN, dim3(GRID), dim3(THREADS), 0, stream, (const T*)x, (const T*)x2, (const T*)residual_in, (T*)residual_out, \
                              (const T*)weight, (const T*)bias, (T*)out, __VA_ARGS__ H, ldx, ldx2, ldr, ldo, eps, kind))
#define LLMSS_COMMA ,
  // from four rows per SM on; fewer rows: a block each, whose loads reach more SMs
  const int wpr = H <= 2048 ? 1 : H <= 4096 ? 2 : 4;
  if (M >= 4 * 148 && H <= 8192) {
    if (wpr == 1) LLMSS_NORM((norm_rows_kernel<T, 1>), (M + 3) / 4, 128, M LLMSS_COMMA);
    else if (wpr == 2) LLMSS_NORM((norm_rows_kernel<T, 2>), (M + 1) / 2, 128, M LLMSS_COMMA);
    else LLMSS_NORM((norm_rows_kernel<T, 4>), M, 128, M LLMSS_COMMA);
    return 0;
  }
  LLMSS_NORM(norm_residual_kernel<T>, M, kThreads, );
#undef LLMSS_COMMA
#undef LLMSS_NORM
  return 0;
}

// ------------------------------------------------------------------------------------------------ 32-bit residual stream
// r = resid + mult * y (y null: r = resid) ; h = LayerNorm / RMS norm of r times weight (+ bias), stored as TO.  One CTA per row, the
// row in registers (VEC = 4: 16-byte accesses; longer rows are read back from `out_r`), two-pass variance, 32-bit throughout.
struct RnArgs {
  const float* resid; int64_t ldr;
  const float* y; int64_t ldy;
  const float* w; const float* bias;
  float* out_r; void* out_h;         // [M, W] contiguous; out_r null: r is not stored (y null)
  int W; float eps; int kind;
  float mult;                        // factor on y
};
constexpr int kRnRegs = 4;

template <int VEC> __device__ __forceinline__ void rn_load(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else v[0] = p[0];
}

template <typename TO, int VEC>
__global__ void __launch_bounds__(kThreads) residual_norm_kernel(RnArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[kThreads / 32];
  const int64_t t = blockIdx.x;
  const int W = a.W;
  constexpr int STEP = kThreads * VEC;
  float keep[kRnRegs][VEC];
  float sum = 0.f;
  const bool rms = a.kind == LLMSS_NORM_RMS;
  auto fetch = [&](int c, float (&v)[VEC]) {
    rn_load<VEC>(a.resid + t * a.ldr + c, v);
    if (a.y != nullptr) {
      float u[VEC];
      rn_load<VEC>(a.y + t * a.ldy + c, u);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] = fmaf(a.mult, u[e], v[e]);
    }
    if (a.out_r != nullptr) {
      float* o = a.out_r + t * (int64_t)W + c;
      if constexpr (VEC == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else o[0] = v[0];
    }
  };
  const float* again = a.out_r != nullptr ? a.out_r + t * (int64_t)W : a.resid + t * a.ldr;   // this thread's own columns of r
#pragma unroll
  for (int i = 0; i < kRnRegs; ++i) {
    const int c = threadIdx.x * VEC + i * STEP;
    if (c < W) {
      fetch(c, keep[i]);
#pragma unroll
      for (int e = 0; e < VEC; ++e) sum += rms ? keep[i][e] * keep[i][e] : keep[i][e];
    }
  }
  for (int c = threadIdx.x * VEC + kRnRegs * STEP; c < W; c += STEP) {
    float v[VEC];
    fetch(c, v);
#pragma unroll
    for (int e = 0; e < VEC; ++e) sum += rms ? v[e] * v[e] : v[e];
  }
  float mean = 0.f, rstd;
  if (rms) {
    rstd = rsqrtf(block_sum(sum, red) / (float)W + a.eps);
  } else {
    mean = block_sum(sum, red) / (float)W;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kRnRegs; ++i) {
      const int c = threadIdx.x * VEC + i * STEP;
      if (c < W) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) { const float d = keep[i][e] - mean; sq = fmaf(d, d, sq); }
      }
    }
    for (int c = threadIdx.x * VEC + kRnRegs * STEP; c < W; c += STEP) {
      float v[VEC];
      rn_load<VEC>(again + c, v);
#pragma unroll
      for (int e = 0; e < VEC; ++e) { const float d = v[e] - mean; sq = fmaf(d, d, sq); }
    }
    rstd = rsqrtf(block_sum(sq, red) / (float)W + a.eps);
  }
  auto emit = [&](int c, const float (&v)[VEC]) {
    float wv[VEC], bv[VEC];
    rn_load<VEC>(a.w + c, wv);
    if (a.bias != nullptr) rn_load<VEC>(a.bias + c, bv);
    TO* ho = reinterpret_cast<TO*>(a.out_h) + t * (int64_t)W + c;
    struct alignas(VEC * sizeof(TO)) Pack { TO v[VEC]; };
    Pack o;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const float h = (v[e] - mean) * rstd * wv[e];
      o.v[e] = from_f32<TO>(a.bias != nullptr ? h + bv[e] : h);
    }
    *reinterpret_cast<Pack*>(ho) = o;
  };
#pragma unroll
  for (int i = 0; i < kRnRegs; ++i) {
    const int c = threadIdx.x * VEC + i * STEP;
    if (c < W) emit(c, keep[i]);
  }
  for (int c = threadIdx.x * VEC + kRnRegs * STEP; c < W; c += STEP) {
    float v[VEC];
    rn_load<VEC>(again + c, v);
    emit(c, v);
  }
}

template <typename TO>
int residual_norm_launch(const RnArgs& a, int M, bool vec, cudaStream_t stream) {
  if (vec) LLMSS_CHECK_CUDA(launch_pdl(residual_norm_kernel<TO, 4>, dim3(M), dim3(kThreads), 0, stream, a));
  else LLMSS_CHECK_CUDA(launch_pdl(residual_norm_kernel<TO, 1>, dim3(M), dim3(kThreads), 0, stream, a));
  return 0;
}

}  // namespace

// The counterpart of llmss_norm_residual over a 32-bit residual stream: resid [M, W] (row stride ldr), y [M, W] or null, weight /
// bias 32-bit (bias may be null), out_r [M, W] contiguous (null with y null), out_h [M, W] contiguous in out_dtype.
// mult: factor on y.
LLMSS_API int llmss_residual_norm_ex(const float* resid, int64_t ldr, const float* y, int64_t ldy, float mult, const float* weight,
                                     const float* bias, float* out_r, void* out_h, int M, int W, float eps, int kind, int out_dtype,
                                     cudaStream_t stream) {
  LLMSS_REQUIRE(W > 0 && weight != nullptr && out_h != nullptr && (y == nullptr || out_r != nullptr), "residual_norm: bad arguments");
  LLMSS_REQUIRE(kind == LLMSS_NORM_LAYER || kind == LLMSS_NORM_RMS, "residual_norm: norm kind %d", kind);
  if (M <= 0) return 0;
  RnArgs a{resid, ldr, y, ldy, weight, bias, out_r, out_h, W, eps, kind, mult};
  const bool vec = W % 4 == 0 && ldr % 4 == 0 && ldy % 4 == 0 &&
                   ((((uintptr_t)resid) | ((uintptr_t)y) | ((uintptr_t)weight) | ((uintptr_t)bias) | ((uintptr_t)out_r) | ((uintptr_t)out_h)) & 15) == 0;
  LLMSS_BY_DTYPE(out_dtype, return (residual_norm_launch<T>(a, M, vec, stream)));
}

LLMSS_API int llmss_residual_norm(const float* resid, int64_t ldr, const float* y, int64_t ldy, const float* weight, const float* bias,
                                  float* out_r, void* out_h, int M, int W, float eps, int kind, int out_dtype, cudaStream_t stream) {
  return llmss_residual_norm_ex(resid, ldr, y, ldy, 1.f, weight, bias, out_r, out_h, M, W, eps, kind, out_dtype, stream);
}

LLMSS_API int llmss_norm_residual(const void* x, const void* x2, const void* residual_in, void* residual_out,
                                  const void* weight, const void* bias, void* out, int M, int H, int64_t ldx,
                                  int64_t ldx2, int64_t ldr, int64_t ldo, float eps, int kind, int dtype,
                                  cudaStream_t stream) {
  LLMSS_REQUIRE(H % 8 == 0 && H <= kThreads * kMaxVec * 8, "norm_residual: H=%d must be a multiple of 8 and <= %d", H,
                kThreads * kMaxVec * 8);
  LLMSS_REQUIRE(dtype == LLMSS_F16 || dtype == LLMSS_BF16, "norm_residual: dtype must be f16/bf16");
  LLMSS_REQUIRE(ldx % 8 == 0 && ldo % 8 == 0 && ldr % 8 == 0 && ldx2 % 8 == 0, "norm_residual: row strides must be multiples of 8");
  if (M == 0) return 0;
  if (dtype == LLMSS_F16) {
    if (int e = launch_norm<__half>(x, x2, residual_in, residual_out, weight, bias, out, M, H, ldx, ldx2, ldr, ldo, eps, kind, stream)) return e;
  } else {
    if (int e = launch_norm<__nv_bfloat16>(x, x2, residual_in, residual_out, weight, bias, out, M, H, ldx, ldx2, ldr, ldo, eps, kind, stream)) return e;
  }
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}
