// Gated delta rule over a packed batch (same batch convention as recurrent.cu: cu_q / seq_lens / state slots).
//
//   per head and token:  S <- g_t S ;  u = beta_t (v_t - S^T k_t) ;  S <- S + k_t u^T ;  o_t = S^T q_t
//
// Every value column of the state is a recurrence of its own (S^T k, the write and the read-out only couple the rows of one
// column), so a thread keeps KPT rows of two columns in registers and the R threads of a column pair meet in warp-shuffle sums.
// One block = one (sequence, head, slice of value columns); the block that reads a slot's old state is the block that writes its new
// one.  Tokens are staged 16 at a time through shared memory: q and k in strips of KPT + 4 floats (the strips a warp reads together
// lie in different banks, every read a 16-byte one; strips beyond dk hold zeros), copied asynchronously one stage ahead; the numbers
// per token (decay, write strength, the norms 1 / sqrt(sum x^2 + eps), k . q) lie beside them.  The state lies in memory
// column-major per head ([dv][dk]).
//
// Long portions go over chunks of 32 tokens on the tensor cores where that is faster (delta_chunk.cu); this file's portions are the others, and what a
// launch over chunks leaves of a sequence.
//
// A batch of single tokens (decode) runs the row-split form instead (delta_step_kernel): one warp per value column, lanes over
// the key rows, so that every state access is one contiguous column (512 bytes at dk = 128) -- a decode step is bound by
// reading and writing the states once.
// Everything here is 32-bit with full-precision exponentials (over chunks: products of 16-bit parts, see delta_chunk.cu on rounding).
#include "common.cuh"
#include "delta.cuh"

namespace {

constexpr int DTCH = 16;
constexpr int kChunkLeast = 32;        // shorter sequences of a batch that goes over chunks stay here: a block over chunks takes 9 us to start and end

__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two 32-bit numbers per instruction: half the issue slots of the same arithmetic (148 SMs, 8 warps each: 126 against 116 multiply-adds
// per clock and SM when nothing else is issued, and the slots left over take the shared-memory loads).
using namespace packed;
__device__ __forceinline__ float sum_of_pair(uint64_t v) {
  const float2 x = unpack(v);
  return x.x + x.y;
}

// Portions.  Per token a thread makes two dot products with its rows of the OLD state (S^T k and S^T q) and then writes; the
// read-out is decay * S^T q + u * (k . q), so only S^T k stands in the chain from token to token, and the norms of q and k and k . q
// are numbers per token that the staging computes (8 lanes a token), never rescaled rows.
// The 32-bit pipe wants 4 operations per state element and token.  Shared memory delivers 128 bytes a clock to an SM's registers
// whether the lanes read one address or 32, so rows that feed one column (64 rows x 1 column: 48 16-byte reads per thread and token in
// the form before this one) bound the kernel; 32 rows x 2 columns read a third of that.  16 rows x 4 columns read less still and lost
// it to shuffles and selects.  16 heads of 128 x 128 on B200: 8 prompts of 1024 tokens 764 -> 666 us, of 576 .. 1472 1083 -> 934,
// one of 1500 1100 -> 633; 32 heads of 64 x 64: 713 -> 407, 1007 -> 572, 1017 -> 578.  A lone block now waits on its own chain
// (about 800 clocks a token), a full SM on issue.  Blocks of 64 threads (32 columns at key size 128): a sequence's chain is as long as its portion, and with
// small blocks every SM holds several sequences at once.
// Stages of 16 tokens are double-buffered: the asynchronous copies of stage s + 1 (global -> shared, no registers) run behind the
// arithmetic of stage s, so the dependent chain of a long portion never waits for memory.
template <int KPT, int R>
__global__ void __launch_bounds__(256) delta_scan_kernel(DeltaArgs a) {
  constexpr int STRIP = KPT + 4, row = R * STRIP, COLS = 2;
  extern __shared__ __align__(16) float sm[];
  const int b = blockIdx.x;
  int q0 = a.cu_q[b], ql = a.cu_q[b + 1] - q0, ctx = a.seq_lens[b] - ql;
  const int slot = a.slots[b], h = blockIdx.y, hk = h / a.rep, j0 = blockIdx.z * a.dvt, nj = min(a.dvt, a.dv - j0);
  if (slot < 0 || ctx < 0 || ql <= 0) return;
  if (a.prepared != nullptr && ql >= a.least) {          // what the launch over chunks has left of this sequence (a slice lies in one of its blocks)
    const uint8_t* first = a.prepared + ((int64_t)(q0 / kDeltaChunk + b) * a.H + h) * LLMSS_DELTA_PREPARED;
    const int done = reinterpret_cast<const int*>(first + kDeltaDoneAt)[j0 / kDeltaCols];
    if (done >= ql) return;
    q0 += done;
    ql -= done;
    ctx += done;
  }
  const int dk = a.dk, nthr = blockDim.x;
  const int r = threadIdx.x % R, c0 = threadIdx.x / R * COLS;          // key strip, first column (inside the slice)
  const int i0 = r * KPT;
  const int stage_floats = 2 * DTCH * row + DTCH * a.dvt + 8 * DTCH;     // q, k [DTCH][row]; v [DTCH][dvt]; eight numbers per token
  uint64_t S[COLS][KPT / 2];
  float* sp = a.state + (((int64_t)slot * a.H + h) * a.dv + j0 + c0) * dk;      // column c0 + c at sp + c * dk
  const bool vec = (dk & 3) == 0;        // every column of the state starts on a 16-byte boundary
#pragma unroll
  for (int c = 0; c < COLS; ++c)
#pragma unroll
    for (int ii = 0; ii < KPT; ii += 4) {
      float4 t4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c0 + c < nj && ctx > 0) {
        const float* p = sp + (int64_t)c * dk;
        if (vec && i0 + ii + 4 <= dk) t4 = *reinterpret_cast<const float4*>(p + i0 + ii);
        else {
          if (i0 + ii < dk) t4.x = p[i0 + ii];
          if (i0 + ii + 1 < dk) t4.y = p[i0 + ii + 1];
          if (i0 + ii + 2 < dk) t4.z = p[i0 + ii + 2];
          if (i0 + ii + 3 < dk) t4.w = p[i0 + ii + 3];
        }
      }
      S[c][ii / 2] = pack(t4.x, t4.y);
      S[c][ii / 2 + 1] = pack(t4.z, t4.w);
    }
  // the strips' padding (beyond dk, and between strips) is read by the arithmetic and never copied into: zero it once
  for (int idx = threadIdx.x; idx < 2 * stage_floats; idx += nthr) sm[idx] = 0.f;
  __syncthreads();
  auto issue = [&](int t0, float* B) {
    const int nt = min(DTCH, ql - t0);
    float* qs = B;
    float* ks = B + DTCH * row;
    float* vs = ks + DTCH * row;
    float* gs = vs + DTCH * a.dvt + 6 * DTCH;
    if (a.vec16) {
      const int n4 = dk >> 2;
      for (int idx = threadIdx.x; idx < nt * n4; idx += nthr) {
        const int tt = idx / n4, c = (idx - tt * n4) << 2;
        const int dst = tt * row + (c / KPT) * STRIP + c % KPT;
        const int64_t t = q0 + t0 + tt;
        cp_async_16(qs + dst, a.q + t * a.ldq + (int64_t)hk * dk + c);
        cp_async_16(ks + dst, a.k + t * a.ldk + (int64_t)hk * dk + c);
      }
      const int v4 = nj >> 2;       // vec16: dv and the slice width are multiples of 4
      for (int idx = threadIdx.x; idx < nt * v4; idx += nthr) {
        const int tt = idx / v4, c = (idx - tt * v4) << 2;
        cp_async_16(vs + tt * a.dvt + c, a.v + (int64_t)(q0 + t0 + tt) * a.ldv + (int64_t)h * a.dv + j0 + c);
      }
    } else {
      for (int idx = threadIdx.x; idx < nt * dk; idx += nthr) {
        const int tt = idx / dk, c = idx - tt * dk;
        const int dst = tt * row + (c / KPT) * STRIP + c % KPT;
        const int64_t t = q0 + t0 + tt;
        cp_async_4(qs + dst, a.q + t * a.ldq + (int64_t)hk * dk + c);
        cp_async_4(ks + dst, a.k + t * a.ldk + (int64_t)hk * dk + c);
      }
      for (int idx = threadIdx.x; idx < nt * nj; idx += nthr) {
        const int tt = idx / nj, c = idx - tt * nj;
        cp_async_4(vs + tt * a.dvt + c, a.v + (int64_t)(q0 + t0 + tt) * a.ldv + (int64_t)h * a.dv + j0 + c);
      }
    }
    if (threadIdx.x < nt) {
      const int64_t t = q0 + t0 + threadIdx.x;
      cp_async_4(gs + threadIdx.x, a.log_decay + t * a.ldg + h);
      cp_async_4(gs + DTCH + threadIdx.x, a.beta + t * a.ldb + h);
    }
    cp_async_commit();
  };
  issue(0, sm);
  const int64_t ldo = (int64_t)a.H * a.dv;
  float* op = a.out + q0 * ldo + (int64_t)h * a.dv + j0 + c0;
  int cur = 0;
  for (int t0 = 0; t0 < ql; t0 += DTCH, cur ^= 1) {
    const int nt = min(DTCH, ql - t0);
    float* qs = sm + cur * stage_floats;
    float* ks = qs + DTCH * row;
    float* vs = ks + DTCH * row;
    float4* f4 = reinterpret_cast<float4*>(vs + DTCH * a.dvt);      // [DTCH] strength; strength * decay / |k|; 1 / |k|; decay
    float2* f2 = reinterpret_cast<float2*>(f4 + DTCH);              // [DTCH] decay * q_scale / |q|; k . q of the scaled vectors
    const float* raw = reinterpret_cast<const float*>(f2 + DTCH);   // [2][DTCH] log decays, write strengths as given
    if (t0 + DTCH < ql) {
      issue(t0 + DTCH, sm + (cur ^ 1) * stage_floats);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    // (whole warps: the shuffles name all lanes; padding and rows past nt are zeros or older numbers that nobody reads)
    for (int t8 = threadIdx.x >> 3; t8 < DTCH; t8 += nthr >> 3) {
      const int l8 = threadIdx.x & 7;
      float sq = 0.f, sk = 0.f, skq = 0.f;
#pragma unroll
      for (int w = 0; w < row; w += 32) {
        if (w + l8 * 4 >= row) break;
        const float4 x = *reinterpret_cast<const float4*>(qs + t8 * row + w + l8 * 4), y = *reinterpret_cast<const float4*>(ks + t8 * row + w + l8 * 4);
        sq = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, sq))));
        sk = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, sk))));
        skq = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, skq))));
      }
      __syncwarp();
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
        skq += __shfl_xor_sync(0xffffffffu, skq, o);
      }
      if (l8 == 0 && t8 < nt) {
        const float fq = (a.unit ? rsqrtf(sq + a.unit_eps) : 1.f) * a.q_scale, fk = a.unit ? rsqrtf(sk + a.unit_eps) : 1.f;
        const float g = expf(raw[t8]), x = raw[DTCH + t8], be = a.beta_sigmoid ? 1.f / (1.f + expf(-x)) : x;
        f4[t8] = make_float4(be, be * g * fk, fk, g);
        f2[t8] = make_float2(g * fq, skq * fk * fq);
      }
    }
    __syncthreads();
    const float* kr = ks + r * STRIP;
    const float* qr = qs + r * STRIP;
    const float* vr = vs + c0;
#pragma unroll 2
    for (int tt = 0; tt < nt; ++tt, kr += row, qr += row, vr += a.dvt, op += ldo) {
      const float4 f = f4[tt];
      const float2 fo = f2[tt], v2 = *reinterpret_cast<const float2*>(vr);
      uint64_t kk[KPT / 2], d0, d1, e0, e1;
#pragma unroll
      for (int ii = 0; ii < KPT / 4; ++ii) {
        const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(kr + 4 * ii), q4 = *reinterpret_cast<const ulonglong2*>(qr + 4 * ii);
        kk[2 * ii] = k4.x;
        kk[2 * ii + 1] = k4.y;
        if (ii == 0) {
          d0 = pmul(S[0][0], k4.x); d1 = pmul(S[1][0], k4.x);
          e0 = pmul(S[0][0], q4.x); e1 = pmul(S[1][0], q4.x);
        } else {
          d0 = pfma(S[0][2 * ii], k4.x, d0); d1 = pfma(S[1][2 * ii], k4.x, d1);
          e0 = pfma(S[0][2 * ii], q4.x, e0); e1 = pfma(S[1][2 * ii], q4.x, e1);
        }
        d0 = pfma(S[0][2 * ii + 1], k4.y, d0); d1 = pfma(S[1][2 * ii + 1], k4.y, d1);
        e0 = pfma(S[0][2 * ii + 1], q4.y, e0); e1 = pfma(S[1][2 * ii + 1], q4.y, e1);
      }
      float x0 = sum_of_pair(d0), x1 = sum_of_pair(d1);
#pragma unroll
      for (int o = R >> 1; o > 0; o >>= 1) {
        x0 += __shfl_xor_sync(0xffffffffu, x0, o);
        x1 += __shfl_xor_sync(0xffffffffu, x1, o);
      }
      const float u0 = fmaf(f.x, v2.x, -f.y * x0), u1 = fmaf(f.x, v2.y, -f.y * x1);
      const float w0 = u0 * f.z, w1 = u1 * f.z;
      const uint64_t g2 = pack(f.w, f.w), p0 = pack(w0, w0), p1 = pack(w1, w1);
#pragma unroll
      for (int ii = 0; ii < KPT / 2; ++ii) {
        S[0][ii] = pfma(g2, S[0][ii], pmul(kk[ii], p0));
        S[1][ii] = pfma(g2, S[1][ii], pmul(kk[ii], p1));
      }
      // S^T q of the old state: the first exchange leaves one column per lane
      const float y0 = sum_of_pair(e0), y1 = sum_of_pair(e1);
      if (R > 1) {
        const bool hi = r & (R >> 1);
        float y = (hi ? y1 : y0) + __shfl_xor_sync(0xffffffffu, hi ? y0 : y1, R >> 1);
#pragma unroll
        for (int o = R >> 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if ((r & ((R >> 1) - 1)) == 0 && c0 + hi < nj) op[hi] = fmaf(fo.x, y, (hi ? u1 : u0) * fo.y);
      } else {
        if (c0 < nj) op[0] = fmaf(fo.x, y0, u0 * fo.y);
        if (c0 + 1 < nj) op[1] = fmaf(fo.x, y1, u1 * fo.y);
      }
    }
    __syncthreads();      // this buffer is copied into again at the start of the next round
  }
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    if (c0 + c >= nj) continue;
    float* p = sp + (int64_t)c * dk;
#pragma unroll
    for (int ii = 0; ii < KPT; ii += 4) {
      float4 t4;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(t4.x), "=f"(t4.y) : "l"(S[c][ii / 2]));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(t4.z), "=f"(t4.w) : "l"(S[c][ii / 2 + 1]));
      if (vec && i0 + ii + 4 <= dk) *reinterpret_cast<float4*>(p + i0 + ii) = t4;
      else {
        if (i0 + ii < dk) p[i0 + ii] = t4.x;
        if (i0 + ii + 1 < dk) p[i0 + ii + 1] = t4.y;
        if (i0 + ii + 2 < dk) p[i0 + ii + 2] = t4.z;
        if (i0 + ii + 3 < dk) p[i0 + ii + 3] = t4.w;
      }
    }
  }
}

// Single tokens: grid (B, H, column groups), 8 warps per block; warp w takes columns j0 + w, j0 + w + 8, ... four at a time.
// Lane l holds rows l, l + 32, ... (KL of them) of q, k and of the column in flight.
constexpr int STEP_WARPS = 8, STEP_COLS = 4;
template <int KL>
__global__ void __launch_bounds__(STEP_WARPS * 32) delta_step_kernel(DeltaArgs a, int cols_per_block) {
  const int b = blockIdx.x;
  const int q0 = a.cu_q[b], ql = a.cu_q[b + 1] - q0, ctx = a.seq_lens[b] - ql, slot = a.slots[b];
  if (slot < 0 || ctx < 0 || ql != 1) return;
  const int h = blockIdx.y, hk = h / a.rep, dk = a.dk, dv = a.dv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t = q0;
  float qv[KL], kv[KL];
  float sq = 0.f, sk = 0.f;
#pragma unroll
  for (int m = 0; m < KL; ++m) {
    const int i = lane + 32 * m;
    qv[m] = i < dk ? a.q[t * a.ldq + (int64_t)hk * dk + i] : 0.f;
    kv[m] = i < dk ? a.k[t * a.ldk + (int64_t)hk * dk + i] : 0.f;
    sq = fmaf(qv[m], qv[m], sq);
    sk = fmaf(kv[m], kv[m], sk);
  }
  if (a.unit || a.q_scale != 1.f) {
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float rq = (a.unit ? rsqrtf(sq + a.unit_eps) : 1.f) * a.q_scale, rk = a.unit ? rsqrtf(sk + a.unit_eps) : 1.f;
#pragma unroll
    for (int m = 0; m < KL; ++m) { qv[m] *= rq; kv[m] *= rk; }
  }
  const float g = expf(a.log_decay[t * a.ldg + h]);
  const float braw = a.beta[t * a.ldb + h];
  const float be = a.beta_sigmoid ? 1.f / (1.f + expf(-braw)) : braw;
  float* sp = a.state + ((int64_t)slot * a.H + h) * dv * dk;
  const float* vp = a.v + t * a.ldv + (int64_t)h * dv;
  float* op = a.out + t * a.H * dv + (int64_t)h * dv;
  const int j0 = blockIdx.z * cols_per_block, j1 = min(dv, j0 + cols_per_block);
  for (int jb = j0 + warp; jb < j1; jb += STEP_WARPS * STEP_COLS) {
    float S[STEP_COLS][KL], d[STEP_COLS], e[STEP_COLS];
#pragma unroll
    for (int c = 0; c < STEP_COLS; ++c) {
      const int j = jb + c * STEP_WARPS;
      d[c] = 0.f;
#pragma unroll
      for (int m = 0; m < KL; ++m) {
        const int i = lane + 32 * m;
        S[c][m] = (j < j1 && ctx > 0 && i < dk) ? sp[(int64_t)j * dk + i] : 0.f;
        d[c] = fmaf(S[c][m], kv[m], d[c]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < STEP_COLS; ++c) d[c] += __shfl_xor_sync(0xffffffffu, d[c], o);
#pragma unroll
    for (int c = 0; c < STEP_COLS; ++c) {
      const int j = jb + c * STEP_WARPS;
      const float u = be * ((j < j1 ? vp[j] : 0.f) - g * d[c]);
      e[c] = 0.f;
#pragma unroll
      for (int m = 0; m < KL; ++m) {
        S[c][m] = fmaf(g, S[c][m], kv[m] * u);
        e[c] = fmaf(S[c][m], qv[m], e[c]);
        const int i = lane + 32 * m;
        if (j < j1 && i < dk) sp[(int64_t)j * dk + i] = S[c][m];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < STEP_COLS; ++c) e[c] += __shfl_xor_sync(0xffffffffu, e[c], o);
#pragma unroll
    for (int c = 0; c < STEP_COLS; ++c) {
      const int j = jb + c * STEP_WARPS;
      if (lane == 0 && j < j1) op[j] = e[c];
    }
  }
}

}  // namespace

namespace {

bool delta_args(DeltaArgs& a, const float* q, int64_t ldq, const float* k, int64_t ldk, const float* v, int64_t ldv, const float* log_decay,
                int64_t ldg, const float* beta, int64_t ldb, float* out, float* state, const int* cu_q, const int* seq_lens, const int* slots,
                int heads, int qk_heads, int dk, int dv, float unit_eps, float q_scale, int beta_sigmoid) {
  if (heads <= 0 || qk_heads <= 0 || heads % qk_heads != 0 || dk <= 0 || dk > 1024 || dv <= 0) return false;
  memset(&a, 0, sizeof(a));
  a.q = q; a.ldq = ldq; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv; a.log_decay = log_decay; a.ldg = ldg; a.beta = beta; a.ldb = ldb;
  a.out = out; a.state = state; a.cu_q = cu_q; a.seq_lens = seq_lens; a.slots = slots;
  a.H = heads; a.rep = heads / qk_heads; a.dk = dk; a.dv = dv;
  a.unit = unit_eps >= 0.f ? 1 : 0; a.unit_eps = unit_eps >= 0.f ? unit_eps : 0.f; a.q_scale = q_scale; a.beta_sigmoid = beta_sigmoid;
  return true;
}

// token by token: all sequences, or what a launch over chunks has left of them
int delta_portions(DeltaArgs a, int B, cudaStream_t stream) {
  const int dk = a.dk, dv = a.dv;
  // up to 32 key rows per thread, R lanes (a power of two) to a column pair
  const int kpt = dk <= 8 ? 8 : (dk <= 16 ? 16 : 32);
  int R = 1;
  while (R * kpt < dk) R *= 2;
  int threads = (((dv + 1) / 2 * R + 31) / 32) * 32;
  const int most = R <= 4 ? 64 : 256;       // long keys: a stage of q and k is shared by more columns
  threads = threads > most ? most : threads;
  a.dvt = threads / R * 2;                  // (key sizes up to 128: 16 to 128, so that a slice lies within 128 columns)
  const dim3 grid(B, a.H, (dv + a.dvt - 1) / a.dvt);
  LLMSS_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "delta_scan: grid too large");
  a.vec16 = (dk % 4 == 0 && dv % 4 == 0 && a.dvt % 4 == 0 && a.ldq % 4 == 0 && a.ldk % 4 == 0 && a.ldv % 4 == 0 &&
             (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v) & 15) == 0) ? 1 : 0;
  const size_t smem = 2 * sizeof(float) * ((size_t)2 * DTCH * R * (kpt + 4) + (size_t)DTCH * a.dvt + 8 * DTCH);
#define LLMSS_DS(K, RR)                                                                     \
  do {                                                                                      \
    static PerDeviceSmem gsm;                                                               \
    if (smem > 48 * 1024) LLMSS_CHECK_CUDA(gsm.ensure(delta_scan_kernel<K, RR>, (int)smem)); \
    delta_scan_kernel<K, RR><<<grid, threads, smem, stream>>>(a);                           \
  } while (0)
  if (kpt == 8) LLMSS_DS(8, 1);
  else if (kpt == 16) LLMSS_DS(16, 1);
  else if (R == 1) LLMSS_DS(32, 1);
  else if (R == 2) LLMSS_DS(32, 2);
  else if (R == 4) LLMSS_DS(32, 4);
  else if (R == 8) LLMSS_DS(32, 8);
  else if (R == 16) LLMSS_DS(32, 16);
  else LLMSS_DS(32, 32);
#undef LLMSS_DS
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace

// q, k [T, qk_heads * dk] (value head h reads q / k head h / (heads / qk_heads)); v [T, heads * dv]; log_decay, beta [T, heads];
// out [T, heads * dv]; state [slots, heads, dv, dk].  unit_eps >= 0: q and k become x / sqrt(sum x^2 + unit_eps) per head first.
LLMSS_API int llmss_delta_scan(const float* q, int64_t ldq, const float* k, int64_t ldk, const float* v, int64_t ldv,
                               const float* log_decay, int64_t ldg, const float* beta, int64_t ldb, float* out, float* state,
                               const int* cu_q, const int* seq_lens, const int* slots, int B, int max_q, int heads, int qk_heads, int dk,
                               int dv, float unit_eps, float q_scale, int beta_sigmoid, cudaStream_t stream) {
  LLMSS_REQUIRE(heads > 0 && qk_heads > 0 && heads % qk_heads == 0, "delta_scan: %d value heads over %d query/key heads", heads, qk_heads);
  LLMSS_REQUIRE(dk > 0 && dk <= 1024 && dv > 0, "delta_scan: key size %d (at most 1024), value size %d", dk, dv);
  if (B <= 0) return 0;
  DeltaArgs a;
  delta_args(a, q, ldq, k, ldk, v, ldv, log_decay, ldg, beta, ldb, out, state, cu_q, seq_lens, slots, heads, qk_heads, dk, dv, unit_eps, q_scale, beta_sigmoid);
  if (max_q <= 1 && dk <= 256) {
    // every sequence brings one token: one warp per value column, lanes over the key rows
    a.dvt = 0;
    const int per_pass = STEP_WARPS * STEP_COLS;
    int groups = 1;
    while ((int64_t)B * heads * groups < 1024 && groups * per_pass < dv) groups *= 2;
    int cols = (dv + groups - 1) / groups;
    cols = ((cols + per_pass - 1) / per_pass) * per_pass;
    const dim3 sgrid(B, heads, (dv + cols - 1) / cols);
    LLMSS_REQUIRE(sgrid.y <= 65535 && sgrid.z <= 65535, "delta_scan: grid too large");
    const int kl = (dk + 31) / 32;
    if (kl <= 1) delta_step_kernel<1><<<sgrid, STEP_WARPS * 32, 0, stream>>>(a, cols);
    else if (kl <= 2) delta_step_kernel<2><<<sgrid, STEP_WARPS * 32, 0, stream>>>(a, cols);
    else if (kl <= 4) delta_step_kernel<4><<<sgrid, STEP_WARPS * 32, 0, stream>>>(a, cols);
    else delta_step_kernel<8><<<sgrid, STEP_WARPS * 32, 0, stream>>>(a, cols);
    LLMSS_CHECK_CUDA(cudaGetLastError());
    return 0;
  }
  return delta_portions(a, B, stream);
}

// Sequences of at least 32 tokens over chunks (delta_chunk.cu), shorter ones beside them token by token.  T: rows of the batch; scratch:
// llmss_delta_scan_chunked_bytes bytes.  Key sizes up to 128 that are multiples of 4; q, k (rows too), state and scratch on 16-byte lines.
LLMSS_API int64_t llmss_delta_scan_chunked_bytes(int T, int B, int heads) { return ((int64_t)T / 32 + B) * heads * LLMSS_DELTA_PREPARED; }
LLMSS_API int llmss_delta_scan_chunked(const float* q, int64_t ldq, const float* k, int64_t ldk, const float* v, int64_t ldv,
                               const float* log_decay, int64_t ldg, const float* beta, int64_t ldb, float* out, float* state,
                               const int* cu_q, const int* seq_lens, const int* slots, int B, int max_q, int heads, int qk_heads, int dk,
                               int dv, float unit_eps, float q_scale, int beta_sigmoid, void* scratch, cudaStream_t stream) {
  DeltaArgs a;
  LLMSS_REQUIRE(delta_args(a, q, ldq, k, ldk, v, ldv, log_decay, ldg, beta, ldb, out, state, cu_q, seq_lens, slots, heads, qk_heads, dk, dv, unit_eps, q_scale, beta_sigmoid),
                "delta_scan_chunked: %d value heads over %d query/key heads, sizes %d, %d", heads, qk_heads, dk, dv);
  LLMSS_REQUIRE(dk <= 128 && dk % 4 == 0 && ldq % 4 == 0 && ldk % 4 == 0 &&
                    (((uintptr_t)q | (uintptr_t)k | (uintptr_t)state | (uintptr_t)scratch) & 15) == 0,
                "delta_scan_chunked: key size %d (at most 128, a multiple of 4), rows of q and k on 16-byte lines", dk);
  LLMSS_REQUIRE(B <= 65535 && heads <= 65535 && (dv + 127) / 128 <= 65535, "delta_scan_chunked: grid too large");
  if (B <= 0) return 0;
  // (lengths lie on the device: the token-by-token launch always follows, also behind a single sequence)
  if (max_q >= kChunkLeast && dv <= kDeltaDone * kDeltaCols) {
    a.prepared = static_cast<uint8_t*>(scratch);
    a.least = kChunkLeast;
    const int rc = delta_chunk_launch(a, B, max_q, stream);
    if (rc != 0) return rc;
  }
  return delta_portions(a, B, stream);
}
