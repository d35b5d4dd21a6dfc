// Long portions of the gated linear recurrence (csrc/recurrent.cu: linear_scan) as products over chunks of 64 tokens.
//
//   S_t = diag(a_t) S_(t-1) + k_t (c_t v_t)^T ;  o_t = S_t^T q_t   or, read before the update,  (S_(t-1) + diag(u) k_t (c_t v_t)^T)^T q_t
//
// Token by token a state element costs three operations and a share of a reduction, twice over (the two passes of the token-serial
// form).  Over a chunk the same sums are products of tiles that live in shared memory, two multiply-adds per state element and token:
//   1. scan_state_kernel   U_c = sum_j (prod_(t > j) a_t * k_j) v_j^T and the chunk's decay D_c, every chunk a block;
//   2. scan_carry_kernel   S_(c+1) = D_c S_c + U_c along a sequence's chunks, an element per thread; U_c is replaced by S_c;
//   3. scan_out_kernel     o = (decayed q) S_c + tril((decayed q) (decayed k)^T) v, every chunk a block.
// Operands, states and results are 32-bit numbers.  Products over channels and over a chunk's keys run on the multiply-add pipe, two numbers
// per instruction where both operands lie in memory order (a 3-term split on the tensor cores would run at 158 against 126 multiply-adds per
// clock and SM); scores x values sum in 64 bits on its tensor form (62 multiply-adds per clock and SM).
//
// Decays without overflow or underflow: a sub-block of 16 tokens takes its middle as reference, q_i gets F(i) and k_j gets 1 / F(j) with
// F the decay from the middle (products of at most 8 factors, one division).  Between sub-blocks no factor is formed that could be below
// what it cancels: the query is first multiplied by its sub-block's first half (what 1 / F may have put in, which leaves the decay from
// the sub-block's start), the key by its sub-block's second half (the decay to its end), and only then the whole sub-blocks that lie
// between.  One factor from middle to middle would be a product of two halves, zero in 32 bits for decays of e^-6 per token, where the pair
// of tokens at the border has weight 1.  Half a sub-block may decay to 2^-80 or grow to 2^15 in any channel: scaled numbers then stay
// normal for q and k down to 2^-46.  A chunk runs token by token (a column per thread) where a half does more, where a scaled number
// leaves the range, or where a value is not finite (the masked half of scores x values is zeros times values: a bad one would reach
// the tokens before it).  Kernel 1 needs no reciprocals: its factors are suffix products.
//
// Rounding.  Two sums stand behind an output (scores, then outputs) where the token-serial form has one, and a chain of products behind a
// decay.  So that the result is not further from 64 bits than token by token:
//   - decays that are one number per token or head are multiplied out in 64 bits, once per chunk (with a constant decay every rounding has
//     the same sign); a key's decay to the chunk's end, per channel, is carried as a pair of numbers;
//   - a score is the sum of parts of 8 channels with the roundings of the additions carried along;
//   - scores x values, the chain of up to 64 additions to a result of full size, sum in 64 bits and are rounded once.
// Against 64 bits, of the norm (token by token in brackets): 64 x 64 with a bonus 9.0e-8 (9.4e-8), 128 x 128 per channel 4.7e-8 (5.0e-8),
// one decay per head 1.3e-7 (1.7e-7), 128 x 64 per token 8.2e-8 (9.8e-8); decays near 1 per channel 2.3e-7 (2.4e-7).  With 32-bit sums
// throughout the first two were 1.0e-7 and 6.9e-8.
//
// B200, 8 prompts of 1024 tokens, against the two passes of the token-serial form: 32 heads of 64 x 64, decay per channel and bonus
// 585 -> 415 us (101 + 37 + 287 under ncu, where the issue slots are half full and shared memory's path 39 %; with 32-bit sums throughout 385);
// 16 heads of 128 x 128, per channel 954 -> 728 us, constant decay 821 -> 630 us; 32 heads of 128 x 64, decay per token 810 -> 620 us.
// Kernel 3 is bound by its phases between barriers, at two or three blocks per SM.  With every chunk token by token: 696, 1522, 1231, 1222 us.
#include "common.cuh"

namespace {

constexpr int C = 64, SB = 16, NS = C / SB, JT = 64;     // chunk, sub-block, value columns per block
constexpr float kLow = 0x1p-80f, kHigh = 0x1p15f;        // decay or growth of half a sub-block that the products take
constexpr float kBig = 0x1p120f;                         // scaled numbers or values above this (or no numbers): token by token

struct ChunkArgs {
  const float* q; int64_t ldq;
  const float* k; int64_t ldk;
  const float* v; int64_t ldv;
  const float* decay; int64_t ldd;     // kind 0: [H] decays; 1: [T, H] log decays; 2: [T, H * dk] log decays
  const float* bonus;                  // [H, dk] or null
  const float* vscale; int64_t ldvs;   // [T, H] or null
  float* out;                          // [T, H * dv]
  float* state;                        // [slots, H, dv, dk]
  const int* cu_q; const int* seq_lens; const int* slots;
  float* chunks;                       // [chunk slots][H][dv][dk]: U_c, then S_c
  float* decays;                       // [chunk slots][H][dk]
  float* decay_rest;                   // [chunk slots][H]: what rounding D_c to 32 bits left (kinds 0 and 1)
  int H, rep, dk, dv, nslices;
  int least;                           // sequences of fewer tokens are left alone
};

// rows and chunk slots of sequence b; the slots of all sequences take T / 64 + B places: cu_q[b] / 64 + b is the first of b's
struct Rows {
  int q0, ql, ctx, slot, first;
};
__device__ __forceinline__ Rows rows_of(const ChunkArgs& a, int b) {
  Rows r;
  r.q0 = a.cu_q[b];
  r.ql = a.cu_q[b + 1] - r.q0;
  r.ctx = a.seq_lens[b] - r.ql;
  r.slot = a.slots[b];
  r.first = r.q0 / C + b;
  if (r.slot < 0 || r.ctx < 0 || r.ql < a.least) r.ql = 0;
  return r;
}

using namespace packed;
__device__ __forceinline__ ulonglong2 lds2(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// Loads never stand behind a branch: rows past the chunk's end and channels past dk are read from the last valid place and replaced
// by a select, so that a thread's loads are all in flight together (behind branches, or moved behind one by the compiler, the same
// loads were two thirds of the time; hence the volatile load).
__device__ __forceinline__ float ld_f32(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
// SB rows of one column, from local row l0 of n; p: the column in the chunk's row 0
__device__ __forceinline__ void load_rows(const float* p, int64_t ld, int l0, int n, float (&x)[SB]) {
  const int first = min(l0, n - 1);
  p += first * ld;
#pragma unroll
  for (int i = 0; i < SB; ++i) {
    x[i] = ld_f32(p);
    p += l0 + i + 1 < n ? ld : 0;
  }
}
// c[8 x 8] += a[8 x 4] b[4 x 8] in 64 bits: lane l holds a(l / 4, l % 4), b(l % 4, l / 4) and c(l / 4, 2 (l % 4) + {0, 1})
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
// 1 / x by one Newton-Raphson step on the approximate reciprocal; x lies in 2^-80 .. 2^15 wherever the result is used
__device__ __forceinline__ float recip(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return fmaf(y, fmaf(-x, y, 1.f), y);
}
// decay factors of SB tokens of a channel (1 where `in` is false or past n)
__device__ __forceinline__ void load_factors(const float* p, int64_t ld, int l0, int n, bool in, float (&x)[SB]) {
  load_rows(p, ld, l0, n, x);
#pragma unroll
  for (int i = 0; i < SB; ++i) {
    const float f = expf(x[i]);
    x[i] = in && l0 + i < n ? f : 1.f;
  }
}
// ROWS tokens of the chunk's value columns from local row l0, NT threads: element i of a thread is (its index + i NT) of [ROWS][JT]
template <int NT, int ROWS>
__device__ __forceinline__ void load_values(const ChunkArgs& a, int64_t t0, int l0, int n, int h, int j0, int nj, float (&x)[ROWS * JT / NT]) {
  const int j = threadIdx.x % JT, t1 = l0 + threadIdx.x / JT;
  constexpr int STEP = NT / JT, E = ROWS * JT / NT;
  const float* p = a.v + t0 * a.ldv + (int64_t)h * a.dv + j0 + min(j, nj - 1);
#pragma unroll
  for (int i = 0; i < E; ++i) x[i] = ld_f32(p + (int64_t)min(t1 + i * STEP, n - 1) * a.ldv);
  if (a.vscale != nullptr) {
    float w[E];
#pragma unroll
    for (int i = 0; i < E; ++i) w[i] = ld_f32(a.vscale + (t0 + min(t1 + i * STEP, n - 1)) * a.ldvs + h);
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] *= w[i];
  }
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (j >= nj || t1 + i * STEP >= n) x[i] = 0.f;
}
// kinds 0 and 1: a chunk's factors per token in 64 bits
template <int KIND>
__device__ __forceinline__ void fill_table(const ChunkArgs& a, double* table, int64_t t0, int n, int h) {
  if (threadIdx.x < C) {
    double x = 1.0;
    if ((int)threadIdx.x < n) x = KIND == 0 ? (double)a.decay[h] : exp((double)a.decay[(t0 + threadIdx.x) * a.ldd + h]);
    table[threadIdx.x] = x;
  }
  __syncthreads();
}
__device__ __forceinline__ double product(const double* table, int lo, int hi) {
  double p = 1.0;
  for (int t = lo; t < hi; ++t) p *= table[t];
  return p;
}

// ---- 1: U_c and D_c, DK threads.  A thread owns 8 key rows x 8 value columns, both as two runs of 4 half a tile apart (the quarter
// warps' 16-byte reads lie in different banks): 4 reads for 32 packed multiply-adds.
template <int DK, int KIND>
__global__ void __launch_bounds__(DK, DK == 64 ? 7 : 4) scan_state_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* ks = sm;                      // [C][DK] keys times the decay behind them, to the chunk's end
  float* vs = ks + C * DK;             // [C][JT]
  float* behind = vs + C * JT;         // [C] decay behind a token, to the chunk's end (kinds 0 and 1)
  double* table = reinterpret_cast<double*>(behind + C);           // [C]
  const Rows r = rows_of(a, blockIdx.z);
  const int t_lo = blockIdx.x * C;
  if (t_lo >= r.ql) return;
  const int n = min(C, r.ql - t_lo), h = blockIdx.y / a.nslices, slice = blockIdx.y % a.nslices;
  const int j0 = slice * JT, nj = min(JT, a.dv - j0);
  const int64_t t0 = r.q0 + t_lo;
  const int hq = h / a.rep;
  float decay = 1.f;                   // of the chunk, this thread's channel
  if (KIND != 2) {
    fill_table<KIND>(a, table, t0, n, h);
    if (threadIdx.x < C) behind[threadIdx.x] = (float)product(table, threadIdx.x + 1, C);
    __syncthreads();
  }
  {
    const int c = threadIdx.x, cc = min(c, a.dk - 1);
    const bool in = c < a.dk;
    const float* kp = a.k + t0 * a.ldk + (int64_t)hq * a.dk + cc;
    const float* dp = KIND == 2 ? a.decay + t0 * a.ldd + (int64_t)h * a.dk + cc : nullptr;
    // last sub-block first.  decay + lo: the product of the factors behind a token, with what its roundings left (a key's weight, and the
    // chunk's decay, have one rounding and not up to 64)
    float lo = 0.f;
#pragma unroll 1
    for (int s = NS - 1; s >= 0; --s) {
      float kx[SB], x[SB], vr[C * JT / DK / NS];
      load_rows(kp, a.ldk, s * SB, n, kx);
      if (KIND == 2) load_factors(dp, a.ldd, s * SB, n, in, x);
      load_values<DK, SB>(a, t0, s * SB, n, h, j0, nj, vr);
#pragma unroll
      for (int i = SB - 1; i >= 0; --i) {
        ks[(s * SB + i) * DK + c] = !(in && s * SB + i < n) ? 0.f : KIND == 2 ? fmaf(kx[i], decay, kx[i] * lo) : kx[i] * behind[s * SB + i];
        if (KIND == 2) {
          const float y = decay * x[i];
          lo = fmaf(lo, x[i], fmaf(decay, x[i], -y));
          decay = y;
        }
      }
#pragma unroll
      for (int i = 0; i < C * JT / DK / NS; ++i) vs[s * SB * JT + threadIdx.x + i * DK] = vr[i];
    }
  }
  __syncthreads();
  constexpr int KG = DK / 8;
  const int kg = threadIdx.x % KG, vg = threadIdx.x / KG;
  const int i0 = kg * 4, i1 = DK / 2 + kg * 4, c0 = vg * 4, c1 = JT / 2 + vg * 4;
  uint64_t acc[4][8];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[p][j] = 0;
#pragma unroll 2
  for (int t = 0; t < C; ++t) {
    const ulonglong2 k0 = lds2(ks + t * DK + i0), k1 = lds2(ks + t * DK + i1);
    const float4 x = *reinterpret_cast<const float4*>(vs + t * JT + c0), y = *reinterpret_cast<const float4*>(vs + t * JT + c1);
    const uint64_t vv[8] = {pack(x.x, x.x), pack(x.y, x.y), pack(x.z, x.z), pack(x.w, x.w), pack(y.x, y.x), pack(y.y, y.y), pack(y.z, y.z), pack(y.w, y.w)};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[0][j] = pfma(k0.x, vv[j], acc[0][j]); acc[1][j] = pfma(k0.y, vv[j], acc[1][j]);
      acc[2][j] = pfma(k1.x, vv[j], acc[2][j]); acc[3][j] = pfma(k1.y, vv[j], acc[3][j]);
    }
  }
  const int64_t at = (int64_t)(r.first + blockIdx.x) * a.H + h;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int col = (j < 4 ? c0 : c1) + (j & 3);
    if (col >= nj) continue;
    float* u = a.chunks + (at * a.dv + j0 + col) * a.dk;
    const float2 p0 = unpack(acc[0][j]), p1 = unpack(acc[1][j]), p2 = unpack(acc[2][j]), p3 = unpack(acc[3][j]);
    if (i0 < a.dk) *reinterpret_cast<float4*>(u + i0) = make_float4(p0.x, p0.y, p1.x, p1.y);     // (dk is a multiple of 4)
    if (i1 < a.dk) *reinterpret_cast<float4*>(u + i1) = make_float4(p2.x, p2.y, p3.x, p3.y);
  }
  if (slice == 0 && (int)threadIdx.x < a.dk) {
    if (KIND != 2) {
      const double all = product(table, 0, C);
      decay = (float)all;
      if (threadIdx.x == 0) a.decay_rest[at] = (float)(all - (double)decay);
    }
    a.decays[at * a.dk + threadIdx.x] = decay;
  }
}

// ---- 2: chunk states, two neighbouring key rows of a value column per thread; grid (plane / 512, B).  Eight chunks' loads in flight
template <bool REST>
__global__ void __launch_bounds__(256) scan_carry_kernel(ChunkArgs a) {
  const Rows r = rows_of(a, blockIdx.y);
  if (r.ql <= 0) return;
  const int per_head = a.dv * a.dk, plane = a.H * per_head;          // (the host checks that it fits)
  const int e = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (e >= plane) return;
  const int h = e / per_head, i = e % a.dk;
  float2* st = reinterpret_cast<float2*>(a.state + (int64_t)r.slot * plane + e);
  float2 S = r.ctx > 0 ? *st : make_float2(0.f, 0.f);
  const int nch = (r.ql + C - 1) / C, dstep = a.H * a.dk;
  float* u = a.chunks + (int64_t)r.first * plane + e;
  const float* d = a.decays + ((int64_t)r.first * a.H + h) * a.dk + i;
  const float* rest = a.decay_rest + (int64_t)r.first * a.H + h;
  for (int c0 = 0; c0 < nch; c0 += 8) {
    float2 uu[8], dd[8];
    float rr[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int c = min(c0 + x, nch - 1);
      asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(uu[x].x), "=f"(uu[x].y) : "l"(u + (int64_t)c * plane));
      asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(dd[x].x), "=f"(dd[x].y) : "l"(d + (int64_t)c * dstep));
      rr[x] = REST ? rest[(int64_t)c * a.H] : 0.f;
    }
#pragma unroll
    for (int x = 0; x < 8; ++x)
      if (c0 + x < nch) {
        *reinterpret_cast<float2*>(u + (int64_t)(c0 + x) * plane) = S;
        if (REST) uu[x] = make_float2(fmaf(rr[x], S.x, uu[x].x), fmaf(rr[x], S.y, uu[x].y));
        S = make_float2(fmaf(dd[x].x, S.x, uu[x].x), fmaf(dd[x].y, S.y, uu[x].y));
      }
  }
  *st = S;
}

// ---- 3: outputs of a chunk, 128 threads.  Thread (tg, cg) owns tokens tg + 8 m and value columns cg + 16 m: every thread has rows of
// every sub-block, so the triangular product is as much work for each.  Rows of q, k and S are padded by 4 floats: 16-byte reads of
// neighbouring rows lie in different banks.  The scores reuse the keys' place, the values lie behind them.
template <int DK> struct OutSmem {
  static constexpr int LD = DK + 4, LA = C + 4;
  static constexpr int Q = C * LD, S = JT * LD, KA = (C * LD > C * LA + C * JT) ? C * LD : C * LA + C * JT;
  static constexpr int FLOATS = Q + KA + S + 2 * NS * DK + 7 * DK + (DK / 32 + 4) * C + 2 * 2 * NS;
  static_assert(C * LA <= Q && LA >= JT, "the outputs pass through the queries' place");
};

template <int DK, int KIND, bool BEFORE>
__global__ void __launch_bounds__(128, DK == 64 ? 3 : 2) scan_out_kernel(ChunkArgs a) {
  using M = OutSmem<DK>;
  constexpr int LD = M::LD, LA = M::LA;
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                       // [C][LD]
  float* ks = qs + M::Q;                // [C][LD], then scores [C][LA] and values [C][JT]
  float* as = ks;
  float* vs = ks + C * LA;
  float* ss = ks + M::KA;               // [JT][LD] start state, columns as rows
  float* halves = ss + M::S;            // [NS][2][DK] decay of the first and second half of a sub-block
  float* between = halves + 2 * NS * DK;   // [4][DK]: ones, decay of sub-block 1, of 2, of both
  float* before = between + 4 * DK;     // [3][DK]: decay of the chunk in front of sub-blocks 1, 2, 3
  float* diag = before + 3 * DK;        // [DK / 32][C] bonus products, a part per 32 channels
  double* table = reinterpret_cast<double*>(diag + (DK / 32) * C);   // [C] (kinds 0 and 1)
  double* thalf = table + C;            // [NS][2]
  float* tq = reinterpret_cast<float*>(thalf + 2 * NS);              // [C] factors on q and, [C], on k
  float* tk = tq + C;
  const Rows r = rows_of(a, blockIdx.z);
  const int t_lo = blockIdx.x * C;
  if (t_lo >= r.ql) return;
  const int n = min(C, r.ql - t_lo), h = blockIdx.y / a.nslices, slice = blockIdx.y % a.nslices;
  const int j0 = slice * JT, nj = min(JT, a.dv - j0);
  const int64_t t0 = r.q0 + t_lo;
  const int hq = h / a.rep, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* S = a.chunks + (((int64_t)(r.first + blockIdx.x) * a.H + h) * a.dv + j0) * a.dk;
  const float* qp = a.q + t0 * a.ldq + (int64_t)hq * a.dk;
  const float* kp = a.k + t0 * a.ldk + (int64_t)hq * a.dk;
  if (KIND != 2) {
    fill_table<KIND>(a, table, t0, n, h);
    if (tid < C) {
      const int mid = tid / SB * SB + SB / 2;          // F(t): from the middle to behind t
      const double f = tid >= mid ? product(table, mid, tid + 1) : 1.0 / product(table, tid + 1, mid);
      tq[tid] = (float)(BEFORE ? (tid >= mid ? product(table, mid, tid) : 1.0 / product(table, tid, mid)) : f);
      tk[tid] = (float)(1.0 / f);
    } else if (tid < C + 2 * NS) {
      thalf[tid - C] = product(table, (tid - C) * (SB / 2), (tid - C + 1) * (SB / 2));
    }
    __syncthreads();
  }
  // start state -> shared memory (asynchronously; a column or channel that is not there is never copied into and zeroed instead)
  for (int i = tid; i < JT * (DK / 4); i += 128) {
    const int j = i / (DK / 4), c = (i % (DK / 4)) * 4;
    if (j < nj && c < a.dk)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(ss + j * LD + c)), "l"(S + (int64_t)j * a.dk + c) : "memory");
    else
      *reinterpret_cast<float4*>(ss + j * LD + c) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  bool deep = false;                    // out of the products' range
  float big = 0.f;
#pragma unroll 1
  for (int task = tid; task < NS * DK; task += 128) {
    const int c = task % DK, cc = min(c, a.dk - 1), s = task / DK, l0 = s * SB;
    const bool in = c < a.dk;
    float x[SB], qx[SB], kx[SB];
    load_rows(qp + cc, a.ldq, l0, n, qx);
    load_rows(kp + cc, a.ldk, l0, n, kx);
    if (KIND == 2) load_factors(a.decay + t0 * a.ldd + (int64_t)h * a.dk + cc, a.ldd, l0, n, in, x);
#pragma unroll
    for (int i = 0; i < SB; ++i)
      if (!in || l0 + i >= n) qx[i] = kx[i] = 0.f;
    if (BEFORE) {
      // bonus products of 16 tokens over this warp's 32 channels: four exchanges leave token (lane bits 4..1) per lane pair
      float d[SB];
      const float u = a.bonus != nullptr ? a.bonus[(int64_t)h * a.dk + cc] : 0.f;
#pragma unroll
      for (int i = 0; i < SB; ++i) d[i] = qx[i] * u * kx[i];
#pragma unroll
      for (int o = 16, w = SB / 2; o > 1; o >>= 1, w >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int i = 0; i < w; ++i) d[i] = (hi ? d[i + w] : d[i]) + __shfl_xor_sync(0xffffffffu, hi ? d[i] : d[i + w], o);
      }
      d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1);
      if (!(lane & 1)) diag[(c >> 5) * C + l0 + (lane >> 1)] = d[0];
    }
    if (KIND != 2) {
#pragma unroll
      for (int i = 0; i < SB; ++i) {
        const float y = qx[i] * tq[l0 + i], z = kx[i] * tk[l0 + i];
        qs[(l0 + i) * LD + c] = y;
        ks[(l0 + i) * LD + c] = z;
        big = fmaxf(big, fmaxf(fabsf(y), fabsf(z)));
      }
      continue;
    }
    float f = 1.f;
#pragma unroll
    for (int i = SB / 2; i < SB; ++i) {
      const float front = f;
      f *= x[i];
      const float y = qx[i] * (BEFORE ? front : f), z = kx[i] * recip(f);
      qs[(l0 + i) * LD + c] = y;
      ks[(l0 + i) * LD + c] = z;
      big = fmaxf(big, fmaxf(fabsf(y), fabsf(z)));
    }
    halves[(2 * s + 1) * DK + c] = f;
    deep |= !(f >= kLow && f <= kHigh);
    f = 1.f;
#pragma unroll
    for (int i = SB / 2 - 1; i >= 0; --i) {
      const float after = f;
      f *= x[i];
      const float y = qx[i] * recip(BEFORE ? f : after), z = kx[i] * after;
      qs[(l0 + i) * LD + c] = y;
      ks[(l0 + i) * LD + c] = z;
      big = fmaxf(big, fmaxf(fabsf(y), fabsf(z)));
    }
    halves[2 * s * DK + c] = f;
    deep |= !(f >= kLow && f <= kHigh);
  }
  if (KIND != 2 && tid < 2 * NS) deep = !(thalf[tid] >= (double)kLow && thalf[tid] <= (double)kHigh);
  // the values: to shared memory where their place is free, otherwise held in registers until the keys are done with it.  Columns are
  // swizzled by the token (the eight columns x four tokens that a product reads lie in different banks)
  float vr[C * JT / 128];
  load_values<128, C>(a, t0, 0, n, h, j0, nj, vr);
#pragma unroll
  for (int i = 0; i < C * JT / 128; ++i) deep |= !(fabsf(vr[i]) < kBig);      // (in a product 0 x infinity would reach earlier tokens)
  deep |= big > kBig;
  auto put_values = [&]() {
#pragma unroll
    for (int i = 0; i < C * JT / 128; ++i) {
      const int t = (tid + i * 128) / JT, j = tid % JT;
      vs[t * JT + (j ^ (8 * (t & 3)))] = vr[i];
    }
  };
  constexpr bool kValuesNow = C * LA >= C * LD;
  if (kValuesNow) put_values();
  asm volatile("cp.async.wait_all;" ::: "memory");
  auto bonus_of = [&](int t) {
    float d = 0.f;
#pragma unroll
    for (int g = 0; g < DK / 32; ++g) d += diag[g * C + t];
    return d;
  };
  float* op = a.out + t0 * a.H * a.dv + (int64_t)h * a.dv + j0;
  const int64_t ldo = (int64_t)a.H * a.dv;
  if (__syncthreads_or(deep)) {
    // ---- token by token: a value column per thread, raw q and k rows and the factors in shared memory
    for (int i = tid; i < C * DK; i += 128) {
      const int t = i / DK, c = i % DK;
      const bool in = t < n && c < a.dk;
      qs[t * DK + c] = in ? qp[(int64_t)t * a.ldq + c] : 0.f;
      ks[t * DK + c] = in ? kp[(int64_t)t * a.ldk + c] : 0.f;
    }
    float col[DK];
    if (tid < JT) {
#pragma unroll
      for (int c = 0; c < DK; ++c) col[c] = ss[tid * LD + c];
    }
    __syncthreads();
    for (int i = tid; i < C * DK; i += 128) {
      const int t = i / DK, c = i % DK;
      ss[t * DK + c] = !(t < n && c < a.dk) ? 1.f : KIND == 2 ? expf(a.decay[(t0 + t) * a.ldd + (int64_t)h * a.dk + c]) : (float)table[t];
    }
    __syncthreads();
    if (tid < nj) {
      for (int t = 0; t < n; ++t) {
        float v = a.v[(t0 + t) * a.ldv + (int64_t)h * a.dv + j0 + tid];
        if (a.vscale != nullptr) v *= a.vscale[(t0 + t) * a.ldvs + h];
        float sums[8], o = 0.f;           // chains of 8 channels, added pairwise: sums[l] is what 2^l of them left
#pragma unroll
        for (int c = 0; c < DK; c += 4) {
          const float4 q4 = *reinterpret_cast<const float4*>(qs + t * DK + c), k4 = *reinterpret_cast<const float4*>(ks + t * DK + c),
                       x4 = *reinterpret_cast<const float4*>(ss + t * DK + c);
          if ((c & 4) == 0) o = 0.f;
          if (BEFORE) o = fmaf(q4.w, col[c + 3], fmaf(q4.z, col[c + 2], fmaf(q4.y, col[c + 1], fmaf(q4.x, col[c], o))));
          col[c] = fmaf(x4.x, col[c], k4.x * v); col[c + 1] = fmaf(x4.y, col[c + 1], k4.y * v);
          col[c + 2] = fmaf(x4.z, col[c + 2], k4.z * v); col[c + 3] = fmaf(x4.w, col[c + 3], k4.w * v);
          if (!BEFORE) o = fmaf(q4.w, col[c + 3], fmaf(q4.z, col[c + 2], fmaf(q4.y, col[c + 1], fmaf(q4.x, col[c], o))));
          if (c & 4) {
            int l = 0;
#pragma unroll
            for (int g = c / 8; g & 1; g >>= 1) o += sums[l++];
            sums[l] = o;
          }
        }
        op[t * ldo + tid] = BEFORE ? fmaf(bonus_of(t), v, o) : o;
      }
    }
    return;
  }
  // factors of whole sub-blocks
  for (int c = tid; c < DK; c += 128) {
    if (KIND == 2) {
      float w[NS - 1];
#pragma unroll
      for (int x = 0; x < NS - 1; ++x) w[x] = halves[2 * x * DK + c] * halves[(2 * x + 1) * DK + c];
      between[c] = 1.f; between[DK + c] = w[1]; between[2 * DK + c] = w[2]; between[3 * DK + c] = w[1] * w[2];
      before[c] = w[0]; before[DK + c] = w[0] * w[1]; before[2 * DK + c] = w[0] * w[1] * w[2];
    } else {
      double w[NS - 1];
#pragma unroll
      for (int x = 0; x < NS - 1; ++x) w[x] = thalf[2 * x] * thalf[2 * x + 1];
      between[c] = 1.f; between[DK + c] = (float)w[1]; between[2 * DK + c] = (float)w[2]; between[3 * DK + c] = (float)(w[1] * w[2]);
      before[c] = (float)w[0]; before[DK + c] = (float)(w[0] * w[1]); before[2 * DK + c] = (float)(w[0] * w[1] * w[2]);
#pragma unroll
      for (int x = 0; x < 2 * NS; ++x) halves[x * DK + c] = (float)thalf[x];
    }
  }
  __syncthreads();
  // ---- scores: 80 tiles of 4 x 8 (eight per 16 x 16 block of the lower triangle), 20 lanes of every warp.  Off the diagonal a query is
  // brought to its sub-block's start and a key to its sub-block's end before they meet: factors of at most what each carries
  uint64_t sc[4][4];                   // two neighbouring keys' scores per number
  int si = 0, sj = 0, sb = 0, sp = 0;
  const bool scorer = lane < 20;
  if (scorer) {
    const int tile = warp * 20 + lane, blk = tile >> 3, w = tile & 7;
    sb = blk < 1 ? 0 : blk < 3 ? 1 : blk < 6 ? 2 : 3;
    sp = blk - sb * (sb + 1) / 2;
    si = sb * SB + (w & 3);            // tokens si + 4 m, keys sj + 2 m: neighbouring lanes read neighbouring rows
    sj = sp * SB + (w >> 2);
    const float* fq = sb == sp ? between : halves + 2 * sb * DK;
    const float* fk = sb == sp ? between : halves + (2 * sp + 1) * DK;
    const float* fb = between + (sb == 2 ? 1 : sp == 1 ? 2 : 3) * DK;          // read where a sub-block lies between
    // sums of 8 channels, added with the roundings of the additions carried along: a score is rounded like one number, and the output
    // (a second sum) not further from 64 bits than token by token
    uint64_t lost[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[i][j] = lost[i][j] = 0;
#pragma unroll 1
    for (int cc = 0; cc < DK; cc += 8) {
      uint64_t acc[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll
      for (int c = cc; c < cc + 8; c += 4) {
        const ulonglong2 f = lds2(fq + c), g = lds2(fk + c);
        ulonglong2 q4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          q4[i] = lds2(qs + (si + 4 * i) * LD + c);
          q4[i].x = pmul(q4[i].x, f.x);
          q4[i].y = pmul(q4[i].y, f.y);
        }
        if (sb > sp + 1) {
          const ulonglong2 b = lds2(fb + c);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            q4[i].x = pmul(q4[i].x, b.x);
            q4[i].y = pmul(q4[i].y, b.y);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ulonglong2 k4 = lds2(ks + (sj + 2 * j) * LD + c);
          k4.x = pmul(k4.x, g.x);
          k4.y = pmul(k4.y, g.y);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][j] = pfma(q4[i].y, k4.y, pfma(q4[i].x, k4.x, acc[i][j]));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 p0 = unpack(acc[i][2 * j]), p1 = unpack(acc[i][2 * j + 1]);
          const uint64_t y = padd(pack(p0.x + p0.y, p1.x + p1.y), lost[i][j]), t = padd(sc[i][j], y);
          lost[i][j] = psub(y, psub(t, sc[i][j]));
          sc[i][j] = t;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[i][j] = padd(sc[i][j], lost[i][j]);
  }
  __syncthreads();
  // ---- scores over the keys, q from its sub-block's middle to the chunk's start
  if (scorer) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int ti = si + 4 * i, tj = sj + 2 * j;
        const float2 pair = unpack(sc[i][j / 2]);
        float x = j & 1 ? pair.y : pair.x;
        if (tj > ti) x = 0.f;
        else if (BEFORE && tj == ti) x = bonus_of(ti);
        as[ti * LA + tj] = x;
      }
  }
  if (!kValuesNow) put_values();
  for (int i = tid; i < C * (DK / 4); i += 128) {
    const int t = i / (DK / 4), c = (i % (DK / 4)) * 4, s = t / SB;
    float4* p = reinterpret_cast<float4*>(qs + t * LD + c);
    const float4 f = *reinterpret_cast<const float4*>(halves + 2 * s * DK + c);
    float4 x = *p;
    x = make_float4(x.x * f.x, x.y * f.y, x.z * f.z, x.w * f.w);
    if (s > 0) {
      const float4 b = *reinterpret_cast<const float4*>(before + (s - 1) * DK + c);
      x = make_float4(x.x * b.x, x.y * b.y, x.z * b.z, x.w * b.w);
    }
    *p = x;
  }
  __syncthreads();
  // ---- o = q S: pairs along the key rows
  const int cg = tid & 15, tg = tid >> 4;
  float o[8][4];
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[m][j] = 0.f;
#pragma unroll 1
  for (int cc = 0; cc < DK; cc += 32) {      // partial sums of 32 channels
    uint64_t acc[8][4];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[m][j] = 0;
#pragma unroll 1
    for (int c = cc; c < cc + 32; c += 4) {
      ulonglong2 s4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) s4[j] = lds2(ss + (cg + 16 * j) * LD + c);
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const ulonglong2 q4 = lds2(qs + (tg + 8 * m) * LD + c);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[m][j] = pfma(q4.y, s4[j].y, pfma(q4.x, s4[j].x, acc[m][j]));
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 p = unpack(acc[m][j]);
        o[m][j] += p.x + p.y;
      }
  }
  // ---- o += scores v in 64-bit products of 8 x 8 x 4 (scores and values are 32-bit numbers, only the sums are wider: a chain of up to
  // 64 additions to a result of full size would cost more than the serial form's whole error).  Warp w takes the token tiles w and 7 - w,
  // together 18 steps of 4 keys; the sums so far change hands through the queries' place
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) qs[(tg + 8 * m) * LA + cg + 16 * j] = o[m][j];
  __syncthreads();
  const int lr = lane >> 2, lk = lane & 3;
  double acc[2][8][2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const float* p = qs + (8 * (x == 0 ? 7 - warp : warp) + lr) * LA + 2 * lk;
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const float2 v = *reinterpret_cast<const float2*>(p + 8 * y);
      acc[x][y][0] = v.x;
      acc[x][y][1] = v.y;
    }
  }
  const float* a0 = as + (8 * (7 - warp) + lr) * LA + lk;
  const float* a1 = as + (8 * warp + lr) * LA + lk;
  const float* vp = vs + lk * JT + lr;
#pragma unroll 2
  for (int t = 0; t < 8 * (8 - warp); t += 4) {
    double b[8];
#pragma unroll
    for (int y = 0; y < 8; ++y) b[y] = vp[t * JT + ((8 * y) ^ (8 * lk))];
    const double w0 = a0[t];
#pragma unroll
    for (int y = 0; y < 8; ++y) mma_f64(acc[0][y], w0, b[y]);
    if (t < 8 * (warp + 1)) {
      const double w1 = a1[t];
#pragma unroll
      for (int y = 0; y < 8; ++y) mma_f64(acc[1][y], w1, b[y]);
    }
  }
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int t = 8 * (x == 0 ? 7 - warp : warp) + lr;
    if (t >= n) continue;
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 8 * y + 2 * lk + e;
        if (j < nj) op[t * ldo + j] = (float)acc[x][y][e];
      }
  }
}

template <int DK, int KIND, bool BEFORE>
int launch_chunks(const ChunkArgs& a, int B, int nch, cudaStream_t stream) {
  const dim3 grid(nch, a.H * a.nslices, B);
  constexpr int s1 = (C * DK + C * JT + 3 * C) * 4, s3 = OutSmem<DK>::FLOATS * 4;
  static PerDeviceSmem g1, g3;
  LLMSS_CHECK_CUDA(g1.ensure(scan_state_kernel<DK, KIND>, s1));
  LLMSS_CHECK_CUDA(g3.ensure(scan_out_kernel<DK, KIND, BEFORE>, s3));
  scan_state_kernel<DK, KIND><<<grid, DK, s1, stream>>>(a);
  const int plane = a.H * a.dv * a.dk;
  scan_carry_kernel<KIND != 2><<<dim3((plane + 511) / 512, B), 256, 0, stream>>>(a);
  scan_out_kernel<DK, KIND, BEFORE><<<grid, 128, s3, stream>>>(a);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace

// Floats of scratch for T packed tokens of B sequences.
LLMSS_API int64_t llmss_linear_scan_chunked_floats(int T, int B, int H, int dk, int dv) {
  return ((int64_t)T / C + B) * H * ((int64_t)dk * (dv + 1) + 1);
}

// llmss_linear_scan over chunks of 64 tokens (see the head of this file): dk a multiple of 4 up to 128, the state and the scratch on
// 16-byte lines; any strides, value size and sequence lengths.  least: sequences of fewer tokens are left alone (a token alone costs a
// whole chunk here; llmss_linear_scan_upto takes them).
LLMSS_API int llmss_linear_scan_chunked_from(const float* q, int64_t ldq, const float* k, int64_t ldk, const float* v, int64_t ldv,
                                             const float* decay, int64_t ldd, int decay_kind, const float* bonus, const float* vscale, int64_t ldvs,
                                             float* out, float* state, const int* cu_q, const int* seq_lens, const int* slots, int B, int T,
                                             int max_q, int heads, int qk_heads, int dk, int dv, int read_before, float* scratch, int least,
                                             cudaStream_t stream) {
  LLMSS_REQUIRE(heads > 0 && qk_heads > 0 && heads % qk_heads == 0, "linear_scan_chunked: %d heads over %d query/key heads", heads, qk_heads);
  LLMSS_REQUIRE(dk > 0 && dk % 4 == 0 && dk <= 128 && dv > 0, "linear_scan_chunked: key size %d (a multiple of 4 up to 128), value size %d", dk, dv);
  LLMSS_REQUIRE(decay_kind >= 0 && decay_kind <= 2 && scratch != nullptr, "linear_scan_chunked: decay kind %d", decay_kind);
  LLMSS_REQUIRE((((uintptr_t)state | (uintptr_t)scratch) & 15) == 0, "linear_scan_chunked: state / scratch off the 16-byte lines");
  if (B <= 0 || max_q <= 0) return 0;
  ChunkArgs a{q, ldq, k, ldk, v, ldv, decay, ldd, bonus, vscale, ldvs, out, state, cu_q, seq_lens, slots, nullptr, nullptr, nullptr, heads, heads / qk_heads,
              dk, dv, (dv + JT - 1) / JT, least};
  a.chunks = scratch;
  a.decays = scratch + ((int64_t)T / C + B) * heads * (int64_t)dk * dv;
  a.decay_rest = a.decays + ((int64_t)T / C + B) * heads * dk;
  const int nch = (max_q + C - 1) / C;
  LLMSS_REQUIRE((int64_t)heads * a.nslices <= 65535 && B <= 65535 && (int64_t)heads * dv * dk < (1ll << 30), "linear_scan_chunked: grid too large");
#define LLMSS_LC(DK, KIND)                                                                      \
  return read_before ? launch_chunks<DK, KIND, true>(a, B, nch, stream) : launch_chunks<DK, KIND, false>(a, B, nch, stream)
  if (dk <= 64) {
    if (decay_kind == 0) LLMSS_LC(64, 0);
    if (decay_kind == 1) LLMSS_LC(64, 1);
    LLMSS_LC(64, 2);
  }
  if (decay_kind == 0) LLMSS_LC(128, 0);
  if (decay_kind == 1) LLMSS_LC(128, 1);
  LLMSS_LC(128, 2);
#undef LLMSS_LC
}

LLMSS_API int llmss_linear_scan_chunked(const float* q, int64_t ldq, const float* k, int64_t ldk, const float* v, int64_t ldv, const float* decay,
                                        int64_t ldd, int decay_kind, const float* bonus, const float* vscale, int64_t ldvs, float* out,
                                        float* state, const int* cu_q, const int* seq_lens, const int* slots, int B, int T, int max_q, int heads,
                                        int qk_heads, int dk, int dv, int read_before, float* scratch, cudaStream_t stream) {
  return llmss_linear_scan_chunked_from(q, ldq, k, ldk, v, ldv, decay, ldd, decay_kind, bonus, vscale, ldvs, out, state, cu_q, seq_lens, slots, B, T,
                                        max_q, heads, qk_heads, dk, dv, read_before, scratch, 0, stream);
}
