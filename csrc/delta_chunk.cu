// Long portions of the gated delta rule (csrc/delta.cu) over chunks of 32 tokens on the tensor cores.
//
//   token by token   S <- g_t S ;  u = beta_t (v_t - S^T k_t) ;  S <- S + k_t u^T ;  o_t = S^T q_t
//
// With G_i the sum of the log decays of a chunk's tokens up to i, w_ij = exp(G_i - G_j) and S_0 the state in front of the chunk, the written
// values of a chunk solve a triangular system, and everything else is products:
//   R_i = beta_i (v_i - exp(G_i) S_0^T k_i)          L_ij = beta_i w_ij k_i . k_j  (j < i)        U = (1 + L)^-1 R
//   o_i = exp(G_i) S_0^T q_i + sum_(j <= i) w_ij (q_i . k_j) U_j          S = exp(G_C) S_0 + sum_j w_Cj k_j U_j^T
// (the chunkwise form of the delta rule of Yang, Wang, Zhang, Shen and Kim, 2024, with the decays of Yang, Kautz and Hatamizadeh, 2024).
// T = (1 + L)^-1 does not depend on the state; for unit keys, strengths up to 1 and decays up to 1 its entries are at most 1.
//
// Two launches.  delta_prep_kernel, a block per chunk and key head: scores, L, T, the outputs' weights and the numbers per token, for every value head;
// T and the weights leave as the shared-memory tiles that the products read.
// delta_chunk_kernel, a block per sequence, head and 128 value columns, carries the state.  Value columns are the lanes of tensor memory, so that a
// thread owns a row of the transposed state, and all scaling and splitting of a row is its own work:
//   warps 0-3    R from S_0^T k (tensor memory), then U = T R, split for the two products that read it
//   warps 4-11   the state, 64 of 128 key rows each, in registers; S_0^T q; the outputs
//   warps 12-14  q and k of the next chunks, scaled and split into shared memory
//   warp  15     issues the copies and the products
// The products that wait for the state (S_0^T k -> R -> T R -> S) are the chain; the others lie in its gaps.
//
// Rounding.  Operands are rows scaled and cut into three 16-bit numbers (split16.cuh); their sums are exact in one accumulator, close to it in
// the other, and meet in one 32-bit addition.  A row's parts carry 2^-34 of its largest number: entries down to 2^-11 of it have the bits of a 32-bit number,
// smaller ones fewer.  That is no loss while the larger ones are in the same sums; where they are not (tokens that a decay has parted, keys of other
// channels, a large value behind the token), `spread` and the count over the state notice.  (With two parts of the state an entry 2^-10 of its column's
// largest entered the products with 14 bits.)  The state itself is a 32-bit number in a register, rounded once per chunk where it was rounded once per
// token.  Log decays sum in 64 bits.
// At a chunk that the products cannot take (decays that grow by more than e^0.25 a token or shrink by more than e^(-2^20), values that are not finite or
// beyond 2^100, entries of T of 4 and more, numbers that differ by more than the parts carry) a block ends: it leaves the state in front of it, and delta_scan_kernel, launched behind, takes the sequence's
// other tokens, so that a value that is no number reaches what it reaches token by token.  (Such chunks token by token in this kernel took 114 us
// each, one after another: 8 prompts of 576 .. 1472 tokens whose decays grow 910 us token by token, 5267 so, 1005 now; a batch takes no longer than
// its chunks in front of such ones and their sequences' other tokens, one launch after the other.)
//
// B200, 16 heads of 128 x 128, against token by token: 8 prompts of 576 .. 1472 tokens 910 -> 343 us (68 + 272 for the two launches, 3 for the one behind),
// 8 of 1024 640 -> 284, one of 1500 610 -> 278, 8 of 64 50 -> 41; without the three tests of the numbers' size 336, 268, 264 and 40.  Against 64 bits, of the
// norm (token by token in brackets): outputs 1.3e-7 (1.5e-7), states 7.9e-8 (1.1e-7); decays near 1 1.3e-7 (2.7e-7) and 1.1e-7 (2.5e-7); worst token 2.3e-7
// (2.7e-7), worst column 1.7e-7 (1.9e-7).  The second launch is bound by its chain, 5.9 us or about 11 000 clocks a chunk: products with
// the state 2000, R 1000, T R 500, U 1000, the update's product 1300, the state 3200, half of each the arithmetic of splitting (24 clocks of a
// scheduler for two numbers) and the rest six hand-overs of 300 to 400 clocks each, part of these figures.  With scores and T in the same launch (no first launch) a chunk took
// 13000 clocks, the scores' products taking shared memory's path from the other warps; with 16 warps for the state 13000 against 11000.  Straight-line
// code of 200 KB, before its loops were rolled, took 24000.
#include "delta.cuh"
#include "split16.cuh"

namespace {

using namespace split16;

constexpr int C = kDeltaChunk, KD = 128, VL = kDeltaCols;            // tokens of a chunk, key rows, value columns of a block
constexpr int kWarps = 16, kThreads = kWarps * 32;
constexpr int SUB = 2 * C * 128;                     // 64 key rows (columns of the tile) of [k; q], 16-bit, 128-byte rows
constexpr int SLICE = 2 * SUB, KQ = 3 * SLICE;       // one of h / l / m; a stage
constexpr int STAGES = 3;
constexpr int TRI = C * 128, TRIS = 3 * TRI;         // a part of [T | outputs' weights]: rows of 2 x 32 numbers
constexpr float kTScale = 0x1p-10f;                  // entries of T, below 4

// tensor memory, columns: products with the state [0, 128) and R over those with k; T R (three runs); over them the state's update [0, 256);
// outputs (three runs); the state's parts (the last one, of two runs, over the update that its own thread has read) and, once both products with the
// state are done, U's
constexpr int tXP = 0, tYP = 64, tU = 128, tR = 0, tR3 = 64, tXS = 0, tYS = 128, tO = 256, tSH = 384, tSL = 448, tSM = 128, tU1 = 384, tU2 = 432;

struct __align__(16) Scalars {      // of a chunk and head, per token
  float be[C], bk[C];               // strength; strength * decay since the chunk's start * scale of k
  float gq[C];                      // decay since the chunk's start * scale of q
  float gend[C];                    // decay to the chunk's end * scale of k, of `most`
  float as[C];                      // scales of the rows of the outputs' weights
  float decay[C];                   // of a token; 0 in a chunk of sparse keys (see spread)
  float all, most, low;             // decay of the chunk; a power of two; the smallest decay since its start, negative in a chunk of sparse keys
  int bad;                          // not for the products
  int pad[31];
  int done[kDeltaDone];             // (of a sequence's first chunk) tokens that the second launch has done, per 128 value columns
};
struct __align__(16) Prepared {     // what the first launch leaves, and the second copies
  uint8_t tri[TRIS];                // [h, l, m][32 rows][T: 64 bytes, the outputs' weights: 64 bytes]
  Scalars sc;
};
static_assert(sizeof(Prepared) == LLMSS_DELTA_PREPARED && sizeof(Prepared) % 1024 == 0, "tiles stay on their swizzle period");
static_assert(sizeof(Scalars) == 1024 && kDeltaDoneAt % 4 == 0, "the tokens done end a record");
struct Bars {
  uint64_t kq_full[STAGES], kq_empty[STAGES], ops_full[4];
  uint64_t s_full, p, pq_read, r_full, tr, u1_full, u2_full, s2, o2, verdict;
};
struct __align__(16) Smem {
  float o[C][VL];                   // decayed products of the state in front of the chunk with the queries
  float s_scale[VL], u1_scale[VL], u2_scale[2][VL], smax[2][VL];
  Bars bar;
  int solve_bad[2], state_bad[2];   // 1 + the last chunk of this parity whose values, or the state in front of it, are not for the products
  int quit, stop;                   // a wait ran out; a chunk is left to the launch behind
  uint32_t tmem;
};
constexpr int kSmemBytes = 1024 + STAGES * KQ + 4 * (int)sizeof(Prepared) + (int)sizeof(Smem);
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

// pairs of operand parts, two bits each, first one lowest: h h, h l, l h, l l, h m, m h
constexpr uint32_t kFirst = 0 | 0 << 2 | 1 << 4 | 1 << 6 | 0 << 8 | 2 << 10, kSecond = 0 | 1 << 2 | 0 << 4 | 1 << 6 | 2 << 8 | 0 << 10;

// 32 scaled numbers of a row into three runs of 16 columns
__device__ __forceinline__ void put_row(uint32_t to, uint32_t to3, const pair_t (&y)[C / 2]) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    uint32_t h[8], l[8], m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split3(y[g * 8 + i], h[i], l[i], m[i]);
    tmem_st8(to + g * 8, h);
    tmem_st8(to + 16 + g * 8, l);
    tmem_st8(to3 + g * 8, m);
  }
  tmem_st_wait();
}
// 2 N numbers of two accumulators, summed
template <int N>
__device__ __forceinline__ void get_sums(uint32_t x, uint32_t y, pair_t (&s)[N]) {
  static_assert(N == 8 || N == 4, "a pair of loads");
  uint32_t p[2 * N], q[2 * N];
  if constexpr (N == 8) {
    tmem_ld_32x32b_x16(x, p);
    tmem_ld_32x32b_x16(y, q);
  } else {
    tmem_ld_32x32b_x8(x, p);
    tmem_ld_32x32b_x8(y, q);
  }
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = padd(pack(p[2 * i], p[2 * i + 1]), pack(q[2 * i], q[2 * i + 1]));
}
// 16 numbers of three accumulators 32 columns apart
__device__ __forceinline__ void get_sums3(uint32_t x, pair_t (&s)[8]) {
  uint32_t p[16], q[16], r[16];
  tmem_ld_32x32b_x16(x, p);
  tmem_ld_32x32b_x16(x + 32, q);
  tmem_ld_32x32b_x16(x + 64, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = padd(pack(p[2 * i], p[2 * i + 1]), padd(pack(q[2 * i], q[2 * i + 1]), pack(r[2 * i], r[2 * i + 1])));
}
__device__ __forceinline__ void lds_pairs(const float* p, pair_t& x, pair_t& y) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  x = v.x;
  y = v.y;
}

// Whether the tokens of a chunk differ by more than a column's parts carry.  What the tokens up to one have written to the column, decayed, and the state in
// front of the chunk give the size n of that token's numbers; where n is below 2^-11 to 2^-12 of the column's largest (us: a column's numbers are scaled to
// 2^11 .. 2^12), fewer than 24 bits of them are left.  One such number is chance (1 in 1400 of normal ones that stand alone); a token that is small
// in all 32 columns of the warp, or five tokens of a column, are not.  s: scale of the column's state.  The same answer for the whole warp.
// The state has the like (in its warps): 8 of a thread's 64 key rows below 2^-11 to 2^-12 of the column's largest, 3 once keys were sparse.  Fewer such rows
// stay: a query that reads nothing but them gets them to 2^-34 of the column's largest.
// Earlier forms: in front of T R in the chain 343 -> 349 us, the state's count beside U 352.
__device__ __forceinline__ bool spread(const pair_t (&y)[C / 2], const Scalars& sc, int tokens, float s, float us) {
  float n = s > 0x1p-98f ? s * 0x1p11f : 0.f;
  if (__all_sync(0xffffffffu, n * sc.low >= us)) return false;          // the usual case: the state alone is not small at any token
  const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(us)));
  uint32_t small = 0, some = 0, few = 0;
#pragma unroll
  for (int i = 0; i < C; i += 4) {
    const float4 f = *reinterpret_cast<const float4*>(sc.decay + i);
    const float2 p = unpack(y[i / 2]), q = unpack(y[i / 2 + 1]);
    const float by[4] = {f.x, f.y, f.z, f.w}, x[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      n = fmaxf(n * by[e], fabsf(x[e]) * us);
      if (n < most) small |= 1u << (i + e);
      if (n > 0.f) some |= 1u << (i + e);
      if (n > 0.f && n < us) few |= 1u << (i + e);
    }
  }
  const uint32_t there = tokens < C ? (1u << tokens) - 1 : ~0u;
  return (__reduce_and_sync(0xffffffffu, small) & __reduce_or_sync(0xffffffffu, some) & there) != 0 || __any_sync(0xffffffffu, __popc(few & there) >= 5);
}

__global__ void __launch_bounds__(kThreads, 1) delta_chunk_kernel(DeltaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.x;
  const int q0 = a.cu_q[b], ql = a.cu_q[b + 1] - q0, ctx = a.seq_lens[b] - ql, slot = a.slots[b];
  if (slot < 0 || ctx < 0 || ql < a.least) return;           // (the same for the whole block)
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sKQ = tiles;                           // [stages][h, l, m][2][64 rows: k, q][128 bytes]
  Prepared* prep = reinterpret_cast<Prepared*>(sKQ + STAGES * KQ);      // [4]: read until a chunk's outputs are stored
  Smem& sm = *reinterpret_cast<Smem*>(prep + 4);
  Bars& bar = sm.bar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, hk = h / a.rep, dk = a.dk;
  const int j0 = blockIdx.z * VL, nj = min(VL, a.dv - j0);
  const int nch = min((ql + C - 1) / C, a.chunks);
  int* quit = &sm.quit;

  if (warp == 15) {
    tmem_alloc(&sm.tmem, 512);
    tmem_relinquish();
    if (lane == 0) {
      for (int i = 0; i < STAGES; ++i) {
        mbar_init(&bar.kq_full[i], 16);
        mbar_init(&bar.kq_empty[i], 1);
      }
      for (int i = 0; i < 4; ++i) mbar_init(&bar.ops_full[i], 1);
      for (int i = 0; i < 2; ++i) sm.solve_bad[i] = sm.state_bad[i] = 0;
      mbar_init(&bar.s_full, 8);
      mbar_init(&bar.p, 2);           // the products and, behind all that it has waited for, the issuing warp
      mbar_init(&bar.pq_read, 8);
      mbar_init(&bar.r_full, 4);
      mbar_init(&bar.tr, 1);
      mbar_init(&bar.u1_full, 4);
      mbar_init(&bar.u2_full, 4);
      mbar_init(&bar.s2, 2);
      mbar_init(&bar.o2, 1);
      mbar_init(&bar.verdict, 4);
      sm.quit = sm.stop = 0;
      fence_mbar_init();
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = sm.tmem;
  // behind the waits for its verdict and for s2 or pq_read: whether chunk c is not for the products
  auto bad = [&](int c) { return prep[c & 3].sc.bad || sm.solve_bad[c & 1] == c + 1 || sm.state_bad[c & 1] == c + 1; };

  if (warp < 4) {
    // ---- R and U: one value column per thread
    const int v = threadIdx.x;
    const uint32_t row = tmem + ((uint32_t)(warp * 32) << 16);
    const float* vp = a.v + (int64_t)h * a.dv + j0 + min(v, nj - 1);
    for (int c = 0; c < nch; ++c) {
      const int st = c & 1, n = min(C, ql - c * C);
      const Scalars& sc = prep[c & 3].sc;
      pair_t x[C / 2];
      {
        float f[C];
#pragma unroll
        for (int i = 0; i < C; ++i) f[i] = ld_nc(vp + (int64_t)(q0 + c * C + min(i, n - 1)) * a.ldv);
        const int rows = v < nj ? n : 0;
#pragma unroll
        for (int i = 0; i < C; i += 2) x[i / 2] = pack(i < rows ? f[i] : 0.f, i + 1 < rows ? f[i + 1] : 0.f);
      }
      wait_bar(&bar.ops_full[c & 3], c >> 2, quit);
      if (c > 0) {
        wait_bar(&bar.s2, c - 1, quit);
        wait_bar(&bar.verdict, c - 1, quit);
        if (bad(c - 1)) break;
      }
      wait_bar(&bar.p, c, quit);
      tcgen05_fence_after();
      const pair_t ss = both(-sm.s_scale[v]);
      float mx = 0.f, mx1 = 0.f;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        pair_t p[8];
        get_sums(row + tXP + g * 16, row + tYP + g * 16, p);
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          pair_t be0, be1, bk0, bk1;
          lds_pairs(sc.be + g * 16 + 2 * i, be0, be1);
          lds_pairs(sc.bk + g * 16 + 2 * i, bk0, bk1);
          pair_t &y0 = x[g * 8 + i], &y1 = x[g * 8 + i + 1];
          y0 = pfma(be0, y0, pmul(pmul(ss, p[i]), bk0));
          y1 = pfma(be1, y1, pmul(pmul(ss, p[i + 1]), bk1));
          mx = max_abs(mx, y0);
          mx1 = max_abs(mx1, y1);
        }
      }
      const Scale r = scale_of(max_abs(mx, mx1, 0.f));
      if (__any_sync(0xffffffffu, r.huge) && lane == 0) sm.solve_bad[st] = c + 1;
#pragma unroll
      for (int i = 0; i < C / 2; ++i) x[i] = pmul(x[i], both(r.inv));
      put_row(row + tR, row + tR3, x);
      arrive_warp(&bar.r_full);
      wait_bar(&bar.tr, c, quit);
      tcgen05_fence_after();
      mx = mx1 = 0.f;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        pair_t p[8];
        get_sums3(row + tU + g * 16, p);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          x[g * 8 + i] = p[i];
          if (i & 1) mx1 = max_abs(mx1, p[i]);
          else mx = max_abs(mx, p[i]);
        }
      }
      const Scale u = scale_of(max_abs(mx, mx1, 0.f));
      const float us = u.s * r.s * kTScale;
      sm.u1_scale[v] = us * sc.most;
      sm.u2_scale[st][v] = us;
      {
        pair_t z[C / 2];
#pragma unroll
        for (int i = 0; i < C / 2; i += 2) {
          pair_t g0, g1;
          lds_pairs(sc.gend + 2 * i, g0, g1);
          x[i] = pmul(x[i], both(u.inv));
          x[i + 1] = pmul(x[i + 1], both(u.inv));
          z[i] = pmul(x[i], g0);
          z[i + 1] = pmul(x[i + 1], g1);
        }
        put_row(row + tU1, row + tU1 + 32, z);
      }
      arrive_warp(&bar.u1_full);
      put_row(row + tU2, row + tU2 + 32, x);
      arrive_warp(&bar.u2_full);
      if (spread(x, sc, n, sm.s_scale[v], us) && lane == 0) sm.solve_bad[st] = c + 1;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.verdict);
    }
  } else if (warp < 12) {
    // ---- the state: a value column and 64 key rows per thread; tokens 16 part .. 16 part + 15 of the outputs
    const int part = (warp - 4) >> 2, quarter = warp & 3, v = quarter * 32 + lane;
    const uint32_t row = tmem + ((uint32_t)(quarter * 32) << 16);
    float* sp = a.state + (((int64_t)slot * a.H + h) * a.dv + j0 + min(v, nj - 1)) * dk + part * 64;
    pair_t S[32];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ctx > 0 && v < nj && part * 64 + 2 * i < dk) t = *reinterpret_cast<const float4*>(sp + 2 * i);      // (dk is a multiple of 4)
      S[i] = pack(t.x, t.y);
      S[i + 1] = pack(t.z, t.w);
    }
    auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); };       // the two warps of 32 columns
    const int64_t ldo = (int64_t)a.H * a.dv;
    float ss = 0.f, mx[4] = {0.f, 0.f, 0.f, 0.f};
    int most_few = 7;                  // once keys are sparse: 2
#pragma unroll
    for (int i = 0; i < 32; ++i) mx[i & 3] = max_abs(mx[i & 3], S[i]);
    int c = 0;
    // parts of the state in front of chunk c; then that chunk
#pragma unroll 1
    for (;; ++c) {
      if (c < nch) {
        const float mine = max_abs(max_abs(mx[0], mx[1], mx[2]), mx[3], 0.f);
        sm.smax[part][v] = mine;
        meet();
        const Scale s = scale_of(max_abs(mine, sm.smax[part ^ 1][v], 0.f));
        ss = s.s;
        if (__any_sync(0xffffffffu, s.huge) && lane == 0) sm.state_bad[c & 1] = c + 1;
        if (part == 0) sm.s_scale[v] = s.s;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint32_t hi[16], lo[16], mi[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) split3(pmul(S[i * 16 + e], both(s.inv)), hi[e], lo[e], mi[e]);
          tmem_st16(row + tSM + part * 64 + i * 16, mi);
          if (i == 0) {
            if (c > 0) wait_bar(&bar.o2, c - 1, quit);         // U's parts, in the same place, have been read
            tcgen05_fence_after();
          }
          tmem_st16(row + tSH + part * 32 + i * 16, hi);
          tmem_st16(row + tSL + part * 32 + i * 16, lo);
        }
        tmem_st_wait();
        arrive_warp(&bar.s_full);
        // key rows (of 64) whose numbers are below 2^-11 to 2^-12 of the column's largest, and not 0: see spread
        int few = 0;
        const uint32_t below = 2 * __float_as_uint(ss) - 1;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float2 x = unpack(S[e]);
          few += (2 * __float_as_uint(x.x) - 1 < below) + (2 * __float_as_uint(x.y) - 1 < below);
        }
        wait_bar(&bar.ops_full[c & 3], c >> 2, quit);
        if (prep[c & 3].sc.low < 0.f) most_few = 2;
        if (__any_sync(0xffffffffu, few > most_few) && lane == 0) sm.state_bad[c & 1] = c + 1;
      } else {
        wait_bar(&bar.o2, c - 1, quit);
        tcgen05_fence_after();
      }
      if (c > 0) {
        // outputs of the chunk before (everything read before the first store: the compiler cannot tell `out` from shared memory)
        const int p = c - 1, n = v < nj ? min(C, ql - p * C) - part * 16 : 0;
        const Scalars& sc = prep[p & 3].sc;
        pair_t o[8];
        get_sums3(row + tO + part * 16, o);
        const pair_t us = both(sm.u2_scale[p & 1][v]);
        float y[16];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          pair_t w0, w1;
          lds_pairs(sc.as + part * 16 + 2 * i, w0, w1);
          const float2 z0 = unpack(pmul(pmul(us, w0), o[i])), z1 = unpack(pmul(pmul(us, w1), o[i + 1]));
          y[2 * i] = z0.x + sm.o[part * 16 + 2 * i][v];
          y[2 * i + 1] = z0.y + sm.o[part * 16 + 2 * i + 1][v];
          y[2 * i + 2] = z1.x + sm.o[part * 16 + 2 * i + 2][v];
          y[2 * i + 3] = z1.y + sm.o[part * 16 + 2 * i + 3][v];
        }
        float* op = a.out + (int64_t)(q0 + p * C + part * 16) * ldo + (int64_t)h * a.dv + j0 + v;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i < n) op[i * ldo] = y[i];
      }
      if (c >= nch) break;
      const Scalars& sc = prep[c & 3].sc;
      const pair_t all = both(sc.all);
      wait_bar(&bar.p, c, quit);
      tcgen05_fence_after();
      {
        pair_t o[8];
        get_sums(row + tXP + C + part * 16, row + tYP + C + part * 16, o);
        arrive_warp(&bar.pq_read);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 y = unpack(pmul(both(ss), o[i]));
          sm.o[part * 16 + 2 * i][v] = y.x * sc.gq[part * 16 + 2 * i];
          sm.o[part * 16 + 2 * i + 1][v] = y.y * sc.gq[part * 16 + 2 * i + 1];
        }
      }
      wait_bar(&bar.verdict, c, quit);
      const pair_t us = both(sm.u1_scale[v]);
      wait_bar(&bar.s2, c, quit);
      tcgen05_fence_after();
      if (bad(c)) break;
      mx[0] = mx[1] = mx[2] = mx[3] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        pair_t p[8];
        get_sums(row + tXS + part * 64 + i * 16, row + tYS + part * 64 + i * 16, p);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          S[i * 8 + e] = pfma(all, S[i * 8 + e], pmul(us, p[e]));
          mx[e & 3] = max_abs(mx[e & 3], S[i * 8 + e]);
        }
      }
    }
    // The state in front of chunk c, and what is left of the sequence.  Where a wait ran out that is all of it: the state in memory is still the one in
    // front of the sequence, and the launch behind writes every output again.  (One answer for all of these warps.)
    uint32_t ran_out = *(volatile int*)&sm.quit;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %0, 0;\n\tbar.red.or.pred q, 5, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "+r"(ran_out)::"memory");
    if (threadIdx.x == 128) {
      if (ran_out) printf("[llmss_b200] delta_chunk: a wait ran out, token by token instead (block %d,%d,%d)\n", b, h, (int)blockIdx.z);
      reinterpret_cast<Prepared*>(a.prepared)[(int64_t)(q0 / C + b) * a.H + h].sc.done[blockIdx.z] = ran_out ? 0 : min(c * C, ql);
    }
    if (v < nj && !ran_out) {
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 x = unpack(S[i]), y = unpack(S[i + 1]);
        if (part * 64 + 2 * i < dk) *reinterpret_cast<float4*>(sp + 2 * i) = make_float4(x.x, x.y, y.x, y.y);
      }
    }
  } else if (warp < 15) {
    // ---- rows of k and q: 16 groups of four a chunk, eight lanes to a row; the three warps take turns
    const int l8 = lane & 7, groups = 16 * nch;
    float4 x[4];
    auto load = [&](int at) {           // at: 16 * chunk + group (eight of k, eight of q).  Loads never stand behind a branch
      const int64_t t = q0 + min((at >> 4) * C + (at & 7) * 4 + (lane >> 3), ql - 1);
      const float* p = ((at & 8) ? a.q + t * a.ldq : a.k + t * a.ldk) + (int64_t)hk * dk;
#pragma unroll
      for (int m = 0; m < 4; ++m) x[m] = ld_nc4(p + min(m * 32 + l8 * 4, dk - 4));
    };
    load(warp - 12);
#pragma unroll 1
    for (int at = warp - 12; at < groups; at += 3) {
      const int c = at >> 4, stage = c % STAGES, i = (at & 7) * 4 + (lane >> 3);
      pair_t y[8];
      float mx = 0.f;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const bool in = c * C + i < ql && m * 32 + l8 * 4 < dk;
        y[2 * m] = in ? pack(x[m].x, x[m].y) : 0;
        y[2 * m + 1] = in ? pack(x[m].z, x[m].w) : 0;
        mx = max_abs(max_abs(mx, y[2 * m]), y[2 * m + 1]);
      }
      load(min(at + 3, groups - 1));
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) mx = max_abs(mx, __shfl_xor_sync(0xffffffffu, mx, o), 0.f);
      const Scale s = scale_of(mx);
      if (c >= STAGES) wait_bar(&bar.kq_empty[stage], c / STAGES - 1, quit);
      if (*(volatile int*)&sm.stop) break;
      uint8_t* to = sKQ + stage * KQ + ((at & 8) ? C * 128 : 0) + i * 128 + ((l8 & 1) << 3);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint2 hh, ll, mm;
        split3(pmul(y[2 * m], both(s.inv)), hh.x, ll.x, mm.x);
        split3(pmul(y[2 * m + 1], both(s.inv)), hh.y, ll.y, mm.y);
        uint8_t* p = to + (m >> 1) * SUB + ((((m & 1) * 4 + (l8 >> 1)) ^ (i & 7)) << 4);
        *reinterpret_cast<uint2*>(p) = hh;
        *reinterpret_cast<uint2*>(p + SLICE) = ll;
        *reinterpret_cast<uint2*>(p + 2 * SLICE) = mm;
      }
      fence_proxy_async_smem();
      arrive_warp(&bar.kq_full[stage]);
    }
  } else {
    // ---- products (whole warp in the loop, one lane issues)
    const uint32_t kq = smem_u32(sKQ);
    const uint8_t* from = a.prepared + ((int64_t)(q0 / C + b) * a.H + h) * sizeof(Prepared);
    auto fetch = [&](int c) {           // T, the outputs' weights and the numbers per token of a chunk
      if (elect_one()) {
        mbar_arrive_expect_tx(&bar.ops_full[c & 3], sizeof(Prepared));
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(prep + (c & 3))),
                     "l"(from + (int64_t)c * a.H * sizeof(Prepared)), "r"((uint32_t)sizeof(Prepared)), "r"(smem_u32(&bar.ops_full[c & 3])) : "memory");
      }
      __syncwarp();
    };
    // a row of U or R (three parts, 32 tokens) times a triangle: h h | h l, l h | h m, l l, m h, an accumulator each.  (Products onto one accumulator are
    // all of one shape: only those are sure to be added one after the other.)
    auto by_triangle = [&](uint32_t d, uint32_t at, uint32_t at3, uint32_t lo) {
#pragma unroll
      for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int y = 0; y < 3 - x; ++y)
#pragma unroll
          for (int k = 0; k < 2; ++k)
            umma_ts(d + (x + y) * C, (x == 2 ? at3 : at + x * 16) + k * 8, lo + y * (TRI / 16) + k * 2, idesc(C, 0), x > 0 || k > 0);
    };
    for (int c = 0; c < min(nch, 3); ++c) fetch(c);
    for (int c = 0; c < nch; ++c) {
      const uint32_t base = kq + (c % STAGES) * KQ, tr = smem_u32(prep[c & 3].tri);
      wait_bar(&bar.kq_full[c % STAGES], c / STAGES, quit);
      wait_bar(&bar.ops_full[c & 3], c >> 2, quit);
      wait_bar(&bar.s_full, c, quit);
      tcgen05_fence_after();
      if (elect_one()) {        // the state times [k; q]
        const uint32_t lo = desc_lo(base);
#pragma unroll 1
        for (int x = 0; x < 6; ++x) {
          const uint32_t first = (kFirst >> (2 * x)) & 3, lb = lo + ((kSecond >> (2 * x)) & 3) * (SLICE / 16);
          const uint32_t at = tmem + (first == 0 ? tSH : first == 1 ? tSL : tSM), skip = first == 2 ? 32 : 0;
          const uint32_t d = tmem + (x == 0 ? tXP : tYP);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_ts(d, at + k * 8 + (k >> 2) * skip, lb + (k >> 2) * (SUB / 16) + (k & 3) * 2, idesc(2 * C, 0), x > 1 || k > 0);
        }
        umma_commit(&bar.p);
        mbar_arrive(&bar.p);
      }
      __syncwarp();
      wait_bar(&bar.r_full, c, quit);
      tcgen05_fence_after();
      if (elect_one()) {
        by_triangle(tmem + tU, tmem + tR, tmem + tR3, desc_lo(tr));
        umma_commit(&bar.tr);
      }
      __syncwarp();
      wait_bar(&bar.pq_read, c, quit);          // (and the outputs of chunk c - 1 have been read)
      wait_bar(&bar.u1_full, c, quit);
      tcgen05_fence_after();
      if (elect_one()) {          // U times the keys, whose rows are the tokens
        const uint32_t lo = desc_lo(base, SUB);
#pragma unroll 1
        for (int x = 0; x < 6; ++x) {
          const uint32_t at = tmem + tU1 + ((kFirst >> (2 * x)) & 3) * 16, lb = lo + ((kSecond >> (2 * x)) & 3) * (SLICE / 16);
          const uint32_t d = tmem + (x == 0 ? tXS : tYS);
          umma_ts(d, at, lb, idesc(KD, 1), x > 1);
          umma_ts(d, at + 8, lb + 16 * 128 / 16, idesc(KD, 1), 1);
        }
        umma_commit(&bar.s2);
        mbar_arrive(&bar.s2);
      }
      __syncwarp();
      wait_bar(&bar.u2_full, c, quit);
      tcgen05_fence_after();
      if (elect_one()) {
        by_triangle(tmem + tO, tmem + tU2, tmem + tU2 + 32, desc_lo(tr) + 4);
        umma_commit(&bar.o2);
      }
      __syncwarp();
      wait_bar(&bar.verdict, c, quit);
      if (bad(c)) {
        wait_bar(&bar.o2, c, quit);
        // nothing reads the later rows of k and q: their warps get this chunk's place and find `stop`.  (No other phase is completed out of turn: a warp that
        // still waits for the one before would never see it.)
        if (lane == 0) {
          *(volatile int*)&sm.stop = 1;
          mbar_arrive(&bar.kq_empty[c % STAGES]);
        }
        for (int f = c + 1; f < min(nch, c + 3); ++f) wait_bar(&bar.ops_full[f & 3], f >> 2, quit);      // copies in flight
        break;
      }
      if (elect_one()) umma_commit(&bar.kq_empty[c % STAGES]);
      __syncwarp();
      if (c + 3 < nch) fetch(c + 3);        // (over chunk c - 1, whose outputs the state's warps have stored)
    }
    // every product has been waited for by the state's warps, except where a wait ran out
    if (sm.quit) {
      const uint64_t t = globaltimer_ns();
      while (globaltimer_ns() - t < 1000000ull) {}
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 15) tmem_dealloc(tmem, 512);
}

// ---- first launch: 128 threads, a block per (chunk, key head, sequence)
struct PrepSmem {
  union {
    float k[C][KD + 4];                                      // rows of k;
    float L[2][C * (C + 4)];                                 // once the scores are there: L of two heads
  };
  float q[C][KD + 4], g[2 * C][C + 4];                       // rows of q; scores of both with the keys
  float kf[C], qf[C], ks[C], qs[C];                          // norm factors, scales
  float bad[2];
};
__global__ void __launch_bounds__(128, 5) delta_prep_kernel(DeltaArgs a) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
  const int b = blockIdx.z, hk = blockIdx.y, c = blockIdx.x;
  const int q0 = a.cu_q[b], ql = a.cu_q[b + 1] - q0, ctx = a.seq_lens[b] - ql, slot = a.slots[b];
  if (slot < 0 || ctx < 0 || ql < a.least || c * C >= ql) return;
  const int n = min(C, ql - c * C), dk = a.dk, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t0 = q0 + c * C;
  bool bad = false;
  {
    // eight lanes to a row, 16 rows of k or q at a time
    const int l8 = lane & 7;
    float4 x[4][4];
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = (it & 1) * 16 + warp * 4 + (lane >> 3);
      const float* p = (it < 2 ? a.k + (t0 + min(i, n - 1)) * a.ldk : a.q + (t0 + min(i, n - 1)) * a.ldq) + (int64_t)hk * dk;
#pragma unroll
      for (int m = 0; m < 4; ++m) x[it][m] = ld_nc4(p + min(m * 32 + l8 * 4, dk - 4));
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = (it & 1) * 16 + warp * 4 + (lane >> 3);
      float sum = 0.f, mx = 0.f;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float4& y = x[it][m];
        if (i >= n || m * 32 + l8 * 4 >= dk) y = make_float4(0.f, 0.f, 0.f, 0.f);
        sum = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, sum))));
        mx = max_abs(max_abs(mx, y.x, y.y), y.z, y.w);
        *reinterpret_cast<float4*>((it < 2 ? sm.k[i] : sm.q[i]) + m * 32 + l8 * 4) = y;
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        mx = max_abs(mx, __shfl_xor_sync(0xffffffffu, mx, o), 0.f);
      }
      const Scale s = scale_of(mx);
      const float f = (a.unit ? rsqrtf(sum + a.unit_eps) : 1.f) * (it < 2 ? 1.f : a.q_scale);
      bad |= i < n && (s.huge || !(fabsf(f) < 0x1p60f));
      if (l8 == 0) {
        (it < 2 ? sm.kf : sm.qf)[i] = f;
        (it < 2 ? sm.ks : sm.qs)[i] = i < n ? f * s.s : 0.f;
      }
    }
  }
  bad = __syncthreads_or(bad);
  int zeros = 0;
  {
    // scores: 4 rows x 4 keys per thread (rows r, r + 16, .. of [k; q], keys j, j + 8, ..), two sums a pair
    const int r = threadIdx.x >> 3, j = threadIdx.x & 7;
    pair_t acc[4][4], all[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) all[x][y] = 0;
#pragma unroll 1
    for (int e0 = 0; e0 < KD; e0 += 16) {          // (sums of 8 terms, then of 16 sums: with sums of 64 terms the outputs had 1.4e-7)
#pragma unroll
      for (int e = e0; e < e0 + 16; e += 4) {
        pair_t u[4][2], w[4][2];
#pragma unroll
        for (int x = 0; x < 4; ++x) lds_pairs((x < 2 ? sm.k[r + 16 * x] : sm.q[r + 16 * (x - 2)]) + e, u[x][0], u[x][1]);
#pragma unroll
        for (int y = 0; y < 4; ++y) lds_pairs(sm.k[j + 8 * y] + e, w[y][0], w[y][1]);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y)
            acc[x][y] = pfma(u[x][0], w[y][0], e == e0 ? pmul(u[x][1], w[y][1]) : pfma(u[x][1], w[y][1], acc[x][y]));
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) all[x][y] = padd(all[x][y], acc[x][y]);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const float2 s = unpack(all[x][y]);
        sm.g[r + 16 * x][j + 8 * y] = s.x + s.y;
        if (x < 2) zeros += s.x + s.y == 0.f && r + 16 * x < n && j + 8 * y < n;
      }
  }
  const bool sparse = __syncthreads_count(zeros >= 2) >= 32;        // scores of the keys with one another that are exactly 0
  // value heads of the key head, two at a time: even warps L and T, odd warps the outputs' weights; a token per lane
  const bool is_q = warp & 1;
  const int w2 = warp >> 1;
  for (int hh = w2; hh < a.rep; hh += 2) {
    const int h = hk * a.rep + hh;
    Prepared& out = reinterpret_cast<Prepared*>(a.prepared)[((int64_t)(q0 / C + b) + c) * a.H + h];
    const int64_t t = t0 + min(lane, n - 1);
    const float lg_raw = a.log_decay[t * a.ldg + h], be_raw = a.beta[t * a.ldb + h];
    const float lg = lane < n ? lg_raw : 0.f, be = lane < n ? (a.beta_sigmoid ? 1.f / (1.f + expf(-be_raw)) : be_raw) : 0.f;
    double G = (double)lg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, G, o);
      if (lane >= o) G += y;
    }
    const float ghi = (float)G, gl = (float)(G - (double)ghi), since = expf(ghi), rest = expf((float)(__shfl_sync(0xffffffffu, G, 31) - G));
    bool no = bad || __any_sync(0xffffffffu, !(lg <= 0.25f && lg >= -0x1p20f) || !(fabsf(be) < 0x1p60f));
    const int last = is_q ? lane : lane - 1;        // keys this row sees
    const float mine = is_q ? sm.qf[lane] : be * sm.kf[lane];
    float d[C], mx = 0.f;
    const float* row = sm.g[(is_q ? C : 0) + lane];
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const float w = expf((ghi - __shfl_sync(0xffffffffu, ghi, j)) + (gl - __shfl_sync(0xffffffffu, gl, j)));
      d[j] = j <= last ? (mine * sm.kf[j]) * row[j] * w : 0.f;
      mx = max_abs(mx, d[j], 0.f);
    }
    if (is_q) {
      const Scale s = scale_of(mx);
      no |= __any_sync(0xffffffffu, s.huge);
      out.sc.as[lane] = s.s;
      out.sc.gq[lane] = since * sm.qs[lane];
      uint8_t* to = out.tri + lane * 128;
#pragma unroll
      for (int j = 0; j < C; j += 8) {
        uint32_t hi[4], lo[4], mi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3(pmul(pack(d[j + 2 * e], d[j + 2 * e + 1]), both(s.inv)), hi[e], lo[e], mi[e]);
        uint8_t* at = to + (((4 + (j >> 3)) ^ (lane & 7)) << 4);
        *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(at + TRI) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(at + 2 * TRI) = make_uint4(mi[0], mi[1], mi[2], mi[3]);
      }
      if (lane == 0) sm.bad[w2] = no ? 1.f : 0.f;
    } else {
      const float ks = sm.ks[lane], end = rest * ks;
      float most = end;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most = max_abs(most, __shfl_xor_sync(0xffffffffu, most, o), 0.f);
      const Scale s = scale_of(most);
      no |= s.huge;
      out.sc.be[lane] = be;
      out.sc.bk[lane] = be * ks * since;
      out.sc.decay[lane] = sparse ? 0.f : expf(lg);
      out.sc.gend[lane] = end * s.inv * 0x1p-12f;
      float low = since;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
      if (lane == 31) {
        out.sc.low = sparse ? -1.f : low;
        out.sc.all = since;
        out.sc.most = s.s * 0x1p12f;
      }
      float* L = sm.L[w2];
#pragma unroll
      for (int j = 0; j < C; j += 4) *reinterpret_cast<float4*>(L + lane * (C + 4) + j) = make_float4(d[j], d[j + 1], d[j + 2], d[j + 3]);
      __syncwarp();
      // T: lane j solves for column j
#pragma unroll
      for (int i = 0; i < C; ++i) {
        float s0 = i == lane ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int m = 0; m < i; m += 4) {
          const float4 x = *reinterpret_cast<const float4*>(L + i * (C + 4) + m);
          const float y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (m + e < i) {
              if (e & 1) s1 = fmaf(-y[e], d[m + e], s1);
              else s0 = fmaf(-y[e], d[m + e], s0);
            }
        }
        d[i] = s0 + s1;
      }
      uint8_t* to = out.tri + ((lane & 7) << 1);
      mx = 0.f;
#pragma unroll
      for (int i = 0; i < C; i += 2) {
        mx = max_abs(mx, d[i], d[i + 1]);
        uint32_t hi, lo, mi;
        split3(pmul(pack(d[i], d[i + 1]), both(1.f / kTScale)), hi, lo, mi);
        uint8_t* p = to + i * 128 + (((lane >> 3) ^ (i & 7)) << 4);
        uint8_t* q = to + (i + 1) * 128 + (((lane >> 3) ^ ((i + 1) & 7)) << 4);
        *reinterpret_cast<uint16_t*>(p) = (uint16_t)hi;
        *reinterpret_cast<uint16_t*>(p + TRI) = (uint16_t)lo;
        *reinterpret_cast<uint16_t*>(p + 2 * TRI) = (uint16_t)mi;
        *reinterpret_cast<uint16_t*>(q) = (uint16_t)(hi >> 16);
        *reinterpret_cast<uint16_t*>(q + TRI) = (uint16_t)(lo >> 16);
        *reinterpret_cast<uint16_t*>(q + 2 * TRI) = (uint16_t)(mi >> 16);
      }
      no |= __any_sync(0xffffffffu, !(mx < 4.f));
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + w2) : "memory");       // (the pair of warps of this head)
    if (!is_q && lane == 0) out.sc.bad = no || sm.bad[w2] != 0.f;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + w2) : "memory");
  }
}

}  // namespace

// sequences of at least a.least tokens; the caller has checked the sizes (dk <= 128, multiple of 4, 16-byte rows)
int delta_chunk_launch(DeltaArgs a, int B, int max_q, cudaStream_t stream) {
  a.chunks = (max_q + C - 1) / C;
  static PerDeviceSmem granted, granted_prep;
  LLMSS_CHECK_CUDA(granted_prep.ensure(delta_prep_kernel, (int)sizeof(PrepSmem)));
  LLMSS_CHECK_CUDA(granted.ensure(delta_chunk_kernel, kSmemBytes));
  delta_prep_kernel<<<dim3(a.chunks, a.H / a.rep, B), 128, sizeof(PrepSmem), stream>>>(a);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  delta_chunk_kernel<<<dim3(B, a.H, (a.dv + VL - 1) / VL), kThreads, kSmemBytes, stream>>>(a);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}
