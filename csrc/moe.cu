// Routed mixture of experts: grouped top-k router and the per-token expert products.
//
//   moe_route : scores s = softmax(z) or sigmoid(z) over all E experts (32-bit); experts are chosen by s plus an optional
//               per-expert correction, weighted by s itself; the experts form `groups` equal groups of neighbours, a
//               group scores as its best expert (or as the sum of its few best), only experts of the `keep` best groups
//               are eligible; the `top` eligible experts with the largest choice scores are chosen; weights = s_chosen
//               (/ (sum + 1e-20) if renormalised) * route_scale.  Ties go to the lower index.  One warp per token.
//   moe_up    : a[t, k, :] = act(W_up[e_k] h_t)            one warp per output feature, weights read row-wise
//   moe_down  : y[t, :]    = sum_k w_k W_down[e_k] a[t, k] 32-bit output; the experts' down matrices lie side by side
//               in one [W, E * F] tensor (row stride ldd), which is also the dense form's GEMM operand
// The two expert kernels gather the chosen experts' weight rows per token: the form for decode and short
// portions, where every token touches its own few experts and the pass is bound by those weight bytes.
// Long prompts use the dense form instead (all experts through the tensor-core GEMM, unchosen ones weighted 0).
#include "common.cuh"

namespace {

constexpr int kMaxPerLane = 8;   // experts per lane: E <= 256

constexpr int kMaxGroupTop = 4;  // a group scores as the sum of at most this many of its best experts

// score_kind 0: s = softmax(z); 1: s = sigmoid(z).  Experts are chosen by c = s + correction (correction may be null); the
// weights are the chosen experts' s.  A group scores as the sum of its `group_top` largest c (1: its best expert).
// renorm: weights / (their sum + 1e-20).  Experts outside the kept groups are never chosen, whatever the sign of c.
// PL experts per lane: 32 * PL >= E
struct RouteArgs {
  int E, top, groups, keep;
  float route_scale;
  int score_kind;
  const float* correction;
  int group_top, renorm;
  int* ids; float* wts; float* dense;
};
// one warp routes token t from its logits zr; cs: 32 * PL numbers of shared memory for the warp
template <int PL>
__device__ __forceinline__ void route_token(const RouteArgs& a, const float* zr, int t, float* cs) {
  const int lane = threadIdx.x & 31;
  const int E = a.E, top = a.top, groups = a.groups, keep = a.keep, score_kind = a.score_kind, group_top = a.group_top, renorm = a.renorm;
  const float route_scale = a.route_scale;
  const float* correction = a.correction;
  int* ids = a.ids;
  float* wts = a.wts;
  float* dense = a.dense;
  float s[PL], c[PL];
  bool ok[PL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = lane + i * 32;
    s[i] = e < E ? zr[e] : -INFINITY;
    mx = fmaxf(mx, s[i]);
  }
  if (score_kind == 0) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      s[i] = e < E ? expf(s[i] - mx) : 0.f;
      sum += s[i];
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int i = 0; i < PL; ++i) s[i] /= sum;
  } else {
#pragma unroll
    for (int i = 0; i < PL; ++i) s[i] = lane + i * 32 < E ? 1.f / (1.f + expf(-s[i])) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = lane + i * 32;
    c[i] = e < E ? s[i] + (correction != nullptr ? correction[e] : 0.f) : -INFINITY;
    ok[i] = false;
    if (e < E) cs[e] = c[i];
  }
  __syncwarp();
  // group scores: lane l owns groups l, l + 32, ...
  const int gsz = E / groups;
  float gs[PL];
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int g = lane + j * 32;
    gs[j] = -INFINITY;
    if (g >= groups) continue;
    float best[kMaxGroupTop];
#pragma unroll
    for (int n = 0; n < kMaxGroupTop; ++n) best[n] = -INFINITY;
    for (int e = g * gsz; e < (g + 1) * gsz; ++e) {
      float v = cs[e];
#pragma unroll
      for (int n = 0; n < kMaxGroupTop; ++n)
        if (n < group_top && v > best[n]) { const float o = best[n]; best[n] = v; v = o; }
    }
    float sum = 0.f;
#pragma unroll
    for (int n = 0; n < kMaxGroupTop; ++n)
      if (n < group_top && n < gsz) sum += best[n];
    gs[j] = sum;
  }
  // best `keep` groups: repeatedly take the group with the largest score (ties: the lower group)
  unsigned long long taken_lo = 0ull, taken_hi = 0ull, taken_2 = 0ull, taken_3 = 0ull;   // up to 256 groups
  for (int n = 0; n < keep; ++n) {
    float bv = -INFINITY;
    int bg = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < PL; ++j) {
      const int g = lane + j * 32;
      if (g >= groups) continue;
      const unsigned long long word = g < 64 ? taken_lo : g < 128 ? taken_hi : g < 192 ? taken_2 : taken_3;
      if ((word >> (g & 63)) & 1ull) continue;
      if (gs[j] > bv || (gs[j] == bv && g < bg) || bg == 0x7fffffff) { bv = gs[j]; bg = g; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int og = __shfl_xor_sync(0xffffffffu, bg, o);
      if (og != 0x7fffffff && (bg == 0x7fffffff || ov > bv || (ov == bv && og < bg))) { bv = ov; bg = og; }
    }
    if (bg < 64) taken_lo |= 1ull << bg; else if (bg < 128) taken_hi |= 1ull << (bg - 64);
    else if (bg < 192) taken_2 |= 1ull << (bg - 128); else if (bg < 256) taken_3 |= 1ull << (bg - 192);
  }
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = lane + i * 32;
    if (e >= E) continue;
    const int g = e / gsz;
    const unsigned long long word = g < 64 ? taken_lo : g < 128 ? taken_hi : g < 192 ? taken_2 : taken_3;
    ok[i] = (word >> (g & 63)) & 1ull;
  }
  // top experts among the eligible ones, by choice score; the weight is the plain score
  float wsum = 0.f;
  float myw = 0.f;      // lane n keeps the n-th pick (top <= 32)
  int myid = 0;
  bool mine = false;
  for (int n = 0; n < top; ++n) {
    float bv = -INFINITY, bs = 0.f;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PL; ++i) {
      const int e = lane + i * 32;
      if (e < E && ok[i] && (be == 0x7fffffff || c[i] > bv || (c[i] == bv && e < be))) { bv = c[i]; be = e; bs = s[i]; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const float os = __shfl_xor_sync(0xffffffffu, bs, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (oe != 0x7fffffff && (be == 0x7fffffff || ov > bv || (ov == bv && oe < be))) { bv = ov; be = oe; bs = os; }
    }
    if (be < E) {
      if ((be & 31) == lane) ok[be >> 5] = false;
      wsum += bs;
      if (lane == n) { myw = bs; myid = be; mine = true; }
    } else if (lane == n) { myw = 0.f; myid = 0; }
  }
  const float inv = renorm ? route_scale / (wsum + 1e-20f) : route_scale;
  if (lane < top) {
    ids[(int64_t)t * top + lane] = myid;
    wts[(int64_t)t * top + lane] = myw * inv;
  }
  if (dense != nullptr) {   // [T, E] routing weights, 0 for experts that were not chosen
    for (int e = lane; e < E; e += 32) dense[(int64_t)t * E + e] = 0.f;
    __syncwarp();
    if (lane < top && mine) dense[(int64_t)t * E + myid] = myw * inv;
  }
}
template <int PL>
__global__ void __launch_bounds__(128) moe_route_kernel(RouteArgs a, const float* __restrict__ z, int64_t ldz, int T) {
  __shared__ float cs_all[4][32 * PL];
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t < T) route_token<PL>(a, z + (int64_t)t * ldz, t, cs_all[threadIdx.x >> 5]);
}

// Logits and routing in one launch, for up to 32 experts: a block has 16 tokens, its 16 warps every 16th piece of 32 channels and then a token each.  A
// product of 16 columns has no use for the tensor-memory tiles (128 features), and its result went through memory to a second launch; here the rows come
// straight into mma fragments.  The order of a sum over channels is free, so a thread's 16-byte pieces of a token's and an expert's row are two steps of
// k = 16 as they lie.  Two launches / one, us: 8192 tokens of 2048, 16 experts 28.7 / 20.7; 2048 of 4096, 32 experts 18.2 / 11.3; 400 of 2048, 16 experts
// 13.6 / 7.2 (with eight warps 20.8, 15.9, 11.2: a block is one chain of loads, sums and choices).  Up to 64 experts it lost (4096 of 4096: 54).
template <typename T, int NT>      // NT: tiles of 8 experts
__global__ void __launch_bounds__(512) moe_router_kernel(RouteArgs a, const T* __restrict__ h, int64_t ldh, const T* __restrict__ w, int64_t ldw,
                                                         const T* __restrict__ bias, int K, int T_) {
  constexpr int WARPS = 16, EP = NT * 8;
  __shared__ float part[WARPS][16][EP + 2];
  __shared__ float z[16][EP];
  __shared__ float cs[WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, l = lane & 3;
  const int t0 = blockIdx.x * 16;
  const T* r0 = h + (int64_t)min(t0 + g, T_ - 1) * ldh;
  const T* r1 = h + (int64_t)min(t0 + g + 8, T_ - 1) * ldh;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float c[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
#pragma unroll 4
  for (int k0 = warp * 32; k0 < K; k0 += WARPS * 32) {
    const int k = k0 + l * 8;
    const bool in = k < K;             // (K is a multiple of 8)
    const int kk = in ? k : 0;
    uint4 x0 = *reinterpret_cast<const uint4*>(r0 + kk), x1 = *reinterpret_cast<const uint4*>(r1 + kk), y[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) y[n] = *reinterpret_cast<const uint4*>(w + (int64_t)min(n * 8 + g, a.E - 1) * ldw + kk);
    if (!in) {                         // (both operands: zeros times what may be no number)
      x0 = x1 = zero;
#pragma unroll
      for (int n = 0; n < NT; ++n) y[n] = zero;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      mma_16816<T>(c[n], x0.x, x1.x, x0.y, x1.y, y[n].x, y[n].y);
      mma_16816<T>(c[n], x0.z, x1.z, x0.w, x1.w, y[n].z, y[n].w);
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][g + (e >> 1) * 8][n * 8 + 2 * l + (e & 1)] = c[n][e];
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * EP; i += WARPS * 32) {
    const int t = i / EP, e = i % EP;
    float s = 0.f;
#pragma unroll
    for (int x = 0; x < WARPS; ++x) s += part[x][t][e];
    z[t][e] = s + (bias != nullptr && e < a.E ? to_f32(bias[e]) : 0.f);
  }
  __syncthreads();
  if (t0 + warp < T_) route_token<1>(a, z[warp], t0 + warp, cs[warp]);
}

// grid (T, top, ceil(F / 8)); 8 warps, one output feature each
template <typename T>
__global__ void __launch_bounds__(256) moe_up_kernel(const T* __restrict__ h, int64_t ldh, const int* __restrict__ ids,
                                                     const T* __restrict__ w_up, T* __restrict__ act_out, int W, int F,
                                                     int top, int act, int gated) {
  extern __shared__ float hs[];
  const int64_t t = blockIdx.x;
  const int k = blockIdx.y;
  for (int c = threadIdx.x; c < W; c += 256) hs[c] = to_f32(h[t * ldh + c]);
  __syncthreads();
  const int f = blockIdx.z * 8 + (threadIdx.x >> 5);
  if (f >= F) return;
  const int lane = threadIdx.x & 31;
  const int e = ids[t * top + k];
  if (gated) {   // rows interleave (gate_f, up_f): hidden = act(gate) * up
    const T* wg = w_up + ((int64_t)e * 2 * F + 2 * f) * W;
    const T* wu = wg + W;
    float g = 0.f, u = 0.f;
    for (int c = lane; c < W; c += 32) { g = fmaf(to_f32(wg[c]), hs[c], g); u = fmaf(to_f32(wu[c]), hs[c], u); }
    g = warp_sum(g); u = warp_sum(u);
    if (lane == 0) act_out[(t * top + k) * F + f] = from_f32<T>(act_exact(g, act) * u);
    return;
  }
  const T* wr = w_up + ((int64_t)e * F + f) * W;
  float s = 0.f;
  for (int c = lane; c < W; c += 32) s = fmaf(to_f32(wr[c]), hs[c], s);
  s = warp_sum(s);
  if (lane == 0) act_out[(t * top + k) * F + f] = from_f32<T>(act_apply(s, act));
}

// grid (T, ceil(W / 8)); 8 warps, one output feature each, summed over the chosen experts in 32-bit
template <typename T>
__global__ void __launch_bounds__(256) moe_down_kernel(const T* __restrict__ act_in, const int* __restrict__ ids,
                                                       const float* __restrict__ wts, const T* __restrict__ w_down, int64_t ldd,
                                                       float* __restrict__ out, int64_t ldo, int W, int F, int top, int add) {
  extern __shared__ float as[];   // [top][F]
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x; c < top * F; c += 256) as[c] = to_f32(act_in[t * top * F + c]);
  __syncthreads();
  const int n = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (n >= W) return;
  const int lane = threadIdx.x & 31;
  float y = 0.f;
  for (int k = 0; k < top; ++k) {
    const int e = ids[t * top + k];
    const T* wr = w_down + (int64_t)n * ldd + (int64_t)e * F;   // row n of expert e inside [W, E * F]
    float s = 0.f;
    for (int c = lane; c < F; c += 32) s = fmaf(to_f32(wr[c]), as[k * F + c], s);
    y += wts[t * top + k] * warp_sum(s);
  }
  if (lane == 0) out[t * ldo + n] = add ? out[t * ldo + n] + y : y;
}

// a[t, e * F + f] *= dense[t, e]   (dense form: weight each expert's block before the shared down projection)
template <typename T>
__global__ void __launch_bounds__(256) moe_scale_kernel(T* __restrict__ a, int64_t lda, const float* __restrict__ dense, int E,
                                                        int F) {
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x; c < E * F; c += 256) {
    const float w = dense[t * E + c / F];
    a[t * lda + c] = from_f32<T>(to_f32(a[t * lda + c]) * w);
  }
}

// the same for 16-bit rows of whole 16-byte pieces (F a multiple of 8): grid (T, pieces / 256), a piece per thread; the pieces of
// unchosen experts are stored as zeros without being read
template <typename T>
__global__ void __launch_bounds__(256) moe_scale_vec_kernel(T* __restrict__ a, int64_t lda, const float* __restrict__ dense, int E, int F) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t t = blockIdx.x;
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (c >= E * F) return;
  const float w = dense[t * E + c / F];
  uint4* p = reinterpret_cast<uint4*>(a + t * lda + c);
  if (w == 0.f) {
    *p = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  float v[8];
  unpack8<T>(*p, v);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] *= w;
  *p = pack8<T>(v);
}


// ---- grouped form for long prompts: (token, chosen expert) pairs sorted by expert, so that every expert multiplies one
// contiguous block of rows.  count -> (host: offsets) -> permute (ordered compaction, one CTA per expert: the order inside an
// expert's block is the pair order, so the result does not depend on scheduling) -> gather rows -> per-expert GEMMs ->
// combine (sum over a token's experts in its own order, 32-bit).
__global__ void __launch_bounds__(256) moe_count_kernel(const int* __restrict__ ids, int P, int* __restrict__ counts) {
  __shared__ int red[8];
  const int e = blockIdx.x;
  int c = 0;
  for (int p = threadIdx.x; p < P; p += 256) c += (ids[p] == e);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < 8; ++i) t += red[i];
    counts[e] = t;
  }
}

__global__ void __launch_bounds__(256) moe_permute_kernel(const int* __restrict__ ids, int P, const int* __restrict__ offsets,
                                                          int* __restrict__ perm, int* __restrict__ inv) {
  __shared__ int wsum[8];
  __shared__ int running;
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) running = offsets[e];
  __syncthreads();
  for (int p0 = 0; p0 < P; p0 += 256) {
    const int p = p0 + threadIdx.x;
    const bool mine = p < P && ids[p] == e;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) wsum[warp] = __popc(m);
    __syncthreads();
    int before = running;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    if (mine) {
      const int pos = before + __popc(m & ((1u << lane) - 1u));
      perm[pos] = p;
      inv[p] = pos;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < 8; ++w) t += wsum[w];
      running += t;
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(256) moe_gather_rows_kernel(const T* __restrict__ h, int64_t ldh, const int* __restrict__ perm,
                                                              int top, T* __restrict__ xs, int W) {
  const int64_t i = blockIdx.x;
  const T* src = h + (int64_t)(perm[i] / top) * ldh;
  for (int c = threadIdx.x; c < W; c += 256) xs[i * W + c] = src[c];
}

__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ inv,
                                                          const float* __restrict__ wts, float* __restrict__ out, int64_t ldo,
                                                          int W, int top, int add) {
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x; c < W; c += 256) {
    float v = 0.f;
    for (int k = 0; k < top; ++k) v += wts[t * top + k] * y[(int64_t)inv[t * top + k] * W + c];
    out[t * ldo + c] = add ? out[t * ldo + c] + v : v;
  }
}

// ---- the same sorting without the host: per-block expert counts, then every block derives its own offsets from all counts and
// places its pairs in pair order (the result does not depend on scheduling).  The table is what llmss_gemm_grouped reads.
constexpr int PAIRS = 1024;      // pairs per block

__global__ void __launch_bounds__(256) moe_hist_kernel(const int* __restrict__ ids, int P, int E, int* __restrict__ hist) {
  __shared__ int c[256];
  c[threadIdx.x] = 0;
  __syncthreads();
  const int p0 = blockIdx.x * PAIRS;
  for (int p = p0 + threadIdx.x; p < min(P, p0 + PAIRS); p += 256) atomicAdd(&c[ids[p]], 1);
  __syncthreads();
  if (threadIdx.x < E) hist[blockIdx.x * E + threadIdx.x] = c[threadIdx.x];
}

// exclusive sum over the block's 256 threads
__device__ __forceinline__ int block_exclusive(int v, int* warps, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();
  if (lane == 31) warps[w] = incl;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    before += i < w ? warps[i] : 0;
    all += warps[i];
  }
  *total = all;
  return before + incl - v;
}

__global__ void __launch_bounds__(256) moe_place_kernel(const int* __restrict__ ids, int P, int E, const int* __restrict__ hist,
                                                        int* __restrict__ table, int* __restrict__ inv, int tile_rows) {
  __shared__ int warps[8];
  __shared__ int next[256];          // next free row of every expert for this block's pairs
  __shared__ int wcount[8][256];     // a round's pairs per warp and expert
  const int e = threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int all = 0, mine = 0;
  if (e < E) {
#pragma unroll 4
    for (int b = 0; b < (int)gridDim.x; ++b) {
      const int v = hist[b * E + e];
      all += v;
      mine += b < (int)blockIdx.x ? v : 0;
    }
  }
  int total, tiles;
  const int first = block_exclusive(all, warps, &total);
  const int tile0 = block_exclusive((all + tile_rows - 1) / tile_rows, warps, &tiles);
  if (blockIdx.x == 0) {
    if (e < E) { table[e] = first; table[E + 1 + e] = tile0; }
    if (e == 0) { table[E] = total; table[2 * E + 1] = tiles; }
  }
  next[e] = first + mine;
  for (int r = 0; r < PAIRS / 256; ++r) {
    const int p = blockIdx.x * PAIRS + r * 256 + threadIdx.x;
    const int id = p < P ? ids[p] : -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) wcount[i][e] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, id);
    if (id >= 0 && lane == __ffs(same) - 1) wcount[w][id] = __popc(same);
    __syncthreads();
    if (id >= 0) {
      int pos = next[id] + __popc(same & ((1u << lane) - 1u));
      for (int i = 0; i < w; ++i) pos += wcount[i][id];
      inv[p] = pos;
    }
    __syncthreads();
    int add = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) add += wcount[i][e];
    next[e] += add;
  }
}

// every token's row to its places in the sorted order: one read, `top` writes.  V: uint4 (rows of whole 16-byte pieces) or T
template <typename V>
__global__ void __launch_bounds__(128) moe_scatter_rows_kernel(const V* __restrict__ h, int64_t ldh, const int* __restrict__ inv, int top,
                                                               V* __restrict__ xs, int n) {
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x; c < n; c += 128) {
    const V v = h[t * ldh + c];
    for (int k = 0; k < top; ++k) xs[(int64_t)inv[t * top + k] * n + c] = v;
  }
}

// moe_combine_kernel on rows of whole 16-byte vectors
__global__ void __launch_bounds__(256) moe_combine4_kernel(const float* __restrict__ y, const int* __restrict__ inv,
                                                           const float* __restrict__ wts, float* __restrict__ out, int64_t ldo, int W,
                                                           int top, int add) {
  const int64_t t = blockIdx.x;
  for (int c = threadIdx.x * 4; c < W; c += 1024) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
      const float w = wts[t * top + k];
      const float4 x = *reinterpret_cast<const float4*>(y + (int64_t)inv[t * top + k] * W + c);
      v.x += w * x.x; v.y += w * x.y; v.z += w * x.z; v.w += w * x.w;
    }
    float4* o = reinterpret_cast<float4*>(out + t * ldo + c);
    if (add) {
      const float4 b = *o;
      v = make_float4(b.x + v.x, b.y + v.y, b.z + v.z, b.w + v.w);
    }
    *o = v;
  }
}

template <typename T>
int launch_experts(const void* h, int64_t ldh, const int* ids, const float* wts, const void* w_up, const void* w_down,
                   int64_t ldd, void* act_scratch, float* out, int64_t ldo, int T_, int W, int F, int top, int act, int gated, int add,
                   cudaStream_t stream) {
  const size_t sm_up = (size_t)W * 4, sm_dn = (size_t)top * F * 4;
  static PerDeviceSmem g1, g2;
  LLMSS_CHECK_CUDA(g1.ensure(moe_up_kernel<T>, (int)sm_up));
  LLMSS_CHECK_CUDA(g2.ensure(moe_down_kernel<T>, (int)sm_dn));
  moe_up_kernel<T><<<dim3(T_, top, (F + 7) / 8), 256, sm_up, stream>>>((const T*)h, ldh, ids, (const T*)w_up, (T*)act_scratch, W, F, top, act, gated);
  moe_down_kernel<T><<<dim3(T_, (W + 7) / 8), 256, sm_dn, stream>>>((const T*)act_scratch, ids, wts, (const T*)w_down, ldd, out, ldo, W, F, top, add);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace

LLMSS_API int llmss_moe_route_ex(const float* z, int64_t ldz, int T_, int E, int top, int groups, int keep, float route_scale,
                                 int score_kind, const float* correction, int group_top, int renorm, int* ids, float* wts,
                                 float* dense, cudaStream_t stream) {
  LLMSS_REQUIRE(E > 0 && E <= 32 * kMaxPerLane, "moe_route: %d experts (at most %d)", E, 32 * kMaxPerLane);
  LLMSS_REQUIRE(top > 0 && top <= 32 && top <= E, "moe_route: top=%d must be in 1..min(32, experts)", top);
  LLMSS_REQUIRE(groups > 0 && E % groups == 0 && keep > 0 && keep <= groups, "moe_route: bad groups %d / keep %d for %d experts",
                groups, keep, E);
  LLMSS_REQUIRE(score_kind == 0 || score_kind == 1, "moe_route: score kind %d (0 softmax, 1 sigmoid)", score_kind);
  LLMSS_REQUIRE(group_top >= 1 && group_top <= kMaxGroupTop, "moe_route: a group sums its %d best (1..%d)", group_top, kMaxGroupTop);
  if (T_ == 0) return 0;
  const RouteArgs a{E, top, groups, keep, route_scale, score_kind, correction, group_top, renorm, ids, wts, dense};
#define LLMSS_ROUTE(PL) \
  moe_route_kernel<PL><<<(T_ + 3) / 4, 128, 0, stream>>>(a, z, ldz, T_)
  if (E <= 32) LLMSS_ROUTE(1);
  else if (E <= 64) LLMSS_ROUTE(2);
  else if (E <= 128) LLMSS_ROUTE(4);
  else LLMSS_ROUTE(kMaxPerLane);
#undef LLMSS_ROUTE
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// Router logits (h [T, K] times w [E, K]^T, plus bias) and routing in one launch: 16-bit operands on 16-byte lines, K, ldh and ldw multiples of 8, E <= 32
LLMSS_API int llmss_moe_router(const void* h, int64_t ldh, const void* w, int64_t ldw, const void* bias, int K, int T_, int E, int top, int groups,
                               int keep, float route_scale, int score_kind, const float* correction, int group_top, int renorm, int* ids, float* wts,
                               float* dense, int dtype, cudaStream_t stream) {
  LLMSS_REQUIRE(E > 0 && E <= 32 && K > 0 && K % 8 == 0 && ldh % 8 == 0 && ldw % 8 == 0 && (((uintptr_t)h | (uintptr_t)w) & 15) == 0,
                "moe_router: %d experts (at most 32), width %d (a multiple of 8, rows on 16-byte lines)", E, K);
  LLMSS_REQUIRE(dtype == LLMSS_F16 || dtype == LLMSS_BF16, "moe_router: dtype must be f16/bf16");
  LLMSS_REQUIRE(top > 0 && top <= 32 && top <= E, "moe_router: top=%d must be in 1..min(32, experts)", top);
  LLMSS_REQUIRE(groups > 0 && E % groups == 0 && keep > 0 && keep <= groups, "moe_router: bad groups %d / keep %d for %d experts", groups, keep, E);
  LLMSS_REQUIRE((score_kind == 0 || score_kind == 1) && group_top >= 1 && group_top <= kMaxGroupTop, "moe_router: score kind %d, group top %d", score_kind, group_top);
  if (T_ <= 0) return 0;
  const RouteArgs a{E, top, groups, keep, route_scale, score_kind, correction, group_top, renorm, ids, wts, dense};
#define LLMSS_ROUTER(T, NT) \
  moe_router_kernel<T, NT><<<(T_ + 15) / 16, 512, 0, stream>>>(a, (const T*)h, ldh, (const T*)w, ldw, (const T*)bias, K, T_)
#define LLMSS_ROUTER_E(T)                  \
  if (E <= 16) LLMSS_ROUTER(T, 2);         \
  else LLMSS_ROUTER(T, 4)
  if (dtype == LLMSS_F16) { LLMSS_ROUTER_E(__half); }
  else { LLMSS_ROUTER_E(__nv_bfloat16); }
#undef LLMSS_ROUTER_E
#undef LLMSS_ROUTER
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

LLMSS_API int llmss_moe_route(const float* z, int64_t ldz, int T_, int E, int top, int groups, int keep, float route_scale,
                              int* ids, float* wts, float* dense, cudaStream_t stream) {
  return llmss_moe_route_ex(z, ldz, T_, E, top, groups, keep, route_scale, 0, nullptr, 1, 1, ids, wts, dense, stream);
}

// add = 1: the weighted sum of the chosen experts is added to out, else it replaces it
LLMSS_API int llmss_moe_experts_ex(const void* h, int64_t ldh, const int* ids, const float* wts, const void* w_up,
                                   const void* w_down, int64_t ldd, void* act_scratch, float* out, int64_t ldo, int T_, int W, int F,
                                   int top, int act, int gated, int add, int dtype, cudaStream_t stream) {
  LLMSS_REQUIRE(T_ <= 0x7fffffff / 1 && top <= 65535 && (F + 7) / 8 <= 65535 && (W + 7) / 8 <= 65535, "moe_experts: grid too large");
  LLMSS_REQUIRE((size_t)W * 4 <= 200 * 1024 && (size_t)top * F * 4 <= 200 * 1024, "moe_experts: width %d / top * ff %d exceed shared memory", W, top * F);
  if (T_ == 0) return 0;
  LLMSS_BY_DTYPE(dtype, return (launch_experts<T>(h, ldh, ids, wts, w_up, w_down, ldd, act_scratch, out, ldo, T_, W, F, top, act, gated, add, stream)));
}

LLMSS_API int llmss_moe_experts(const void* h, int64_t ldh, const int* ids, const float* wts, const void* w_up,
                                const void* w_down, int64_t ldd, void* act_scratch, float* out, int64_t ldo, int T_, int W, int F, int top,
                                int act, int gated, int dtype, cudaStream_t stream) {
  return llmss_moe_experts_ex(h, ldh, ids, wts, w_up, w_down, ldd, act_scratch, out, ldo, T_, W, F, top, act, gated, 0, dtype, stream);
}

LLMSS_API int llmss_moe_scale(void* a, int64_t lda, const float* dense, int T_, int E, int F, int dtype, cudaStream_t stream) {
  if (T_ == 0) return 0;
  const int64_t pieces = (int64_t)E * F / 8;
  if (dtype != LLMSS_F32 && F % 8 == 0 && lda % 8 == 0 && ((uintptr_t)a) % 16 == 0 && (pieces + 255) / 256 <= 65535) {
    const dim3 grid(T_, (unsigned)((pieces + 255) / 256));
    if (dtype == LLMSS_F16) LLMSS_CHECK_CUDA(launch_pdl(moe_scale_vec_kernel<__half>, grid, dim3(256), 0, stream, (__half*)a, lda, dense, E, F));
    else LLMSS_CHECK_CUDA(launch_pdl(moe_scale_vec_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, (__nv_bfloat16*)a, lda, dense, E, F));
    return 0;
  }
  LLMSS_BY_DTYPE(dtype, (moe_scale_kernel<T><<<T_, 256, 0, stream>>>((T*)a, lda, dense, E, F)));
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

LLMSS_API int llmss_moe_count(const int* ids, int P, int E, int* counts, cudaStream_t stream) {
  if (E <= 0) return 0;
  moe_count_kernel<<<E, 256, 0, stream>>>(ids, P, counts);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// offsets[e] = first row of expert e's block; perm[row] = pair index (token * top + k); inv[pair] = row
LLMSS_API int llmss_moe_permute(const int* ids, int P, int E, const int* offsets, int* perm, int* inv, cudaStream_t stream) {
  if (E <= 0 || P <= 0) return 0;
  moe_permute_kernel<<<E, 256, 0, stream>>>(ids, P, offsets, perm, inv);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

LLMSS_API int llmss_moe_gather_rows(const void* h, int64_t ldh, const int* perm, int top, void* xs, int P, int W, int dtype,
                                    cudaStream_t stream) {
  if (P <= 0) return 0;
  LLMSS_BY_DTYPE(dtype, (moe_gather_rows_kernel<T><<<P, 256, 0, stream>>>((const T*)h, ldh, perm, top, (T*)xs, W)));
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// add = 1: added to out, else out is replaced
LLMSS_API int llmss_moe_combine_ex(const float* y, const int* inv, const float* wts, float* out, int64_t ldo, int T_, int W, int top,
                                   int add, cudaStream_t stream) {
  if (T_ <= 0) return 0;
  if (W % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)y | (uintptr_t)out) & 15) == 0) {
    moe_combine4_kernel<<<T_, 256, 0, stream>>>(y, inv, wts, out, ldo, W, top, add);
    LLMSS_CHECK_CUDA(cudaGetLastError());
    return 0;
  }
  moe_combine_kernel<<<T_, 256, 0, stream>>>(y, inv, wts, out, ldo, W, top, add);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}

LLMSS_API int llmss_moe_combine(const float* y, const int* inv, const float* wts, float* out, int64_t ldo, int T_, int W, int top,
                                cudaStream_t stream) {
  return llmss_moe_combine_ex(y, inv, wts, out, ldo, T_, W, top, 0, stream);
}

// Sorts the P = T * top (token, expert) pairs by expert on the device.  inv[pair] = row in the sorted order; table [2 * (E + 1)]:
// first row of every expert (and P), first token tile (of tile_rows rows; llmss_moe_group: of 256) of every expert (and their number); hist: scratch of
// ceil(P / 1024) * E numbers.
LLMSS_API int llmss_moe_group_tiles(const int* ids, int P, int E, int* hist, int* table, int* inv, int tile_rows, cudaStream_t stream) {
  LLMSS_REQUIRE(tile_rows > 0 && P > 0 && E > 0 && E <= 256, "moe_group: %d pairs, %d experts (at most 256)", P, E);
  const int blocks = (P + PAIRS - 1) / PAIRS;
  moe_hist_kernel<<<blocks, 256, 0, stream>>>(ids, P, E, hist);
  moe_place_kernel<<<blocks, 256, 0, stream>>>(ids, P, E, hist, table, inv, tile_rows);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}
LLMSS_API int llmss_moe_group(const int* ids, int P, int E, int* hist, int* table, int* inv, cudaStream_t stream) {
  return llmss_moe_group_tiles(ids, P, E, hist, table, inv, 256, stream);
}

// xs[inv[t * top + k]] = h[t] for every token and choice; h, xs 16-bit
LLMSS_API int llmss_moe_scatter_rows(const void* h, int64_t ldh, const int* inv, int top, void* xs, int T_, int W, cudaStream_t stream) {
  if (T_ <= 0) return 0;
  if (W % 8 == 0 && ldh % 8 == 0 && (((uintptr_t)h | (uintptr_t)xs) & 15) == 0)
    moe_scatter_rows_kernel<uint4><<<T_, 128, 0, stream>>>((const uint4*)h, ldh / 8, inv, top, (uint4*)xs, W / 8);
  else
    moe_scatter_rows_kernel<uint16_t><<<T_, 128, 0, stream>>>((const uint16_t*)h, ldh, inv, top, (uint16_t*)xs, W);
  LLMSS_CHECK_CUDA(cudaGetLastError());
  return 0;
}
