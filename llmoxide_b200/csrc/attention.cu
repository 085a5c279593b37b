// Attention over the paged cache, general form: any number of heads and
// groups, any head size up to 256, a window or none, whole prompts and single
// tokens alike.  Two kernels: attention_f32_kernel (tiles of keys) for float32
// without pooled blocks and with sizes that are multiples of 4, and
// attention_paged_kernel for everything else: the bfloat16 path's sizes that
// the tiled kernels of other files refuse, pooled blocks, odd sizes.
//
// For the query at position p of head hq (crates/model/src/qwen35/cpu.rs:325-355):
// kv head g = hq / (H/G); keys first..p are visible, first = 0 or p-(w-1) under
// a window (crates/model/src/cache.rs:31-37); s_j = (q . k_j) * scale; softmax
// with the maximum subtracted; out = sum_j w_j v_j.  All of it in float32.
// With `keep_first` > 0 the keys 0..keep_first-1 stay visible under the window
// as well (they are taken first, then the window's keys).  Values may have a
// size Dv of their own; a query row may sit in a wider row (q_stride elements
// from token to token), e.g. the q|k|v row of a fused product.  With `sink` > 0
// the softmax's denominator has that much added: w_j = exp(s_j) / (sink + sum exp(s_j)).
// With `chunk` > 0 positions are cut into chunks of that many, counted from the sequence's position 0, and a
// query sees only the keys of its own chunk: first = p - p % chunk (beside a window, the later of the two).
//
// With `pool` > 0 every block of `pool` positions that lies wholly before the window (block b = positions
// b*pool .. b*pool+pool-1, seen from p when b*pool+pool-1 <= p - window) is seen as one key and one value: row b of
// a second store (pool_k, pool_v, with a block table of its own), taken first, in the same softmax.
// With `gate` a head's output is multiplied by sigmoid(gate[t * gate_stride + hq]).
// With `softcap` c > 0 a scaled score s becomes c * tanh(s / c) before the softmax.  With `sinks` (float32 [H]) the
// denominator of head hq has exp(sinks[hq]) added: a learned score without key and value, neither scaled nor capped.
// With `score_bias` (float32 [H, bias_len]) the scaled score of the key at j has score_bias[hq, min(p - j, bias_len - 1)]
// added: a learned number per distance and head (not beside pooled blocks or a cap).
//
// attention_paged_kernel: one warp per (token, head).  Keys are taken 32 at a time starting at the
// range's first key: lane j scores key lo + c*32 + j with a sequential dot over
// D, the chunk's maximum and sum update a running softmax, and the lanes then
// own dims (lane, lane+32, ...) of the output and add the chunk's values key
// by key.  Chunk boundaries depend on (keep_first, first, p) only, so a
// position's result does not depend on how tokens were cut into steps or batched.
#include "common.cuh"

#define ATT_WARPS 4
#define ATT_MAX_D 256

template <typename TA, typename TC>
__global__ void attention_paged_kernel(const TA* __restrict__ q, TA* __restrict__ out,
                                       const TC* __restrict__ k_cache_w, const TC* __restrict__ v_cache_w,
                                       const int* __restrict__ block_table, int table_width,
                                       const int* __restrict__ token_seq, const int* __restrict__ token_pos,
                                       int H, int G, int D, int Dv, size_t q_stride, int window, int keep_first,
                                       float scale, float sink, int chunk, int pool,
                                       const TC* __restrict__ pool_k, const TC* __restrict__ pool_v,
                                       const int* __restrict__ pool_table, const float* __restrict__ gate,
                                       size_t gate_stride, float softcap, const float* __restrict__ sinks,
                                       const float* __restrict__ score_bias, int bias_len) {
  extern __shared__ float q_buf[];  // [ATT_WARPS][D]
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x;                        // tokens on x: a step may bring more than 65535
  const int hq = blockIdx.y * ATT_WARPS + warp;
  if (hq >= H) return;
  const int g = hq / (H / G);
  const int p = token_pos[t];
  int first = (window > 0 && p - (window - 1) > 0) ? p - (window - 1) : 0;
  if (chunk > 0) first = max(first, p - p % chunk);
  const int* pages = block_table + (size_t)token_seq[t] * table_width;     // (re-pointed per range below)

  float* qs = q_buf + warp * D;
  const TA* qrow = q + (size_t)t * q_stride + (size_t)hq * D;
  for (int i = lane; i < D; i += 32) qs[i] = to_f32(qrow[i]);
  __syncwarp();

  constexpr int MAX_OWN = ATT_MAX_D / 32;
  float acc[MAX_OWN];
#pragma unroll
  for (int i = 0; i < MAX_OWN; ++i) acc[i] = 0.f;
  float m = -INFINITY, l = 0.f;

  // two ranges of keys: the kept first ones that lie before the window (or the pooled blocks that do, out of their
  // own store), then the window up to p
  int n_kept = keep_first < first ? keep_first : first;
  if (pool > 0) n_kept = p - window + 1 >= pool ? (p - window + 1) / pool : 0;
  const int* pages_w = pages;
  const int* pages_0 = pool > 0 ? pool_table + (size_t)token_seq[t] * table_width : pages;
  const TC* kc0 = pool > 0 ? pool_k : k_cache_w;
  const TC* vc0 = pool > 0 ? pool_v : v_cache_w;
  for (int range = n_kept > 0 ? 0 : 1; range < 2; ++range) {
  const int lo = range ? first : 0, last = range ? p : n_kept - 1;
  const TC* k_cache = range ? k_cache_w : kc0;
  const TC* v_cache = range ? v_cache_w : vc0;
  pages = range ? pages_w : pages_0;
  for (int base = lo; base <= last; base += 32) {
    const int j = base + lane;
    const bool live = j <= last;
    float s = -INFINITY;
    if (live) {
      const TC* krow = k_cache + cache_row_offset(pages[j / LLMX_PAGE], g, j % LLMX_PAGE, G, D);
      float dot = 0.f;
      for (int i = 0; i < D; ++i) dot += qs[i] * to_f32(krow[i]);
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      if (score_bias) s += score_bias[(size_t)hq * bias_len + min(p - j, bias_len - 1)];
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float corr = expf(m - m_new);  // exp(-inf) = 0 on the first chunk; lane 0 of a chunk is always live
    const float e = live ? expf(s - m_new) : 0.f;
    l = l * corr + warp_sum(e);
#pragma unroll
    for (int i = 0; i < MAX_OWN; ++i) acc[i] *= corr;
    const int n_live = (last - base + 1) < 32 ? (last - base + 1) : 32;
    for (int jj = 0; jj < n_live; ++jj) {
      const float w = __shfl_sync(0xffffffffu, e, jj);
      const int key = base + jj;
      const TC* vrow = v_cache + cache_row_offset(pages[key / LLMX_PAGE], g, key % LLMX_PAGE, G, Dv);
#pragma unroll
      for (int i = 0; i < MAX_OWN; ++i) {
        const int dim = lane + 32 * i;
        if (dim < Dv) acc[i] += w * to_f32(vrow[dim]);
      }
    }
    m = m_new;
  }
  }
  // a sink: `sink` keys of score 0 that have no value; they only add to the denominator
  if (sink > 0.f) l += sink * expf(-m);
  if (sinks) l += expf(sinks[hq] - m);
  float inv = 1.0f / l;
  if (gate) inv *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + hq]));
  TA* orow = out + ((size_t)t * H + hq) * Dv;
#pragma unroll
  for (int i = 0; i < MAX_OWN; ++i) {
    const int dim = lane + 32 * i;
    if (dim < Dv) orow[dim] = from_f32<TA>(acc[i] * inv);
  }
}

// ---------------------------------------------------------------------------
// The same in float32, by tiles.  The kernel above takes a warp per (token, head), reads every key row once per head and
// query, and follows one chain of loads; this one shares a tile of 64 keys (one page) among the query rows of a CTA.
//
// A query row's keys are cut at multiples of 64 positions.  Within a tile: scores from two chains over the even and the
// odd dims (packed multiply-adds), the tile's maximum, exponentials against it, their sum (four keys a lane, then a
// butterfly over 16 lanes) and the weighted values key by key.  The tiles' (maximum, sum, values) then join a running
// state in the order of the tiles.  That order depends on the query's position and mask alone, and both forms below
// follow it step by step, so a position's result does not depend on how tokens were cut into steps or batched.
//   SPLIT false   a CTA owns 8 TR query rows (tokens of one sequence x the heads that share a kv head) and walks the tiles
//   SPLIT true    a cluster of 8 CTAs owns 8 such rows; CTA r takes tiles r, r + 8, ..., and after every round of 8 tiles
//                 each CTA joins a slice of the dims out of the eight partial results
// A key that a row must not see is left out, not multiplied by zero (its value may be anything).
// A few tokens are bound by the latency of a round of tiles (copy, scores, values, join, one after the other), prompts by
// the shared-memory reads; measurements at the rule below.
// ---------------------------------------------------------------------------
#define AF_KEYS 64             // keys per tile = LLMX_PAGE
#define AF_THREADS 128         // 8 (rows) x 16 (keys, then dims)
#define AF_SPLIT 8             // CTAs of a cluster
static_assert(AF_KEYS == LLMX_PAGE, "a tile is a page");

struct AfArgs {
  const float *q, *k_cache, *v_cache, *gate, *sinks, *score_bias;
  float* out;
  const int *block_table, *token_seq, *token_pos, *seq_start;
  size_t q_stride, gate_stride;
  int n_seqs;
  int table_width, n_tokens, H, G, D, Dv, window, keep_first, chunk, bias_len;
  int heads_per_cta, tokens_per_cta, head_blocks;
  bool q_vec;                    // rows of q are whole 16-byte pieces
  float scale, sink, softcap;
};

__device__ __forceinline__ void af_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long af_pair(float x, float y) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float af_lo(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float af_hi(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
// rows x d floats (d a multiple of 4), 16 bytes a copy, a warp per row
__device__ __forceinline__ void af_copy_rows(float* dst, int pitch, const float* src, size_t ld, int rows, int d) {
  for (int r = threadIdx.x >> 5; r < rows; r += AF_THREADS / 32)
    for (int c = (threadIdx.x & 31) * 4; c < d; c += 128)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(dst + r * pitch + c)), "l"(src + r * ld + c) : "memory");
}
// What exponentials are taken against: a maximum of -inf stands for scores that are all -inf, whose exponentials are 0.
__device__ __forceinline__ float af_against(float m) { return m == -INFINITY ? 0.f : m; }
// A partial result joins a running one: the maximum, and the factors of both.
__device__ __forceinline__ float af_join(float m, float pm, float& c1, float& c2) {
  const float mn = fmaxf(m, pm), ref = af_against(mn);
  c1 = expf(m - ref), c2 = expf(pm - ref);
  return mn;
}
__device__ __forceinline__ float af_remote(const float* local, unsigned rank) {      // the same word of another CTA of the cluster
  uint32_t a = (uint32_t)__cvta_generic_to_shared(local), b;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(b) : "memory");
  return v;
}
__device__ __forceinline__ void af_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// shared memory (floats): Q [8 TR][D + 4], K [64][D + 4], V [64][64 NC], P [8 TR][68], row facts, and for SPLIT two
// buffers of partial results [8][64 NC + 2]
template <int TR, int NC>
__host__ __device__ constexpr size_t af_smem(int D, bool split) {
  return 4 * ((size_t)8 * TR * (D + 4) + AF_KEYS * (D + 4) + AF_KEYS * 64 * NC + 8 * TR * (AF_KEYS + 4) + 3 * 8 * TR +
              (split ? 2 * 8 * (64 * NC + 2) : 0));
}

template <int TR, int NC, bool SPLIT>
__global__ void __launch_bounds__(AF_THREADS) attention_f32_kernel(const AfArgs a) {
  constexpr int BR = 8 * TR, VP = 64 * NC, PP = AF_KEYS + 4, PART = VP + 2;
  extern __shared__ __align__(16) float af_buf[];
  const int D = a.D, DP = D + 4, Dv = a.Dv;
  float* Qs = af_buf;
  float* Ks = Qs + BR * DP;
  float* Vs = Ks + AF_KEYS * DP;
  float* Ps = Vs + AF_KEYS * VP;
  int* row_pos = reinterpret_cast<int*>(Ps + BR * PP);       // position, first key of the window, sequence (-1: no row)
  int* row_first = row_pos + BR;
  int* row_seq = row_first + BR;
  float* part = reinterpret_cast<float*>(row_seq + BR);      // SPLIT: [2][8][PART] = maximum, sum (-1: no key), values
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tn = lane & 15, tm = warp * 2 + (lane >> 4);     // a row's 16 threads are half a warp
  const int rank = SPLIT ? (int)(blockIdx.x % AF_SPLIT) : 0;
  // A decode step's keys and values come from memory: the first two tiles of the CTA's first token are on their way to L2
  // while the kernel before runs (positions and block tables are the step's inputs).  Three tokens at depths of 138 to 525, 16
  // heads over 4: 22.9 us of a step's chain, 21.0 with this and the partial results of a round asked for together.
  if (SPLIT && !a.seq_start) {
    const int t = (int)(blockIdx.x / AF_SPLIT) * a.tokens_per_cta;
    if (t < a.n_tokens) {
      const int p = a.token_pos[t], kv = blockIdx.y / a.head_blocks;
      int first = a.window > 0 ? max(p - (a.window - 1), 0) : 0;
      if (a.chunk > 0) first = max(first, p - p % a.chunk);
      const int* pages = a.block_table + (size_t)a.token_seq[t] * a.table_width;
      for (int tile = first / AF_KEYS + rank, i = 0; i < 2 && tile <= p / AF_KEYS; ++i, tile += AF_SPLIT) {
        const float* k = a.k_cache + cache_row_offset(pages[tile], kv, 0, a.G, D);
        const float* v = a.v_cache + cache_row_offset(pages[tile], kv, 0, a.G, Dv);
        for (int at = threadIdx.x * 32; at < AF_KEYS * D; at += AF_THREADS * 32) prefetch_l2(k + at);
        for (int at = threadIdx.x * 32; at < AF_KEYS * Dv; at += AF_THREADS * 32) prefetch_l2(v + at);
      }
    }
  }
  pdl_wait();
  const int R = a.H / a.G, g = blockIdx.y / a.head_blocks, h0 = (blockIdx.y % a.head_blocks) * a.heads_per_cta;
  // this CTA's tokens (prompts: the last ones, which see most keys, start first)
  const int slot = SPLIT ? (int)(blockIdx.x / AF_SPLIT) : (int)gridDim.x - 1 - (int)blockIdx.x, per = a.tokens_per_cta;
  int t0 = slot * per, n_tok = min(per, a.n_tokens - t0);
  if (a.seq_start) {                       // of one sequence: its slots start at seq_start / per + its number
    int b = 0;
    for (int hi = a.n_seqs - 1; b < hi;) {
      const int mid = (b + hi + 1) >> 1;
      if (a.seq_start[mid] / per + mid <= slot) b = mid; else hi = mid - 1;
    }
    const int row0 = a.seq_start[b], row1 = min(a.seq_start[b + 1], a.n_tokens);
    t0 = row0 + (slot - (row0 / per + b)) * per;
    n_tok = min(per, row1 - t0);
  }
  // Without seq_start neighbouring tokens may be different sequences'; the z-th of gridDim.z CTAs takes every gridDim.z-th
  // run of tokens of one sequence.
  auto new_run = [&](int tok) { return a.token_seq[t0 + tok] != a.token_seq[t0 + tok - 1]; };
  if (gridDim.z > 1) {
    int n_runs = 1;
    for (int i = 1; i < n_tok; ++i) n_runs += new_run(i);
    if ((int)blockIdx.z >= n_runs) return;
  }
  if (n_tok <= 0) return;                  // (uniform over a cluster, as is the return above)

  for (int r = threadIdx.x; r < BR; r += AF_THREADS) {
    const int tok = r / a.heads_per_cta, h = h0 + r % a.heads_per_cta;
    bool here = tok < n_tok && h < R;
    if (here && gridDim.z > 1) {
      int run = 0;
      for (int i = 1; i <= tok; ++i) run += new_run(i);
      here = run % (int)gridDim.z == (int)blockIdx.z;
    }
    const int p = here ? a.token_pos[t0 + tok] : 0;
    int first = (a.window > 0 && p - (a.window - 1) > 0) ? p - (a.window - 1) : 0;
    if (a.chunk > 0) first = max(first, p - p % a.chunk);
    row_pos[r] = p, row_first[r] = first, row_seq[r] = here ? a.token_seq[t0 + tok] : -1;
  }
  if (Dv < VP)                             // dims past Dv
    for (int i = threadIdx.x; i < AF_KEYS * VP; i += AF_THREADS) Vs[i] = 0.f;
  __syncthreads();
  for (int r = warp; r < BR; r += AF_THREADS / 32) {
    const int tok = r / a.heads_per_cta, h = h0 + r % a.heads_per_cta;
    float* dst = Qs + r * DP;
    const float* src = a.q + (size_t)(t0 + tok) * a.q_stride + (size_t)(g * R + h) * D;
    if (row_seq[r] < 0) {
      for (int i = lane; i < D; i += 32) dst[i] = 0.f;
    } else if (a.q_vec) {                  // (they come with the first tile of keys)
      for (int c = lane * 4; c < D; c += 128)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + c)), "l"(src + c)
                     : "memory");
    } else {
      for (int i = lane; i < D; i += 32) dst[i] = src[i];
    }
  }

  int pos[TR], first[TR], seq[TR];
  float m[TR], l[TR];
  unsigned long long acc[TR][2 * NC];
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    pos[i] = row_pos[i * 8 + tm], first[i] = row_first[i * 8 + tm], seq[i] = row_seq[i * 8 + tm];
    m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * NC; ++c) acc[i][c] = 0ull;
  }
  // SPLIT: this thread's elements of the CTA's slice of the dims, and their running state
  const int slice = (Dv + AF_SPLIT - 1) / AF_SPLIT;
  constexpr int OWN = SPLIT ? (8 * 8 * NC + AF_THREADS - 1) / AF_THREADS : 1;
  float om[OWN], ol[OWN], oa[OWN];
#pragma unroll
  for (int e = 0; e < OWN; ++e) om[e] = -INFINITY, ol[e] = 0.f, oa[e] = 0.f;

  // tokens of one sequence that follow one another share its tiles
  int parity = 0;                               // SPLIT: of the rounds so far
  for (int run = 0; run < n_tok;) {
    const int s = row_seq[run * a.heads_per_cta];
    if (s < 0) {                                // (another CTA's)
      ++run;
      continue;
    }
    int lo = row_first[run * a.heads_per_cta], hi = row_pos[run * a.heads_per_cta], end = run + 1;
    for (; end < n_tok && row_seq[end * a.heads_per_cta] == s; ++end) {
      lo = min(lo, row_first[end * a.heads_per_cta]);
      hi = max(hi, row_pos[end * a.heads_per_cta]);
    }
    const int tok_lo = run, tok_hi = end;
    run = end;
    const int tile_first = lo / AF_KEYS, tile_last = hi / AF_KEYS;
    const int n_kept = a.window > 0 && a.keep_first > 0 ? min(tile_first, (a.keep_first + AF_KEYS - 1) / AF_KEYS) : 0;
    const int n_tiles = n_kept + tile_last - tile_first + 1;
    const int* pages = a.block_table + (size_t)s * a.table_width;
    bool mine[TR];              // whether the row belongs to this run
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      const int tok = (i * 8 + tm) / a.heads_per_cta;
      mine[i] = seq[i] >= 0 && tok >= tok_lo && tok < tok_hi;
    }
    auto tile_at = [&](int j) { return j < n_kept ? j : tile_first + (j - n_kept); };
    auto load_k = [&](int j) {
      if (j < n_tiles)
        af_copy_rows(Ks, DP, a.k_cache + cache_row_offset(pages[tile_at(j)], g, 0, a.G, D), D, AF_KEYS, D);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto load_v = [&](int j) {
      if (j < n_tiles)
        af_copy_rows(Vs, VP, a.v_cache + cache_row_offset(pages[tile_at(j)], g, 0, a.G, Dv), Dv, AF_KEYS, Dv);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int STEP = SPLIT ? AF_SPLIT : 1;
    __syncthreads();                            // (a run before is done with K and V)
    load_k(rank), load_v(rank);
    for (int j = rank, round = 0; j - rank < n_tiles; j += STEP, ++round, parity ^= 1) {
      unsigned long long pacc[TR][2 * NC];
      float pm[TR], pl[TR];
      bool any[TR];
      if (j < n_tiles) {
        const int k0 = tile_at(j) * AF_KEYS;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        // ---- scores: TR rows x keys tn, tn + 16, tn + 32, tn + 48 ----
        unsigned long long sc[TR][4];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) sc[i][c] = 0ull;
        const float* qs = Qs + tm * DP;
        const float* ks = Ks + tn * DP;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          ulonglong2 x[TR];
#pragma unroll
          for (int i = 0; i < TR; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(qs + i * 8 * DP + d);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ks + c * 16 * DP + d);
#pragma unroll
            for (int i = 0; i < TR; ++i) af_fma2(sc[i][c], x[i].x, y.x);
#pragma unroll
            for (int i = 0; i < TR; ++i) af_fma2(sc[i][c], x[i].y, y.y);
          }
        }
        __syncthreads();                        // everyone has read K
        load_k(j + STEP);
        // ---- the tile's maximum, exponentials and their sum; P to shared memory, -1 where the row does not see the key
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          const int p = pos[i], f = first[i];
          any[i] = mine[i] && k0 <= p && (k0 + AF_KEYS - 1 >= f || k0 < a.keep_first);
          float sv[4];
          bool live[4];
          pm[i] = -INFINITY;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int key = k0 + tn + 16 * c;
            live[c] = any[i] && key <= p && (key >= f || key < a.keep_first);
            float v = __fmul_rn(__fadd_rn(af_lo(sc[i][c]), af_hi(sc[i][c])), a.scale);
            if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);
            if (a.score_bias && live[c])
              v = __fadd_rn(v, a.score_bias[(size_t)(g * R + h0 + (i * 8 + tm) % a.heads_per_cta) * a.bias_len +
                                            min(p - key, a.bias_len - 1)]);
            sv[c] = v;
            if (live[c]) pm[i] = fmaxf(pm[i], v);
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) pm[i] = fmaxf(pm[i], __shfl_xor_sync(0xffffffffu, pm[i], o));
          pl[i] = 0.f;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float e = live[c] ? expf(sv[c] - af_against(pm[i])) : -1.f;
            if (live[c]) pl[i] = __fadd_rn(pl[i], e);
            Ps[(i * 8 + tm) * PP + tn + 16 * c] = e;
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) pl[i] = __fadd_rn(pl[i], __shfl_xor_sync(0xffffffffu, pl[i], o));
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                        // V is there (and P)
        // ---- weighted values: TR rows x dims 4 tn .. 4 tn + 3 of every 64 ----
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int c = 0; c < 2 * NC; ++c) pacc[i][c] = 0ull;
        const float* vs = Vs + tn * 4;
#pragma unroll 1
        for (int key = 0; key < AF_KEYS; key += 4) {
          float4 w[TR];
#pragma unroll
          for (int i = 0; i < TR; ++i) w[i] = *reinterpret_cast<const float4*>(Ps + (i * 8 + tm) * PP + key);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            ulonglong2 v[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) v[c] = *reinterpret_cast<const ulonglong2*>(vs + (key + kk) * VP + 64 * c);
#pragma unroll
            for (int i = 0; i < TR; ++i) {
              const float e = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
              if (!(e < 0.f)) {
                const unsigned long long ee = af_pair(e, e);
#pragma unroll
                for (int c = 0; c < NC; ++c) af_fma2(pacc[i][2 * c], ee, v[c].x), af_fma2(pacc[i][2 * c + 1], ee, v[c].y);
              }
            }
          }
        }
        __syncthreads();                        // everyone has read V and P
        load_v(j + STEP);
      }
      if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          if (!any[i]) continue;
          float c1, c2;
          m[i] = af_join(m[i], pm[i], c1, c2);
          l[i] = __fmaf_rn(pl[i], c2, __fmul_rn(l[i], c1));
#pragma unroll
          for (int c = 0; c < 2 * NC; ++c)
            acc[i][c] = af_pair(__fmaf_rn(af_lo(pacc[i][c]), c2, __fmul_rn(af_lo(acc[i][c]), c1)),
                                __fmaf_rn(af_hi(pacc[i][c]), c2, __fmul_rn(af_hi(acc[i][c]), c1)));
        }
      } else {
        float* mine_part = part + ((size_t)parity * 8 + tm) * PART;
        if (j < n_tiles) {
          if (tn == 0) mine_part[0] = pm[0], mine_part[1] = any[0] ? pl[0] : -1.f;
#pragma unroll
          for (int c = 0; c < 2 * NC; ++c) {
            const int d = (c >> 1) * 64 + tn * 4 + (c & 1) * 2;
            mine_part[2 + d] = af_lo(pacc[0][c]), mine_part[3 + d] = af_hi(pacc[0][c]);
          }
        }
        af_cluster_sync();                      // (a buffer is written again two rounds on, behind the next barrier)
        const int here = min(AF_SPLIT, n_tiles - round * AF_SPLIT);
#pragma unroll
        for (int e = 0; e < OWN; ++e) {
          const int idx = e * AF_THREADS + threadIdx.x, row = idx / slice, d = rank * slice + idx % slice;
          if (row >= 8 || d >= Dv) continue;
          const float* src = part + ((size_t)parity * 8 + row) * PART;
          float km[AF_SPLIT], kl[AF_SPLIT], ka[AF_SPLIT];    // (all on their way together: one trip, not one a tile)
#pragma unroll
          for (int k = 0; k < AF_SPLIT; ++k)
            if (k < here) km[k] = af_remote(src, k), kl[k] = af_remote(src + 1, k), ka[k] = af_remote(src + 2 + d, k);
#pragma unroll
          for (int k = 0; k < AF_SPLIT; ++k) {
            if (k >= here || kl[k] < 0.f) continue;
            float c1, c2;
            om[e] = af_join(om[e], km[k], c1, c2);
            ol[e] = __fmaf_rn(kl[k], c2, __fmul_rn(ol[e], c1));
            oa[e] = __fmaf_rn(ka[k], c2, __fmul_rn(oa[e], c1));
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // ---- sinks, the output's gate, the division ----
  auto inverse = [&](float mm, float ll, int tok, int h) {
    if (a.sink > 0.f) ll = __fadd_rn(ll, __fmul_rn(a.sink, expf(-mm)));
    if (a.sinks) ll = __fadd_rn(ll, expf(a.sinks[h] - mm));
    float inv = __fdiv_rn(1.0f, ll);
    if (a.gate) inv = __fmul_rn(inv, __fdiv_rn(1.0f, 1.0f + expf(-a.gate[(size_t)tok * a.gate_stride + h])));
    return inv;
  };
  if (SPLIT) {
#pragma unroll
    for (int e = 0; e < OWN; ++e) {
      const int idx = e * AF_THREADS + threadIdx.x, row = idx / slice, d = rank * slice + idx % slice;
      if (row >= 8 || d >= Dv || row_seq[row] < 0) continue;
      const int tok = t0 + row / a.heads_per_cta, h = g * R + h0 + row % a.heads_per_cta;
      a.out[((size_t)tok * a.H + h) * Dv + d] = __fmul_rn(oa[e], inverse(om[e], ol[e], tok, h));
    }
    af_cluster_sync();                          // nobody leaves while its partial results may be read
  } else {
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      if (seq[i] < 0) continue;
      const int r = i * 8 + tm, tok = t0 + r / a.heads_per_cta, h = g * R + h0 + r % a.heads_per_cta;
      const float inv = inverse(m[i], l[i], tok, h);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int d = c * 64 + tn * 4;
        if (d < Dv)
          *reinterpret_cast<float4*>(a.out + ((size_t)tok * a.H + h) * Dv + d) =
              make_float4(__fmul_rn(af_lo(acc[i][2 * c]), inv), __fmul_rn(af_hi(acc[i][2 * c]), inv),
                          __fmul_rn(af_lo(acc[i][2 * c + 1]), inv), __fmul_rn(af_hi(acc[i][2 * c + 1]), inv));
      }
    }
  }
}

template <int TR, int NC, bool SPLIT>
static int launch_f32(AfArgs a, bool single_tokens, cudaStream_t stream) {
  const int R = a.H / a.G, rows = 8 * TR;
  a.heads_per_cta = R < rows ? R : rows;
  a.tokens_per_cta = single_tokens ? 1 : rows / a.heads_per_cta;
  a.head_blocks = (R + a.heads_per_cta - 1) / a.heads_per_cta;
  if (a.tokens_per_cta == 1) a.seq_start = nullptr;             // (a token is a run by itself)
  const unsigned slots = a.seq_start ? a.n_tokens / a.tokens_per_cta + a.n_seqs
                                     : (a.n_tokens + a.tokens_per_cta - 1) / a.tokens_per_cta;
  const unsigned runs = a.seq_start || a.tokens_per_cta == 1 ? 1 : a.tokens_per_cta < 8 ? a.tokens_per_cta : 8;
  auto kernel = attention_f32_kernel<TR, NC, SPLIT>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)af_smem<TR, NC>(ATT_MAX_D, SPLIT));
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const size_t smem = af_smem<TR, NC>(a.D, SPLIT);
  const dim3 grid(slots * (SPLIT ? AF_SPLIT : 1), a.G * a.head_blocks, runs);
  if (SPLIT)
    launch_pdl_cluster(kernel, grid, dim3(AF_THREADS), smem, stream, AF_SPLIT, a);
  else
    launch_pdl(kernel, grid, dim3(AF_THREADS), smem, stream, a);
  return LLMX_LAUNCH_STATUS();
}

// launch: 0: rows of 8 in a cluster, 1: rows of 8, 2: rows of 32, -1: by the rule.
// Rule: the cheapest by what 90 steps took (heads of 64, 128 and 256, 1 to 8 rows and more a kv head, single tokens, prompts,
// portions of prompts and mixtures, depths of 17 to 4096).  The unit is what a CTA of 8 rows takes for a tile with an SM to
// itself (5.6, 7.8 and 10.8 us by head size), a cluster's round costs 1.55 of it and a tile of 32 rows 1.75; where CTAs
// share the SMs, a CTA-tile costs an SM what the table says.  us by cluster / 8 rows / 32 rows (heads of 128): one
// token at depth 4096, 16 heads over 4: 97 / 502 / 849; 64 tokens at depth 300, 16 over 16: 486 / 165 / 327; three prompts
// of 500, 16 over 4: 1575 / 376 / 262; 40 tokens at depth 2048 beside a prompt of 64, 16 over 16: 1273 / 667 / 1425.  The
// kernel above takes 2655, 458, 3353 and 2981.
static int attention_f32(const AfArgs& a, bool single_tokens, int launch, cudaStream_t stream) {
  if (launch < 0) {
    static const double share[3][3] = {{0.45, 0.38, 1.07}, {0.97, 0.55, 1.45}, {1.93, 1.2, 3.1}};     // [head size][launch]
    const int size = a.D > a.Dv ? a.D : a.Dv, R = a.H / a.G;
    const double* cost = share[size <= 64 ? 0 : size <= 128 ? 1 : 2];
    double tiles = a.table_width;
    if (a.window > 0) tiles = fmin(tiles, (a.window + a.keep_first) / AF_KEYS + 2.0);
    const auto per_sm = [&](int rows) {                     // CTAs of that many rows
      const int heads = R < rows ? R : rows, tokens = single_tokens ? 1 : rows / heads;
      const double slots = a.n_tokens / tokens + (a.seq_start && tokens > 1 ? a.n_seqs : 0);
      return fmax(slots, 1.0) * a.G * ((R + heads - 1) / heads) / llmx_sm_count();
    };
    const double by_cluster = 0.85 * ceil(tiles / AF_SPLIT) * fmax(1.55, per_sm(8) * AF_SPLIT * cost[0]);
    const double by_8 = tiles * fmax(1.0, per_sm(8) * cost[1]), by_32 = tiles * fmax(1.75, per_sm(32) * cost[2]);
    launch = by_cluster < by_8 && by_cluster < by_32 ? 0 : by_8 <= by_32 ? 1 : 2;
  }
#define GO(NC)                                                                  \
  return launch == 0   ? launch_f32<1, NC, true>(a, single_tokens, stream)      \
         : launch == 1 ? launch_f32<1, NC, false>(a, single_tokens, stream)     \
                       : launch_f32<4, NC, false>(a, single_tokens, stream)
  switch ((a.Dv + 63) / 64) {
    case 1: GO(1);
    case 2: GO(2);
    case 3: GO(3);
    default: GO(4);
  }
#undef GO
}

// pool > 0: pool_k / pool_v hold one row per block of `pool` positions, paged like the cache, with the block table
// pool_table (as wide as block_table); needs a window and no kept first keys.  gate: null, or float32 with
// gate[t * gate_stride + head] the logit of head's output gate.
// softcap <= 0: scores are not capped; sinks: null, or float32 [H]; score_bias: null, or float32 [H, bias_len].
// Hints, which pick the launch and not the result: single_tokens: every token is a sequence's only one in this step;
// seq_start: null, or [n_seqs + 1]: the tokens lie sequence after sequence from there; launch: see attention_f32.
LLMX_API int llmx_attention_paged_biased(const void* q, void* out, int act_dtype, const void* k_cache,
                                  const void* v_cache, int cache_dtype, const int* block_table, int table_width,
                                  const int* token_seq, const int* token_pos, int n_tokens, int H, int G, int D,
                                  int Dv, long long q_stride, int window, int keep_first, float scale, float sink,
                                  int chunk, int pool, const void* pool_k, const void* pool_v, const int* pool_table,
                                  const float* gate, long long gate_stride, float softcap, const float* sinks,
                                  const float* score_bias, int bias_len, int single_tokens, const int* seq_start,
                                  int n_seqs, int launch, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (launch > 2 || (seq_start && n_seqs <= 0)) return LLMX_REFUSED(1);
  if (score_bias && (bias_len <= 0 || pool > 0 || softcap > 0.f)) return LLMX_REFUSED(1);
  if (chunk < 0 || (chunk > 0 && keep_first > 0)) return LLMX_REFUSED(1);
  if (pool < 0 || (pool > 0 && (window <= 0 || keep_first > 0 || chunk > 0 || !pool_k || !pool_v || !pool_table)))
    return LLMX_REFUSED(1);
  if (gate && gate_stride < H) return LLMX_REFUSED(1);
  if (H <= 0 || G <= 0 || H % G != 0 || D <= 0 || D > ATT_MAX_D || window < 0) return LLMX_REFUSED(1);
  if (Dv <= 0 || Dv > ATT_MAX_D || keep_first < 0 || q_stride < (long long)H * D) return LLMX_REFUSED(1);
  // float32 by tiles: whole 16-byte rows (a layer's sizes and strides, the same for every step), no pooled blocks
  const auto aligned = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  if (act_dtype == LLMX_F32 && cache_dtype == LLMX_F32 && pool == 0 && D % 4 == 0 && Dv % 4 == 0 && aligned(k_cache) &&
      aligned(v_cache) && aligned(out) && n_tokens <= 0x7fffffff / AF_SPLIT && (long long)H <= 65535) {
    AfArgs a = {};
    a.q = (const float*)q, a.k_cache = (const float*)k_cache, a.v_cache = (const float*)v_cache, a.gate = gate;
    a.sinks = sinks, a.score_bias = score_bias, a.out = (float*)out, a.block_table = block_table;
    a.token_seq = token_seq, a.token_pos = token_pos, a.q_stride = (size_t)q_stride, a.gate_stride = (size_t)gate_stride;
    a.table_width = table_width, a.n_tokens = n_tokens, a.H = H, a.G = G, a.D = D, a.Dv = Dv, a.window = window;
    a.keep_first = keep_first, a.chunk = chunk, a.bias_len = bias_len, a.scale = scale, a.sink = sink, a.softcap = softcap;
    a.seq_start = seq_start, a.n_seqs = n_seqs, a.q_vec = aligned(q) && q_stride % 4 == 0;
    return attention_f32(a, single_tokens != 0, launch, stream);
  }
  dim3 grid(n_tokens, (H + ATT_WARPS - 1) / ATT_WARPS);
  const size_t smem = (size_t)ATT_WARPS * D * sizeof(float);
#define CASE(TA, TC)                                                                                      \
  launch_pdl(attention_paged_kernel<TA, TC>, grid, dim3(ATT_WARPS * 32), smem, stream,                    \
      (const TA*)q, (TA*)out, (const TC*)k_cache, (const TC*)v_cache, block_table, table_width, token_seq, \
      token_pos, H, G, D, Dv, (size_t)q_stride, window, keep_first, scale, sink, chunk, pool, (const TC*)pool_k,  \
      (const TC*)pool_v, pool_table, gate, (size_t)gate_stride, softcap, sinks, score_bias, bias_len)
  if (act_dtype == LLMX_F32 && cache_dtype == LLMX_F32) CASE(float, float);
  else if (act_dtype == LLMX_BF16 && cache_dtype == LLMX_BF16) CASE(bf16, bf16);
  else if (act_dtype == LLMX_F32 && cache_dtype == LLMX_BF16) CASE(float, bf16);
  else if (act_dtype == LLMX_BF16 && cache_dtype == LLMX_F32) CASE(bf16, float);
  else return LLMX_REFUSED(2);
#undef CASE
  return LLMX_LAUNCH_STATUS();
}

LLMX_API int llmx_attention_paged_capped(const void* q, void* out, int act_dtype, const void* k_cache,
                                  const void* v_cache, int cache_dtype, const int* block_table, int table_width,
                                  const int* token_seq, const int* token_pos, int n_tokens, int H, int G, int D,
                                  int Dv, long long q_stride, int window, int keep_first, float scale, float sink,
                                  int chunk, int pool, const void* pool_k, const void* pool_v, const int* pool_table,
                                  const float* gate, long long gate_stride, float softcap, const float* sinks,
                                  cudaStream_t stream) {
  return llmx_attention_paged_biased(q, out, act_dtype, k_cache, v_cache, cache_dtype, block_table, table_width,
                                     token_seq, token_pos, n_tokens, H, G, D, Dv, q_stride, window, keep_first, scale,
                                     sink, chunk, pool, pool_k, pool_v, pool_table, gate, gate_stride, softcap, sinks,
                                     nullptr, 0, 0, nullptr, 0, -1, stream);
}

LLMX_API int llmx_attention_paged_pooled(const void* q, void* out, int act_dtype, const void* k_cache,
                                  const void* v_cache, int cache_dtype, const int* block_table, int table_width,
                                  const int* token_seq, const int* token_pos, int n_tokens, int H, int G, int D,
                                  int Dv, long long q_stride, int window, int keep_first, float scale, float sink,
                                  int chunk, int pool, const void* pool_k, const void* pool_v, const int* pool_table,
                                  const float* gate, long long gate_stride, cudaStream_t stream) {
  return llmx_attention_paged_capped(q, out, act_dtype, k_cache, v_cache, cache_dtype, block_table, table_width,
                                     token_seq, token_pos, n_tokens, H, G, D, Dv, q_stride, window, keep_first, scale,
                                     sink, chunk, pool, pool_k, pool_v, pool_table, gate, gate_stride, 0.f, nullptr,
                                     stream);
}

LLMX_API int llmx_attention_paged_chunked(const void* q, void* out, int act_dtype, const void* k_cache,
                                  const void* v_cache, int cache_dtype, const int* block_table, int table_width,
                                  const int* token_seq, const int* token_pos, int n_tokens, int H, int G, int D,
                                  int Dv, long long q_stride, int window, int keep_first, float scale, float sink,
                                  int chunk, cudaStream_t stream) {
  return llmx_attention_paged_pooled(q, out, act_dtype, k_cache, v_cache, cache_dtype, block_table, table_width,
                                     token_seq, token_pos, n_tokens, H, G, D, Dv, q_stride, window, keep_first, scale,
                                     sink, chunk, 0, nullptr, nullptr, nullptr, nullptr, 0, stream);
}

LLMX_API int llmx_attention_paged(const void* q, void* out, int act_dtype, const void* k_cache,
                                  const void* v_cache, int cache_dtype, const int* block_table, int table_width,
                                  const int* token_seq, const int* token_pos, int n_tokens, int H, int G, int D,
                                  int Dv, long long q_stride, int window, int keep_first, float scale, float sink,
                                  cudaStream_t stream) {
  return llmx_attention_paged_chunked(q, out, act_dtype, k_cache, v_cache, cache_dtype, block_table, table_width,
                                      token_seq, token_pos, n_tokens, H, G, D, Dv, q_stride, window, keep_first, scale,
                                      sink, 0, stream);
}

// ---------------------------------------------------------------------------
// The store of one row per block of `pool` positions: when a step writes the last position of block b
// (position b*pool + pool - 1), that block's key is the mean of its `pool` keys as the cache holds them, its value
// the mean of the values, summed in float32 in an order that `pool` alone decides, times 1 / pool, and stored as
// row b of the second store.
// The cache must still hold the block's positions: its window is at least `pool`.
// ---------------------------------------------------------------------------
// A lane owns V consecutive dims (16 bytes of the cache where the sizes allow it) and walks positions in order
// with several loads in flight.
template <int V>
__device__ __forceinline__ void pb_load(const float* p, float* o) {
  if (V == 1) {
    o[0] = p[0];
  } else {
    const float4 x = *reinterpret_cast<const float4*>(p);
    o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w;
  }
}
template <int V>
__device__ __forceinline__ void pb_load(const bf16* p, float* o) {
  if (V == 1) {
    o[0] = to_f32(p[0]);
  } else {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h2[e]);
      o[2 * e] = f.x, o[2 * e + 1] = f.y;
    }
  }
}

#define PB_WARPS 8

// One CTA per (block that ends in the step, kv head, keys or values).  A block's positions are cut into PB_WARPS runs of equal length; warp w
// sums its run in position order (a lane owns V consecutive dims), and the runs' sums are added in the order of the
// runs: an order that depends on `pool` alone.
template <typename TC, int V>
__global__ void pool_blocks_kernel(const TC* __restrict__ k_cache, const TC* __restrict__ v_cache,
                                   const int* __restrict__ block_table, TC* __restrict__ pool_k,
                                   TC* __restrict__ pool_v, const int* __restrict__ pool_table, int table_width,
                                   const int* __restrict__ seq_start, const int* __restrict__ seq_past, int n_seqs,
                                   int G, int D, int Dv, int pool, int n_pages, int n_pool_pages) {
  extern __shared__ float pb_part[];                    // [PB_WARPS][width]
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int unit = blockIdx.y;                          // unit: kv head g's keys (2g) or values (2g+1)
  // The grid's x axis counts the blocks that end in this step, sequence after sequence: sequence s, which held
  // `past` positions and brings n, ends the blocks past / pool .. (past + n) / pool - 1.  CTAs beyond the step's
  // count leave at once (the grid is sized from the step's shape alone: tokens / pool + sequences).
  int left = blockIdx.x, seq = -1, p = 0;
  for (int s2 = 0; s2 < n_seqs; ++s2) {
    const int past = seq_past[s2], n = seq_start[s2 + 1] - seq_start[s2];
    const int first = past / pool, count = (past + n) / pool - first;
    if (left < count) {
      seq = s2;
      p = (first + left) * pool + pool - 1;               // the block's last position
      break;
    }
    left -= count;
  }
  if (seq < 0) return;                                    // uniform over the CTA
  const int g = unit >> 1, is_v = unit & 1;
  const int b = p / pool;
  const int* pages = block_table + (size_t)seq * table_width;
  const int dst_page = pool_table[(size_t)seq * table_width + b / LLMX_PAGE];
  if (dst_page < 0 || dst_page >= n_pool_pages) {
    if (threadIdx.x == 0) llmx_report(1);
    return;
  }
  const int width = is_v ? Dv : D;
  const TC* src = is_v ? v_cache : k_cache;
  TC* dst = (is_v ? pool_v : pool_k) + cache_row_offset(dst_page, g, b % LLMX_PAGE, G, width);
  pdl_wait();
  const int run = (pool + PB_WARPS - 1) / PB_WARPS;
  const int j_lo = p - pool + 1 + warp * run, j_hi = min(j_lo + run, p + 1);     // this warp's positions
  bool bad = false;
  for (int d0 = lane * V; d0 < width; d0 += 32 * V) {
    float sum[V];
#pragma unroll
    for (int e = 0; e < V; ++e) sum[e] = 0.f;
    for (int jb = j_lo; jb < j_hi; jb += 8) {              // eight positions' loads go out together
      float x[8][V];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = jb + u;
        if (j < j_hi) {
          int page = pages[j / LLMX_PAGE];
          if (page < 0 || page >= n_pages) bad = true, page = 0;
          pb_load<V>(src + cache_row_offset(page, g, j % LLMX_PAGE, G, width) + d0, x[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (jb + u < j_hi) {
#pragma unroll
          for (int e = 0; e < V; ++e) sum[e] += x[u][e];
        }
    }
#pragma unroll
    for (int e = 0; e < V; ++e) pb_part[warp * width + d0 + e] = sum[e];
  }
  if (bad) llmx_report(2);
  __syncthreads();
  const float inv = 1.0f / (float)pool;
  for (int d = threadIdx.x; d < width; d += PB_WARPS * 32) {
    float sum = pb_part[d];
#pragma unroll
    for (int w = 1; w < PB_WARPS; ++w) sum += pb_part[w * width + d];
    dst[d] = from_f32<TC>(sum * inv);
  }
}

// seq_start [n_seqs + 1], seq_past [n_seqs]: where each sequence's tokens start in the step and how many positions it
// held before; n_tokens: the step's tokens.
LLMX_API int llmx_pool_blocks(const void* k_cache, const void* v_cache, int cache_dtype, const int* block_table,
                              void* pool_k, void* pool_v, const int* pool_table, int table_width, const int* seq_start,
                              const int* seq_past, int n_seqs, int n_tokens, int G, int D, int Dv, int pool,
                              long long n_pages, long long n_pool_pages, cudaStream_t stream) {
  if (n_tokens <= 0 || n_seqs <= 0) return 0;
  if (G <= 0 || D <= 0 || Dv <= 0 || pool < 1 || n_pages < 1 || n_pool_pages < 1) return LLMX_REFUSED(1);
  if (2 * G > 65535) return LLMX_REFUSED(3);
  dim3 grid(n_tokens / pool + n_seqs, 2 * G);             // at least as many as blocks can end in such a step
  const size_t smem = (size_t)PB_WARPS * (D > Dv ? D : Dv) * sizeof(float);
  if (smem > 48 * 1024) return LLMX_REFUSED(3);
  const int v = cache_dtype == LLMX_BF16 ? 8 : 4;
  const bool vec = D % v == 0 && Dv % v == 0 && !(((uintptr_t)k_cache | (uintptr_t)v_cache) & 15);
#define CASE(TC, V)                                                                                           \
  launch_pdl(pool_blocks_kernel<TC, V>, grid, dim3(PB_WARPS * 32), smem, stream, (const TC*)k_cache,           \
             (const TC*)v_cache, block_table, (TC*)pool_k, (TC*)pool_v, pool_table, table_width, seq_start,    \
             seq_past, n_seqs, G, D, Dv, pool, (int)n_pages, (int)n_pool_pages)
  if (cache_dtype == LLMX_F32) {
    if (vec) CASE(float, 4); else CASE(float, 1);
  } else if (cache_dtype == LLMX_BF16) {
    if (vec) CASE(bf16, 8); else CASE(bf16, 1);
  } else {
    return LLMX_REFUSED(2);
  }
#undef CASE
  return LLMX_LAUNCH_STATUS();
}
