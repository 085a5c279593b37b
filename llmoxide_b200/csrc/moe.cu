// Routed experts (a mixture of small gated feed-forward layers of which each token uses a few).
//
//   route      per token: scores from the router's float32 logits, the groups of experts a token may choose
//              from, its `top` experts and their weights
//   sort       the step's (token, choice) pairs ordered by expert, and the list of row tiles per expert
//   grouped products on the sorted rows: gate|up with the gated activation, then down times the pair's weight
//
// Everything a token gets depends on that token alone: routing is per token, and every output element of the
// products is accumulated by one thread in the order k = 0..K-1 whatever tile the row falls into, so results
// do not depend on what else is in the batch or on how a prompt was cut.  The order of rows inside an
// expert's segment is whatever the sort's atomics gave; no value depends on it.
#include "common.cuh"

#include <type_traits>

#define MOE_TILE 64          // rows (and columns) per tile of the grouped products
#define MOE_BK 16
#define MOE_MAX_TOP 16
#define MOE_MAX_EXPERTS 1024

// SOFTMAX_TOP: the choice goes by the logits themselves, and the weights are the softmax over the chosen logits only.
enum { MOE_SCORE_SIGMOID = 0, MOE_SCORE_SOFTMAX = 1, MOE_SCORE_SOFTMAX_TOP = 2 };

// ---------------------------------------------------------------------------
// Routing.  One warp per token.  s = sigmoid(z) (or softmax(z)).  The expert indices are cut into n_groups
// contiguous blocks of E / n_groups; a block ranks by the sum of its group_top highest s, and only the
// keep_groups top-ranked blocks stay eligible.  Among the eligible experts the `top` highest s win (ties: the
// lower index); a winner's weight is its s, over (the winners' sum + norm_eps) when `normalize`, times `scale`.
// With a correction (`bias`, one number per expert) the groups are ranked and the experts chosen by s + bias,
// while the weights stay the chosen experts' s.
// ---------------------------------------------------------------------------
// The largest v of the warp above -inf and the lowest i that goes with it; none: i = 0x7fffffff.  (NaN is not above -inf.)
// Two reductions over the warp by the hardware, on integers in the order of the floats, in place of five rounds of two shuffles.
__device__ __forceinline__ int warp_argmax(float v, int i) {
  const int bits = __float_as_int(v + 0.0f);                       // (-0 and +0 are equal)
  const unsigned key = v > -INFINITY ? (unsigned)bits ^ (bits < 0 ? 0xffffffffu : 0x80000000u) : 0u;
  const unsigned top = __reduce_max_sync(0xffffffffu, key);
  return (int)__reduce_min_sync(0xffffffffu, top != 0u && key == top ? (unsigned)i : 0x7fffffffu);
}

// One token, by one warp: z its E logits (global or shared memory), s, c and gs scratch of E, E and n_groups
// floats (c: the scores the choice goes by).  Lane k < top returns the k-th choice and its weight.  report: whether a choice
// that cannot be made is one.
__device__ __forceinline__ void moe_route_token(const float* z, float* s, float* c, float* gs, int& id, float& weight, int lane, int E, int top, int n_groups,
                                                int keep_groups, int group_top, int score_kind, int normalize,
                                                float norm_eps, float scale, const float* __restrict__ bias, bool report = true) {
  if (score_kind == MOE_SCORE_SOFTMAX) {
    float m = -INFINITY;
    for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
    m = warp_max(m);
    float sum = 0.f;
    for (int e = lane; e < E; e += 32) sum += expf(z[e] - m);
    sum = warp_sum(sum);
    for (int e = lane; e < E; e += 32) s[e] = expf(z[e] - m) / sum;
  } else if (score_kind == MOE_SCORE_SOFTMAX_TOP) {
    for (int e = lane; e < E; e += 32) s[e] = z[e];
  } else {
    for (int e = lane; e < E; e += 32) s[e] = 1.0f / (1.0f + expf(-z[e]));
  }
  __syncwarp();
  for (int e = lane; e < E; e += 32) c[e] = bias ? s[e] + bias[e] : s[e];
  __syncwarp();
  const int per = E / n_groups;
  if (n_groups > 1 && keep_groups < n_groups) {
    // a group's score: the sum of its group_top (at most 8) largest, largest first; they are kept in order as the group's
    // scores come by (a NaN never gets in)
    for (int g = lane; g < n_groups; g += 32) {
      float best[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) best[k] = -INFINITY;
      const int n_pick = group_top < per ? group_top : per;
      for (int e = g * per; e < (g + 1) * per; ++e) {
        float v = c[e];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < n_pick && v > best[k]) {
            const float w = best[k];
            best[k] = v, v = w;
          }
      }
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < n_pick) sum += best[k];
      gs[g] = sum;
    }
    __syncwarp();
    // the keep_groups best groups stay; the others' experts get a score no expert can have
    for (int k = 0; k < keep_groups; ++k) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
      for (int g = lane; g < n_groups; g += 32)
        if (gs[g] > best) best = gs[g], bi = g;     // ascending g: the lower index wins a tie
      bi = warp_argmax(best, bi);
      if (lane == 0 && bi < n_groups) gs[bi] = -INFINITY;            // kept: marked (no group: all their scores are NaN)
      __syncwarp();
    }
    for (int e = lane; e < E; e += 32)
      if (gs[e / per] != -INFINITY) c[e] = -INFINITY;   // not kept
    __syncwarp();
  }
  float sum = 0.f, mine = 0.f;
  int my_id = 0;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32)
      if (c[e] > best) best = c[e], bi = e;
    bi = warp_argmax(best, bi);
    if (bi >= E) {
      // No score compares greater than -inf: the token's row holds a NaN (or every score is -inf).  That is
      // reported (code 1); the lowest expert not chosen yet stands in, so that no index leaves its array.
      bi = 0x7fffffff;
      for (int e = lane; e < E; e += 32)
        if (!(c[e] == -INFINITY) && e < bi) bi = e;
      bi = (int)__reduce_min_sync(0xffffffffu, (unsigned)bi);
      if (bi >= E) bi = k % E;
      if (lane == 0 && report) llmx_report(1);
    }
    if (lane == 0) c[bi] = -INFINITY;               // chosen: out of the running
    __syncwarp();
    const float sb = s[bi];
    if (lane == k) mine = sb, my_id = bi;
    sum += sb;
  }
  if (score_kind == MOE_SCORE_SOFTMAX_TOP) {
    // lane k holds the k-th chosen logit: softmax over those (all lanes take part in the butterflies)
    const float zk = lane < top ? mine : -INFINITY;
    const float z_max = warp_max(zk);
    const float ek = lane < top ? expf(zk - z_max) : 0.f;
    const float total = warp_sum(ek);
    id = my_id, weight = (ek / total) * scale;
    return;
  }
  const float w = normalize ? mine / (sum + norm_eps) : mine;
  id = my_id, weight = w * scale;
}

__global__ void moe_route_kernel(const float* __restrict__ logits, int* __restrict__ ids, float* __restrict__ wts,
                                 int n_tokens, int E, int top, int n_groups, int keep_groups, int group_top,
                                 int score_kind, int normalize, float norm_eps, float scale,
                                 const float* __restrict__ bias) {
  extern __shared__ float route_smem[];            // per warp: E scores, E choice scores, n_groups group scores
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * 4 + warp;
  if (t >= n_tokens) return;
  float* s = route_smem + warp * (2 * E + n_groups);
  int id;
  float weight;
  moe_route_token(logits + (size_t)t * E, s, s + E, s + 2 * E, id, weight, lane, E, top, n_groups, keep_groups, group_top,
                  score_kind, normalize, norm_eps, scale, bias);
  if (lane < top) ids[(size_t)t * top + lane] = id, wts[(size_t)t * top + lane] = weight;
}

// Eight values as they lie in memory, asked for in the order of the source.
template <typename T>
struct Moe8;
template <>
struct Moe8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "l"(p) : "memory");
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p + 4) : "memory");
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  }
};
template <>
struct Moe8<bf16> {
  uint32_t raw[4];
  __device__ __forceinline__ void load(const bf16* p) {
    asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(raw[0]), "=r"(raw[1]), "=r"(raw[2]), "=r"(raw[3]) : "l"(p) : "memory");
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[2 * i] = __uint_as_float(raw[i] << 16), v[2 * i + 1] = __uint_as_float(raw[i] & 0xffff0000u);
  }
};

__device__ __forceinline__ void moe_load8(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void moe_load8(const bf16* p, float* v) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x, v[2 * i + 1] = f.y;
  }
}

struct MoePlaces {             // what moe_sort_kernel writes, and the rows in that order (bfloat16 [P, K])
  int *perm, *dest, *tiles;
  float* sorted_weight;
  bf16* xs;
  int max_tiles, tile_rows, n_tiled;
};
#define MOE_PLACE_TOKENS 8     // a CTA each, in one cluster

// Behind the routing: own_ids/own_wts hold the `top` pairs of token t, row its values (eight a thread, the first 8 THREADS).
template <int THREADS>
__device__ __forceinline__ void moe_place(const MoePlaces pl, const int* own_ids, const float* own_wts, int* all_ids, int* count,
                                          int* place, const bf16* __restrict__ xr, uint4 row, int t, int n_tokens, int K, int E,
                                          int top) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, P = n_tokens * top;
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int i = tid; i < P; i += THREADS) {
    const int cta = i / top;
    uint32_t there;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(own_ids + (i - cta * top))), "r"(cta));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(there) : "memory");
    all_ids[i] = v;
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // (waited for at the end: others may still read)
  for (int p = warp; p < top; p += THREADS / 32) {
    const int e = own_ids[p], r = t * top + p;
    unsigned before = 0;
    for (int i = lane; i < P; i += 32) before += all_ids[i] < e || (all_ids[i] == e && i < r);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
      place[p] = (int)before;
      pl.perm[before] = r;
      pl.dest[before] = p * n_tokens + t;
      pl.sorted_weight[before] = own_wts[p];
    }
  }
  __syncthreads();
  for (int c = tid * 8; c < K; c += THREADS * 8) {
    if (c != tid * 8) row = *reinterpret_cast<const uint4*>(xr + c);
    for (int p = 0; p < top; ++p) *reinterpret_cast<uint4*>(pl.xs + (size_t)place[p] * K + c) = row;
  }
  if (t == 0) {                // the first CTA: rows and tiles of the experts, in one scan (rows below, tiles above 16 bits)
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += THREADS) {
      const int e = e0 + tid;
      int n = 0;
      for (int i = 0; i < P; ++i) n += all_ids[i] == e;
      const int mine = e < E ? n | ((e < pl.n_tiled ? (n + pl.tile_rows - 1) / pl.tile_rows : 0) << 16) : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (lane == 31) count[warp] = sum;
      __syncthreads();
      sum += carry;
      for (int w = 0; w < THREADS / 32; ++w) {
        if (w < warp) sum += count[w];
        carry += count[w];
      }
      int at = (sum - mine) & 0xffff, tl = (sum - mine) >> 16;
      if (e < E && e < pl.n_tiled)
        for (int k = 0; k < n; k += pl.tile_rows, ++tl) {
          pl.tiles[3 * tl] = e;
          pl.tiles[3 * tl + 1] = at + k;
          pl.tiles[3 * tl + 2] = min(n - k, pl.tile_rows);
        }
      __syncthreads();
    }
    for (int tl = (carry >> 16) + tid; tl < pl.max_tiles; tl += THREADS) pl.tiles[3 * tl] = -1;
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The router's product and the routing in one kernel: a CTA takes TOK tokens; warp w of n computes the float32 logits of
// experts w, w + n, ... two at a time (a lane adds its share of k in ascending order, eight consecutive k at a time, then
// the lanes are added by a butterfly: the order depends on nothing but K), then warp j routes token j.  The matrix may
// hold n_extra rows behind the experts' (a gate that reads the same input): their logits are written to extra_out
// [T, n_extra] as they are.
// Prompts: four tokens a CTA.  (Eight, and sixteen with their rows by asynchronous copies through shared memory, read
// the matrix less often and took longer: 4100 tokens, 16 experts 23.5 us by four, 29 and 24.5 by eight and sixteen; 64 experts
// 73, 87 and 77.)
// Four such CTAs an SM, where unbounded registers let two in and three leave another round: 64 experts, 2000 tokens 44 us (56 by
// three), 4100 tokens 72 (74 and 87); inside a prompt of 4100 tokens, 16 experts, 32 -> 27; float32 rows, 2000 tokens 65 (79 by three).
// Steps of few tokens wait for nothing but loads: the matrix is brought to L2 while the kernel before still runs, and sixteen
// warps share the experts.
// PLACE (steps of up to 8 tokens): the CTAs are one cluster, which knows every choice behind one barrier, so each CTA also
// finds its own pairs' places in the order by experts (what moe_sort_kernel makes in a launch of its own, with the places
// inside an expert in the order of the pairs), copies its token's row there, and the first one writes the list of tiles.
// Four tokens, top 4, K = 2048, the three launches and this one: 16 experts 9.9 and 7.8 us, 64 experts 20.1 and 12.7.  (With
// several tokens a CTA it took longer than the three from 12 tokens on: 9.7 and 9.2 us, 64 experts 17.1 and 9.3.)
template <typename TX, int TOK, int THREADS, bool PLACE>
__global__ void __launch_bounds__(THREADS, TOK == 1 ? 1 : 4)
moe_router_kernel(const TX* __restrict__ x, long long ldx, const float* __restrict__ w, int* __restrict__ ids,
                  float* __restrict__ wts, int n_tokens, int K, int E, int top, int n_groups, int keep_groups,
                  int group_top, int score_kind, int normalize, float norm_eps, float scale, int vec,
                  const float* __restrict__ bias, int n_extra, float* __restrict__ extra_out,
                  const float* __restrict__ logit_bias, int rehearse, const MoePlaces places) {
  // per token: E + n_extra logits, E scores, n_groups group scores; PLACE: this CTA's choices and weights, all choices,
  // sums of the warps, places
  extern __shared__ float route_smem[];
  constexpr int WARPS = THREADS / 32;
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = blockIdx.x * TOK;
  const int per_tok = 2 * E + n_extra + n_groups;
  const int n_rows = E + n_extra;
  if (TOK == 1) {                                  // the CTAs share the lines of the matrix among themselves
    const size_t bytes = (size_t)n_rows * K * sizeof(float);
    for (size_t at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 128; at < bytes; at += (size_t)gridDim.x * blockDim.x * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(w) + at));
  }
  const TX* x0 = x + (size_t)t0 * ldx;
  const int last = n_tokens - 1 - t0;              // (rows past the last token repeat it)
  uint4 row = {};                                  // PLACE: this thread's piece of the token's row, for its places
  // Up to 16 float32 rows of 16 warps: by eight warps in pairs, which read the token's row half as often (16 experts, K = 4096,
  // one token: 8.4 us by a row each, 7.6 like this); bfloat16 rows are read in no time.
  const int span = TOK == 1 && sizeof(TX) == 4 && n_rows > 8 && n_rows <= 16 ? 8 : WARPS;
  // rows e and, of two, e + span (a warp that has one row left does not read it twice)
  auto products = [&](int e, auto rows) {
    constexpr int Q = decltype(rows)::value;
    float acc[Q][TOK];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int j = 0; j < TOK; ++j) acc[q][j] = 0.f;
    const float* wr = w + (size_t)e * K;
    if (vec && TOK > 1) {           // K a multiple of 8 and rows 16-byte aligned: 8 consecutive k per lane and step
      constexpr int UNROLL = Q == 1 ? 2 : 1;
#pragma unroll UNROLL
      for (int k = lane * 8; k < K; k += 256) {
        float wv[Q][8], xv[TOK][8];
#pragma unroll
        for (int q = 0; q < Q; ++q) moe_load8(wr + (size_t)q * span * K + k, wv[q]);
#pragma unroll
        for (int j = 0; j < TOK; ++j) moe_load8(x0 + (size_t)min(j, last) * ldx + k, xv[j]);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
          for (int j = 0; j < TOK; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[q][j] = fmaf(xv[j][i], wv[q][i], acc[q][j]);
      }
    } else if (vec) {
      // U steps at a time, all their loads asked for before the first is used
      auto steps = [&](int k, auto count) {
        constexpr int U = decltype(count)::value;
        Moe8<float> wv[U][Q];
        Moe8<TX> xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int q = 0; q < Q; ++q) wv[u][q].load(wr + (size_t)q * span * K + k + u * 256);
          xv[u].load(x0 + k + u * 256);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float v[8], f[8];
          xv[u].get(v);
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            wv[u][q].get(f);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[q][0] = fmaf(v[i], f[i], acc[q][0]);
          }
        }
      };
      constexpr int U = 8 / Q;
      int k = lane * 8;
      for (; k + (U - 1) * 256 < K; k += U * 256) steps(k, std::integral_constant<int, U>());
      for (; k < K; k += 256) steps(k, std::integral_constant<int, 1>());
    } else {
      for (int k0 = lane * 8; k0 < K; k0 += 256)
        for (int k = k0; k < k0 + 8 && k < K; ++k)
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const float wv = wr[(size_t)q * span * K + k];
#pragma unroll
            for (int j = 0; j < TOK; ++j) acc[q][j] = fmaf(to_f32(x0[(size_t)min(j, last) * ldx + k]), wv, acc[q][j]);
          }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int j = 0; j < TOK; ++j) {
        const float v = warp_sum(acc[q][j]);
        const int row = e + span * q;
        if (lane == 0) route_smem[j * per_tok + row] = (logit_bias && row < E) ? v + logit_bias[row] : v;
      }
  };
  int* own_ids = reinterpret_cast<int*>(route_smem + TOK * per_tok);
  float* own_wts = reinterpret_cast<float*>(own_ids + TOK * top);
  // One token a CTA: the routing is run once ahead of the wait, on zeros and for nothing, so that its instructions are in the
  // SM when the step waits for them.  (Only where this kernel may start before the one ahead of it ends: launched in
  // order, four float32 rows of 2048, 16 experts, took 9.6 us with it and take 6.4.)
#pragma unroll 1
  for (int pass = TOK == 1 && rehearse ? 0 : 1; pass < 2; ++pass) {
    if (pass == 0) {
      for (int i = threadIdx.x; i < per_tok; i += THREADS) route_smem[i] = 0.f;
    } else {
      __syncthreads();
      pdl_wait();
      if constexpr (PLACE)
        if ((int)threadIdx.x * 8 < K) row = *reinterpret_cast<const uint4*>(x0 + threadIdx.x * 8);
      for (int e = warp < span ? warp : n_rows; e < n_rows; e += 2 * span) {
        if (e + span < n_rows) products(e, std::integral_constant<int, 2>());
        else products(e, std::integral_constant<int, 1>());
      }
    }
    __syncthreads();
    for (int j = warp; j < TOK && t0 + j < n_tokens; j += WARPS) {
      const int t = t0 + j;
      float* z = route_smem + j * per_tok;
      if (pass && lane < n_extra) extra_out[(size_t)t * n_extra + lane] = z[E + lane];
      // (the logits are not needed once the scores exist: their place holds the choice scores)
      int id;
      float weight;
      moe_route_token(z, z + n_rows, z, z + n_rows + E, id, weight, lane, E, top, n_groups, keep_groups, group_top, score_kind,
                      normalize, norm_eps, scale, bias, pass != 0);
      if (pass && lane < top) {
        ids[(size_t)t * top + lane] = id, wts[(size_t)t * top + lane] = weight;
        if (PLACE) own_ids[j * top + lane] = id, own_wts[j * top + lane] = weight;
      }
    }
  }
  if constexpr (PLACE) {
    int* all_ids = reinterpret_cast<int*>(own_wts + TOK * top);
    int* count = all_ids + n_tokens * top;
    moe_place<THREADS>(places, own_ids, own_wts, all_ids, count, count + WARPS, x0, row, t0, n_tokens, K, E, top);
  }
}

// x [T, K] (float32 or bfloat16, row stride ldx), w float32 [E, K] -> ids int32 [T, top], wts float32 [T, top].
// logit_bias: null, or float32 [E] added to the experts' logits before anything is made of them.
// places: null, or what to fill beside (bfloat16 rows of whole vectors, up to MOE_PLACE_TOKENS tokens).
static int moe_router(const void* x, int x_dtype, long long ldx, const float* w, int* ids, float* wts, int n_tokens, int K, int E,
                      int top, int n_groups, int keep_groups, int group_top, int score_kind, int normalize, float norm_eps,
                      float scale, const float* bias, int n_extra, float* extra_out, const float* logit_bias,
                      const MoePlaces* places, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (score_kind < MOE_SCORE_SIGMOID || score_kind > MOE_SCORE_SOFTMAX_TOP || top > 32) return LLMX_REFUSED(1);
  if (n_extra < 0 || n_extra > 32 || (n_extra > 0 && !extra_out)) return LLMX_REFUSED(1);
  if (K <= 0 || ldx < K || E <= 0 || E > MOE_MAX_EXPERTS || top <= 0 || top > MOE_MAX_TOP || n_groups <= 0 || E % n_groups ||
      keep_groups <= 0 || keep_groups > n_groups || group_top <= 0 || group_top > 8 ||
      top > E / n_groups * keep_groups)
    return LLMX_REFUSED(1);
  const int esz = x_dtype == LLMX_F32 ? 4 : 2;
  const int vec = (K % 8 == 0) && ((ldx * esz) % 16 == 0) && !((uintptr_t)x & 15) && !((uintptr_t)w & 15);
  if (places && (x_dtype != LLMX_BF16 || !vec || n_tokens > MOE_PLACE_TOKENS || ((uintptr_t)places->xs & 15) ||
                 places->tile_rows <= 0 || places->n_tiled < 0 || places->n_tiled > E ||
                 places->max_tiles < (n_tokens * top + places->tile_rows - 1) / places->tile_rows + E))
    return LLMX_REFUSED(1);
  const size_t per_tok = (size_t)(2 * E + n_extra + n_groups) * sizeof(float);
  const int tok = n_tokens <= 64 ? 1 : 4;
  const MoePlaces none = {};
  const int rehearse = llmx_pdl_allowed();
#define GO(TX, TOK, THREADS, PLACE, SMEM)                                                                                 \
  {                                                                                                                       \
    auto kernel = moe_router_kernel<TX, TOK, THREADS, PLACE>;                                                             \
    const dim3 grid((n_tokens + TOK - 1) / TOK);                                                                          \
    if (PLACE)                                                                                                            \
      launch_pdl_cluster(kernel, grid, dim3(THREADS), SMEM, stream, grid.x, (const TX*)x, ldx, w, ids, wts, n_tokens, K, E, \
                         top, n_groups, keep_groups, group_top, score_kind, normalize, norm_eps, scale, vec, bias, n_extra, \
                         extra_out, logit_bias, rehearse, *places);                                                               \
    else                                                                                                                  \
      launch_pdl(kernel, grid, dim3(THREADS), SMEM, stream, (const TX*)x, ldx, w, ids, wts, n_tokens, K, E, top, n_groups, \
                 keep_groups, group_top, score_kind, normalize, norm_eps, scale, vec, bias, n_extra, extra_out, logit_bias, \
                 rehearse, none);                                                                                             \
    return LLMX_LAUNCH_STATUS();                                                                                          \
  }
  if (places) {
    const size_t smem = per_tok + (size_t)top * 12 + (size_t)n_tokens * top * 4 + 64;      // (16 KB at most)
    GO(bf16, 1, 512, true, smem)
  }
  if (x_dtype != LLMX_F32 && x_dtype != LLMX_BF16) return LLMX_REFUSED(2);
  if (tok == 1 && x_dtype == LLMX_F32) GO(float, 1, 512, false, per_tok)
  if (tok == 1) GO(bf16, 1, 512, false, per_tok)
  if (x_dtype == LLMX_F32) GO(float, 4, 256, false, 4 * per_tok)
  GO(bf16, 4, 256, false, 4 * per_tok)
#undef GO
}

LLMX_API int llmx_moe_router_biased(const void* x, int x_dtype, long long ldx, const float* w, int* ids, float* wts,
                             int n_tokens, int K, int E, int top, int n_groups, int keep_groups, int group_top,
                             int score_kind, int normalize, float norm_eps, float scale, const float* bias,
                             int n_extra, float* extra_out, const float* logit_bias, cudaStream_t stream) {
  return moe_router(x, x_dtype, ldx, w, ids, wts, n_tokens, K, E, top, n_groups, keep_groups, group_top, score_kind, normalize,
                    norm_eps, scale, bias, n_extra, extra_out, logit_bias, nullptr, stream);
}

// The router, the order of the pairs by expert (perm, dest, sorted_weight [P], tiles, as llmx_moe_sort makes them) and the
// tokens' rows in that order (xs [P, K], as llmx_moe_gather_rows makes them) in one launch: bfloat16 rows, up to 8 tokens.
LLMX_API int llmx_moe_router_placed(const void* x, long long ldx, const float* w, int* ids, float* wts, int n_tokens, int K,
                                    int E, int top, int n_groups, int keep_groups, int group_top, int score_kind, int normalize,
                                    float norm_eps, float scale, const float* bias, int n_extra, float* extra_out,
                                    const float* logit_bias, int* perm, int* dest, float* sorted_weight, int* tiles,
                                    int max_tiles, int tile_rows, int n_tiled, void* xs, cudaStream_t stream) {
  if (!perm || !dest || !sorted_weight || !tiles || !xs) return LLMX_REFUSED(4);
  const MoePlaces places = {perm, dest, tiles, sorted_weight, (bf16*)xs, max_tiles, tile_rows, n_tiled};
  return moe_router(x, LLMX_BF16, ldx, w, ids, wts, n_tokens, K, E, top, n_groups, keep_groups, group_top, score_kind, normalize,
                    norm_eps, scale, bias, n_extra, extra_out, logit_bias, &places, stream);
}

LLMX_API int llmx_moe_router(const void* x, int x_dtype, long long ldx, const float* w, int* ids, float* wts,
                             int n_tokens, int K, int E, int top, int n_groups, int keep_groups, int group_top,
                             int score_kind, int normalize, float norm_eps, float scale, const float* bias,
                             int n_extra, float* extra_out, cudaStream_t stream) {
  return llmx_moe_router_biased(x, x_dtype, ldx, w, ids, wts, n_tokens, K, E, top, n_groups, keep_groups, group_top,
                                score_kind, normalize, norm_eps, scale, bias, n_extra, extra_out, nullptr, stream);
}

LLMX_API int llmx_moe_route(const float* logits, int* ids, float* wts, int n_tokens, int E, int top, int n_groups,
                            int keep_groups, int group_top, int score_kind, int normalize, float norm_eps,
                            float scale, const float* bias, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (E <= 0 || E > MOE_MAX_EXPERTS || top <= 0 || top > MOE_MAX_TOP || top > 32 || n_groups <= 0 || E % n_groups ||
      keep_groups <= 0 || keep_groups > n_groups || group_top <= 0 || group_top > 8 ||
      top > E / n_groups * keep_groups)
    return LLMX_REFUSED(1);
  const size_t smem = 4 * (size_t)(2 * E + n_groups) * sizeof(float);
  launch_pdl(moe_route_kernel, dim3((n_tokens + 3) / 4), dim3(128), smem, stream, logits, ids, wts, n_tokens, E, top,
             n_groups, keep_groups, group_top, score_kind, normalize, norm_eps, scale, bias);
  return LLMX_LAUNCH_STATUS();
}

// ---------------------------------------------------------------------------
// Sort.  One CTA.  P = n_tokens * top pairs, pair r = t * top + choice.  Out: perm[P] (sorted place -> pair),
// tiles: for every row tile of tile_rows sorted rows that lie in one expert's segment, (expert, first row,
// number of rows); the used tiles come first, unused ones have expert -1.  max_tiles >= P / tile_rows + E.
// Experts n_tiled..E-1 have no products (identity experts): their pairs are placed but get no tiles.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int* __restrict__ ids, const float* __restrict__ pair_weight, int P, int E, int top,
                int n_tokens, int* __restrict__ perm, int* __restrict__ dest, float* __restrict__ sorted_weight,
                int* __restrict__ tiles, int max_tiles, int tile_rows, int n_tiled) {
  __shared__ int count[MOE_MAX_EXPERTS];
  __shared__ int start[MOE_MAX_EXPERTS + 1];
  __shared__ int tile0[MOE_MAX_EXPERTS + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  for (int e = tid; e < E; e += blockDim.x) count[e] = 0;
  __syncthreads();
  // (an expert id outside 0..E-1 cannot come from this library's routing; it is reported, code 2, and counted as the
  // last expert, so that no index leaves its array)
  for (int r = tid; r < P; r += blockDim.x) {
    int e = ids[r];
    if ((unsigned)e >= (unsigned)E) {
      llmx_report(2);
      e = E - 1;
    }
    atomicAdd(&count[e], 1);
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0, tl = 0;
    for (int e = 0; e < E; ++e) {
      start[e] = at;
      tile0[e] = tl;
      at += count[e];
      if (e < n_tiled) tl += (count[e] + tile_rows - 1) / tile_rows;
    }
    start[E] = at;
    tile0[E] = tl;
  }
  __syncthreads();
  for (int e = tid; e < E; e += blockDim.x) {
    const int n = count[e];
    for (int k = 0, tl = tile0[e]; k < n && e < n_tiled; k += tile_rows, ++tl) {
      tiles[3 * tl] = e;
      tiles[3 * tl + 1] = start[e] + k;
      tiles[3 * tl + 2] = (n - k) < tile_rows ? (n - k) : tile_rows;
    }
    count[e] = 0;          // reused as the segment's fill counter
  }
  for (int tl = tile0[E] + tid; tl < max_tiles; tl += blockDim.x) tiles[3 * tl] = -1;
  __syncthreads();
  for (int r = tid; r < P; r += blockDim.x) {
    int e = ids[r];
    if ((unsigned)e >= (unsigned)E) e = E - 1;
    const int place = start[e] + atomicAdd(&count[e], 1);
    perm[place] = r;
    if (dest) {             // where the pair's result goes in [top, n_tokens, ...], and its weight, in sorted order
      const int t = r / top;
      dest[place] = (r - t * top) * n_tokens + t;
      sorted_weight[place] = pair_weight[r];
    }
  }
}

// dest, sorted_weight (both [P]) may be null; with them pair_weight [P], top and n_tokens are needed.
LLMX_API int llmx_moe_sort(const int* ids, const float* pair_weight, int P, int E, int top, int n_tokens, int* perm,
                           int* dest, float* sorted_weight, int* tiles, int max_tiles, int tile_rows, int n_tiled,
                           cudaStream_t stream) {
  if (P <= 0) return 0;
  if (n_tiled < 0 || n_tiled > E) return LLMX_REFUSED(1);
  if (E <= 0 || E > MOE_MAX_EXPERTS || tile_rows <= 0 || max_tiles < (P + tile_rows - 1) / tile_rows + E)
    return LLMX_REFUSED(1);
  if (dest && (!sorted_weight || !pair_weight || top <= 0 || n_tokens <= 0)) return LLMX_REFUSED(4);
  launch_pdl(moe_sort_kernel, dim3(1), dim3(P >= 4096 ? 1024 : 256), 0, stream, ids, pair_weight, P, E, top, n_tokens,
             perm, dest, sorted_weight, tiles, max_tiles, tile_rows, n_tiled);
  return LLMX_LAUNCH_STATUS();
}

// ---------------------------------------------------------------------------
// Grouped products on the FMA units (float32 accumulation, k = 0..K-1 per output element).
//
// GATED: rows are tokens' rows of x gathered through perm (token = pair / top); W = [E][2F][K], gate rows then
//   up rows; out act[place][f] = gated_act(gate, up) (common.cuh), in sorted order.
// PLAIN: the same rows; W = [E][F][K]; out act[place][f] = the activation of an expert without a gate.
// else:  rows are act[place]; W = [E][N][K]; out y[choice][token][n] = weight[pair] * sum, float32: one partial
//   per choice, which whoever adds them to the residual stream sums in the order of the choices.
// ---------------------------------------------------------------------------
template <typename TX, typename TW, typename TY, bool GATED, bool PLAIN>
__global__ void __launch_bounds__(256)
moe_grouped_fma_kernel(const TX* __restrict__ X, long long ldx, const TW* __restrict__ W, TY* __restrict__ Y,
                       const int* __restrict__ perm, const int* __restrict__ tiles,
                       const float* __restrict__ pair_weight, int top, int n_tokens, int N, int K, const GateAct act) {
  __shared__ float Xs[MOE_BK][MOE_TILE + 4];
  __shared__ float Ws[MOE_BK][MOE_TILE + 4];
  __shared__ float Us[GATED ? MOE_BK : 1][MOE_TILE + 4];
  __shared__ int row_src[MOE_TILE];
  pdl_launch_dependents();
  pdl_wait();
  const int tl = blockIdx.y;
  const int e = tiles[3 * tl];
  if (e < 0) return;
  const int row0 = tiles[3 * tl + 1], n_rows = tiles[3 * tl + 2];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int n0 = blockIdx.x * MOE_TILE;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;
  if (tid < MOE_TILE) row_src[tid] = tid < n_rows ? perm[row0 + tid] : -1;
  __syncthreads();
  const int pair = row_src[lrow];
  const TX* xrow = nullptr;
  if (pair >= 0) xrow = GATED || PLAIN ? X + (size_t)(pair / top) * ldx : X + (size_t)(row0 + lrow) * ldx;
  const size_t w_rows = GATED ? 2 * (size_t)N : (size_t)N;
  const TW* We = W + (size_t)e * w_rows * K;
  const int n_load = n0 + lrow;
  const TW* wrow = n_load < N ? We + (size_t)n_load * K : nullptr;
  const TW* urow = (GATED && n_load < N) ? We + ((size_t)N + n_load) * K : nullptr;

  float acc[4][4], acu[GATED ? 4 : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[i][j] = 0.f;
      if constexpr (GATED) acu[i][j] = 0.f;
    }
  for (int k0 = 0; k0 < K; k0 += MOE_BK) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int k = k0 + lk + c;
      Xs[lk + c][lrow] = (xrow && k < K) ? to_f32(xrow[k]) : 0.f;
      Ws[lk + c][lrow] = (wrow && k < K) ? to_f32(wrow[k]) : 0.f;
      if constexpr (GATED) Us[lk + c][lrow] = (urow && k < K) ? to_f32(urow[k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MOE_BK; ++kk) {
      float a[4], b[4], u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = Xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b[j] = Ws[kk][tx * 4 + j];
        if constexpr (GATED) u[j] = Us[kk][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
          if constexpr (GATED) acu[i][j] = fmaf(a[i], u[j], acu[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = ty * 4 + i;
    const int pr = row_src[lr];
    if (pr < 0) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      if constexpr (GATED) {
        Y[(size_t)(row0 + lr) * N + n] = from_f32<TY>(gated_act(act, acc[i][j], acu[i][j]));
      } else if constexpr (PLAIN) {
        Y[(size_t)(row0 + lr) * N + n] = from_f32<TY>(plain_act(act, acc[i][j]));
      } else {
        const int t = pr / top, choice = pr - t * top;
        Y[((size_t)choice * n_tokens + t) * N + n] = from_f32<TY>(pair_weight[pr] * acc[i][j]);
      }
    }
  }
}

// gated 1: X = x [n_tokens, K] (row stride ldx), W [E, 2N, K], Y = act [P, N]; gated 2: W [E, N, K] without a gate.
// gated 0:       X = act [P, K], W [E, N, K], Y = float32 [top, n_tokens, N].
// The tile list must have been made with MOE_TILE rows per tile.
LLMX_API int llmx_moe_grouped_fma(const void* X, int x_dtype, long long ldx, const void* W, int w_dtype, void* Y,
                                  int y_dtype, const int* perm, const int* tiles, int max_tiles,
                                  const float* pair_weight, int top, int n_tokens, int N, int K, int gated,
                                  int act_kind, float slope, float limit, float shift, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (act_kind < LLMX_ACT_SILU || act_kind > (gated == 2 ? LLMX_ACT_LAST_PLAIN : LLMX_ACT_LAST)) return LLMX_REFUSED(1);
  const GateAct act = {act_kind, slope, limit, shift};
  if (N <= 0 || K <= 0 || top <= 0 || max_tiles <= 0 || max_tiles > 65535 || ldx < K) return LLMX_REFUSED(1);
  if (x_dtype != w_dtype) return LLMX_REFUSED(2);
  dim3 grid((N + MOE_TILE - 1) / MOE_TILE, max_tiles);
#define GO(TX, TY, G, P)                                                                                       \
  launch_pdl(moe_grouped_fma_kernel<TX, TX, TY, G, P>, grid, dim3(256), 0, stream, (const TX*)X, ldx, (const TX*)W, \
             (TY*)Y, perm, tiles, pair_weight, top, n_tokens, N, K, act)
  if (gated) {
    if (gated < 0 || gated > 2) return LLMX_REFUSED(1);
    const bool plain = gated == 2;
    if (x_dtype == LLMX_F32 && y_dtype == LLMX_F32) {
      if (plain) GO(float, float, false, true); else GO(float, float, true, false);
    } else if (x_dtype == LLMX_BF16 && y_dtype == LLMX_BF16) {
      if (plain) GO(bf16, bf16, false, true); else GO(bf16, bf16, true, false);
    } else {
      return LLMX_REFUSED(2);
    }
  } else {
    if (y_dtype != LLMX_F32) return LLMX_REFUSED(2);
    if (x_dtype == LLMX_F32) GO(float, float, false, false);
    else if (x_dtype == LLMX_BF16) GO(bf16, float, false, false);
    else return LLMX_REFUSED(2);
  }
#undef GO
  return LLMX_LAUNCH_STATUS();
}

// ---------------------------------------------------------------------------
// Identity experts and a gated shared expert, both written as further partials of the feed-forward's result, in
// one launch.
//
// CTAs 0 .. T*top-1, one per pair (t, choice): if the pair's expert id is >= n_real (an identity expert, whose
//   output is its input), y[choice][t][:] = weight * x[t][:]; pairs of real experts are left alone.
// CTAs T*top .. T*top+T-1 (with a shared expert), one per token: y[top][t][:] = sigmoid(z[t * ldz]) * sum_p
//   shared[p][t][:], the shared expert's result times one number per token.
// ---------------------------------------------------------------------------
template <typename TX, typename TS, int VEC>
__global__ void __launch_bounds__(256)
moe_extras_kernel(const TX* __restrict__ x, long long ldx, const int* __restrict__ ids, const float* __restrict__ wts,
                  float* __restrict__ y, int n_tokens, int top, int d, int n_real, const TS* __restrict__ shared,
                  int n_split, size_t split_stride, const float* __restrict__ z, int ldz) {
  pdl_launch_dependents();
  pdl_wait();
  const int n_pairs = n_tokens * top;
  if ((int)blockIdx.x < n_pairs) {
    const int pair = blockIdx.x;
    if (ids[pair] < n_real) return;
    const int t = pair / top, choice = pair - t * top;
    const float w = wts[pair];
    const TX* xr = x + (size_t)t * ldx;
    float* yr = y + ((size_t)choice * n_tokens + t) * d;
    for (int i = threadIdx.x * VEC; i < d; i += blockDim.x * VEC) {
      if (VEC == 8) {
        float v[8];
        moe_load8(xr + i, v);
        *reinterpret_cast<float4*>(yr + i) = make_float4(w * v[0], w * v[1], w * v[2], w * v[3]);
        *reinterpret_cast<float4*>(yr + i + 4) = make_float4(w * v[4], w * v[5], w * v[6], w * v[7]);
      } else {
        yr[i] = w * to_f32(xr[i]);
      }
    }
    return;
  }
  const int t = blockIdx.x - n_pairs;
  const float gate = z ? 1.0f / (1.0f + expf(-z[(size_t)t * ldz])) : 1.0f;      // no logit: the result joins as it is
  float* yr = y + ((size_t)top * n_tokens + t) * d;
  for (int i = threadIdx.x * VEC; i < d; i += blockDim.x * VEC) {
    if (VEC == 8) {
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int p = 0; p < n_split; ++p) {
        float a[8];
        moe_load8(shared + (size_t)p * split_stride + (size_t)t * d + i, a);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += a[e];
      }
      *reinterpret_cast<float4*>(yr + i) = make_float4(gate * v[0], gate * v[1], gate * v[2], gate * v[3]);
      *reinterpret_cast<float4*>(yr + i + 4) = make_float4(gate * v[4], gate * v[5], gate * v[6], gate * v[7]);
    } else {
      float v = 0.f;
      for (int p = 0; p < n_split; ++p) v += to_f32(shared[(size_t)p * split_stride + (size_t)t * d + i]);
      yr[i] = gate * v;
    }
  }
}

// x [T, d] (row stride ldx); ids, wts [T, top]; y float32 [top (+1), T, d]; identity experts are ids >= n_real
// (n_real >= all ids: none).  shared: null, or the shared expert's result [T, d] as n_split partials, with z (one
// float per token, ldz apart) the logit of its gate, or null for no gate.
LLMX_API int llmx_moe_extras(const void* x, int x_dtype, long long ldx, const int* ids, const float* wts, float* y,
                             int n_tokens, int top, int d, int n_real, const void* shared, int shared_dtype, int n_split,
                             long long split_stride, const float* z, int ldz, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (top <= 0 || d <= 0 || ldx < d || (shared && ((z && ldz < 1) || n_split < 1))) return LLMX_REFUSED(1);
  const dim3 grid((unsigned)n_tokens * top + (shared ? (unsigned)n_tokens : 0u));
  // eight columns per thread and load where every row starts on a 32-byte boundary
  const bool vec = d % 8 == 0 && ldx % 8 == 0 && split_stride % 8 == 0 &&
                   !(((uintptr_t)x | (uintptr_t)y | (uintptr_t)shared) & 31);
  const int threads = d >= 2048 ? 256 : 128;
#define GO(TX, TS)                                                                                                      \
  do {                                                                                                                  \
    if (vec)                                                                                                            \
      launch_pdl(moe_extras_kernel<TX, TS, 8>, grid, dim3(threads), 0, stream, (const TX*)x, ldx, ids, wts, y, n_tokens, \
                 top, d, n_real, (const TS*)shared, n_split, (size_t)split_stride, z, ldz);                             \
    else                                                                                                                \
      launch_pdl(moe_extras_kernel<TX, TS, 1>, grid, dim3(threads), 0, stream, (const TX*)x, ldx, ids, wts, y, n_tokens, \
                 top, d, n_real, (const TS*)shared, n_split, (size_t)split_stride, z, ldz);                             \
  } while (0)
  const int key = x_dtype * 2 + (shared ? shared_dtype : LLMX_F32);
  switch (key) {
    case 0: GO(float, float); break;
    case 1: GO(float, bf16); break;
    case 2: GO(bf16, float); break;
    case 3: GO(bf16, bf16); break;
    default: return LLMX_REFUSED(2);
  }
#undef GO
  return LLMX_LAUNCH_STATUS();
}

// ---------------------------------------------------------------------------
// Routing by a table: a token's experts are row `token id` of an integer table [vocab, top], each with the same
// weight.  An id outside the vocabulary or an expert outside [0, E) is reported (code 3) and expert 0 stands in,
// so that nothing later indexes with it.
// ---------------------------------------------------------------------------
__global__ void moe_table_route_kernel(const int* __restrict__ tokens, const int* __restrict__ table, int vocab,
                                       int E, int top, float weight, int* __restrict__ ids, float* __restrict__ wts,
                                       int n_tokens) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tokens * top) return;
  const int t = i / top, k = i % top;
  const int tok = tokens[t];
  int e = 0;
  if (tok < 0 || tok >= vocab) {
    llmx_report(3);
  } else {
    e = table[(size_t)tok * top + k];
    if (e < 0 || e >= E) {
      llmx_report(3);
      e = 0;
    }
  }
  ids[i] = e;
  wts[i] = weight;
}

LLMX_API int llmx_moe_table_route(const int* tokens, const int* table, int vocab, int E, int top, float weight, int* ids,
                                  float* wts, int n_tokens, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (vocab <= 0 || E <= 0 || top <= 0 || top > E) return LLMX_REFUSED(1);
  const int n = n_tokens * top;
  launch_pdl(moe_table_route_kernel, dim3((n + 127) / 128), dim3(128), 0, stream, tokens, table, vocab, E, top, weight,
             ids, wts, n_tokens);
  return LLMX_LAUNCH_STATUS();
}
