// Matrix product on the FMA units: Y[M,N] = X[M,K] * W[N,K]^T with float32
// accumulation and no reduced-precision mode of any kind.  It is the matrix
// product of the true 32-bit path (gemm_f32_kernel), and the fallback of the
// bfloat16 path for shapes the tensor-core kernel refuses (K not a multiple of
// 8) and for weights that the checkpoint stores in 32-bit (gemm_fma_kernel).
//
// y[t,o] = sum_i W[o,i] x[t,i], W row-major [out, in]
// (crates/model/src/ops.rs:83-101).  Every output element is accumulated by
// one thread in an order that K alone decides, so a row's result does not
// depend on M, on the tile it falls into or on what else is in the batch.
#include "common.cuh"

// ---------------------------------------------------------------------------
// float32 x float32 -> float32.  K is cut into segments of F32_SEG.  Within a segment an element has two chains, one
// over the even and one over the odd k, each from the segment's first k up and added at its end: the two halves of one
// packed multiply-add (fma.rn.f32x2), whose operands are neighbouring k as they lie in memory, so nothing is transposed or
// duplicated on the way.  The segments' sums are added in their order.  Both kernels follow that order.
// ---------------------------------------------------------------------------
#define F32_SEG 512

// BYTES from global to shared memory; where not valid nothing is read and zeros are written
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const float* src, bool valid) {
  const int n = valid ? BYTES : 0;
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(unsigned long long v) {          // the even chain plus the odd one
  return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}
// One thread's share of the copies of a [ROWS x BK] block of a row-major matrix into rows BK + 4 floats apart, VEC floats a
// copy: the thread keeps its columns, walks down the rows, and moves on by whole k blocks, so that a copy costs an
// addition.  Rows past the matrix and columns past K read nothing and give zeros.
template <int ROWS, int BK, int VEC>
struct BlockCopy {
  static constexpr int PER_ROW = BK / VEC, STEP = PER_ROW < 128 ? 128 / PER_ROW : 1, N = (ROWS + STEP - 1) / STEP;
  static_assert(128 % PER_ROW == 0, "a thread keeps its columns");
  const float* src;            // this thread's first element of the block at k = 0
  long long row_step;
  uint32_t to;                 // its place in the block, bytes
  int k, live;                 // its column; how many of its rows exist
  __device__ __forceinline__ BlockCopy(const float* matrix, long long ld, int row0, int rows) {
    const int r = (int)threadIdx.x / PER_ROW;
    k = ((int)threadIdx.x % PER_ROW) * VEC;
    live = row0 + r < rows && r < ROWS ? (min(rows - row0, ROWS) - r + STEP - 1) / STEP : 0;
    src = matrix + (live ? (size_t)(row0 + r) * ld + k : 0);
    row_step = live > 1 ? STEP * ld : 0;
    to = (uint32_t)(r * (BK + 4) + k) * 4u;
  }
  __device__ __forceinline__ void operator()(uint32_t block, int k0, int K) const {
    const int n = k0 + k < K ? live : 0;
    const float* p = n ? src + k0 : src;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (ROWS % STEP && (int)threadIdx.x / PER_ROW + i * STEP >= ROWS) break;
      copy_async<VEC * 4>(block + to + (uint32_t)(i * STEP * (BK + 4) * 4), p, i < n);
      if (i + 1 < n) p += row_step;
    }
  }
};

// Prompts: 128 threads as 8 (tokens) x 16 (features), TM x TN elements each.  Rows in shared memory are 20 floats apart,
// so eight rows read at the same k lie in different banks; 8 x 8 elements take 16 shared-memory reads per 128 packed
// multiply-adds.  The sums of earlier segments wait in shared memory.  Bound by the FMA units and the reads that feed
// them.  970 tokens, N = K = 2048: 231 us (35 TFLOP/s;
// the one-chain 64 x 64 kernel that this replaced: 16 TFLOP/s); 2500 tokens, N = 4096: 971 us (43 TFLOP/s).
// SHARED: where the tiles are too few for the SMs, a cluster's CTAs take a segment of K each and add the segments' sums in
// their order through distributed shared memory, so the bits are those of one CTA.  N = K = 2048: 40 tokens 49.7 -> 34.8 us,
// 100 tokens 96.8 -> 38.6, 256 tokens 126 -> 64.4; 970 tokens, N = 3072: 345 -> 327.
template <int TM, int TN>
struct F32Tile {
  static constexpr int BM = 8 * TM, BN = 16 * TN, BK = 16, STAGES = 4, PITCH = BK + 4;
  static constexpr int STAGE = (BM + BN) * PITCH;                      // floats
  static constexpr int TOTAL_PITCH = BN + 8;
  static constexpr size_t SMEM = ((size_t)STAGES * STAGE + (size_t)BM * TOTAL_PITCH) * sizeof(float);
};

template <int TM, int TN, int VEC, bool SHARED>
__global__ void __launch_bounds__(128, TM * TN >= 64 ? 2 : 4)
gemm_f32_tile_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N, int K,
                     long long ldx, long long ldw, long long ldy, int n_tiles, int n_seg) {
  using Tile = F32Tile<TM, TN>;
  constexpr int BM = Tile::BM, BN = Tile::BN, BK = Tile::BK, STAGES = Tile::STAGES, PITCH = Tile::PITCH, STAGE = Tile::STAGE;
  extern __shared__ __align__(16) float tiles[];                      // per stage: W [BN][PITCH], X [BM][PITCH]; totals
  float* totals = tiles + STAGES * STAGE;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(tiles);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tn = (warp & 1) * 8 + (lane & 7), tm = (warp >> 1) * 4 + (lane >> 3);      // 16 x 8
  const int rank = SHARED ? (int)blockIdx.x % n_seg : 0, tile = SHARED ? (int)blockIdx.x / n_seg : (int)blockIdx.x;
  const int n0 = (tile % n_tiles) * BN, m0 = (tile / n_tiles) * BM;
  const int k_first = rank * F32_SEG, n_kb = ((SHARED ? min(K - k_first, F32_SEG) : K) + BK - 1) / BK;
  const BlockCopy<BN, BK, VEC> copy_w(W, ldw, n0, N);
  const BlockCopy<BM, BK, VEC> copy_x(X, ldx, m0, M);
  auto load = [&](int kb) {
    const uint32_t dst = base + (uint32_t)((kb % STAGES) * STAGE) * 4u;
    copy_w(dst, k_first + kb * BK, K);
    copy_x(dst + (uint32_t)(BN * PITCH) * 4u, k_first + kb * BK, K);
  };
  pdl_launch_dependents();
  pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_kb) load(s);
    copy_commit();
  }
  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  for (int kb = 0; kb < n_kb; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                           // tile kb is there, and everyone is done with the stage that is filled next
    if (kb + STAGES - 1 < n_kb) load(kb + STAGES - 1);
    copy_commit();
    const float* ws = tiles + (kb % STAGES) * STAGE + tn * PITCH;
    const float* xs = tiles + (kb % STAGES) * STAGE + BN * PITCH + tm * PITCH;
    constexpr int UNROLL = TM * TN >= 64 ? 1 : BK / 4;        // (8 x 8: the next reads' registers would be spilled)
#pragma unroll UNROLL
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * 8 * PITCH + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * 16 * PITCH + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].y, b.y);
      }
    }
    if (!SHARED && (kb + 1) % (F32_SEG / BK) == 0 && kb + 1 < n_kb) {           // a segment ends and another follows
      const bool first = kb + 1 == F32_SEG / BK;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          float* t = totals + (i * 8 + tm) * Tile::TOTAL_PITCH + j * 16 + tn;          // this thread's own word
          *t = first ? both(acc[i][j]) : __fadd_rn(*t, both(acc[i][j]));
          acc[i][j] = 0ull;
        }
    }
  }
  if (SHARED) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) totals[(i * 8 + tm) * Tile::TOTAL_PITCH + j * 16 + tn] = both(acc[i][j]);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t own = (uint32_t)__cvta_generic_to_shared(totals);
    uint32_t there[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there[q]) : "r"(own), "r"(min(q, n_seg - 1)));
    for (int r = rank; r < BM && m0 + r < M; r += n_seg)              // rows of the tile, a row's segments in their order
      for (int c = threadIdx.x; c < BN; c += 128) {
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < n_seg)
            asm volatile("ld.shared::cluster.f32 %0, [%1];"
                         : "=f"(v[q]) : "r"(there[q] + (uint32_t)(r * Tile::TOTAL_PITCH + c) * 4u) : "memory");
#pragma unroll
        for (int q = 1; q < 8; ++q)
          if (q < n_seg) v[0] = __fadd_rn(v[0], v[q]);
        if (n0 + c < N) Y[(size_t)(m0 + r) * ldy + n0 + c] = v[0];
      }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // nobody leaves while its sums may be read
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + i * 8 + tm;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + j * 16 + tn;
      const float v = both(acc[i][j]);
      if (n < N)
        Y[(size_t)m * ldy + n] = K > F32_SEG ? __fadd_rn(totals[(i * 8 + tm) * Tile::TOTAL_PITCH + j * 16 + tn], v) : v;
    }
  }
}

// Few tokens (up to 2 MT a CTA): 16 features, four segments of K at a time.  Thread (feature f, segment g, token half h)
// follows its feature's chain over segment g for MT tokens, so a value of W is read from shared memory once per token
// half and the tokens' values are broadcasts; a quarter of the chain's length and four streams of each row are what a
// row costs.  The first lines of W travel to L2 before the kernel before has ended.  Four tokens, K = 2048: 10 us at
// N = 2048 (the 64 x 64 kernel, 32 CTAs with one chain of 2048 steps: 184 us a product), 25 us at N = 8192 (2.7 TB/s);
// bound by the latency of a CTA's first tiles at the former, by that and the reads of X at the latter.
template <int MT>
struct F32Rows {
  static constexpr int BM = 2 * MT, BN = 16, GROUPS = 4, BK = 32, PITCH = BK + 4;
  static constexpr int STAGES = 6;
  static constexpr int STAGE = GROUPS * (BN + BM) * PITCH;             // floats
  static constexpr size_t SMEM = ((size_t)STAGES * STAGE + GROUPS * BN * BM) * sizeof(float);
};

template <int MT, int VEC>
__global__ void __launch_bounds__(128)
gemm_f32_rows_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N, int K,
                     long long ldx, long long ldw, long long ldy, int n_tiles) {
  using Rows = F32Rows<MT>;
  constexpr int BM = Rows::BM, BN = Rows::BN, G = Rows::GROUPS, BK = Rows::BK, PITCH = Rows::PITCH, STAGES = Rows::STAGES;
  constexpr int STAGE = Rows::STAGE, PER_SEG = F32_SEG / BK;
  extern __shared__ __align__(16) float tiles[];           // per stage: W [G][BN][PITCH], X [G][BM][PITCH]; segment sums
  float* sums = tiles + STAGES * STAGE;                    // [G][BM][BN]
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(tiles);
  const int f = threadIdx.x & 15, g = (threadIdx.x >> 4) & 3, h = threadIdx.x >> 6;
  const int n0 = (blockIdx.x % n_tiles) * BN, m0 = (blockIdx.x / n_tiles) * BM;
  const int n_seg = (K + F32_SEG - 1) / F32_SEG, n_rounds = (n_seg + G - 1) / G;
  // step i: k block i % PER_SEG of the segments of round i / PER_SEG; a last round of one segment ends where K does
  const int n_steps = n_seg % G == 1 ? (n_rounds - 1) * PER_SEG + (K - (n_seg - 1) * F32_SEG + BK - 1) / BK : n_rounds * PER_SEG;
  const BlockCopy<BN, BK, VEC> copy_w(W, ldw, n0, N);
  const BlockCopy<BM, BK, VEC> copy_x(X, ldx, m0, M);
  auto load_w = [&](int i) {
#pragma unroll
    for (int q = 0; q < G; ++q)
      copy_w(base + (uint32_t)((i % STAGES) * STAGE + q * BN * PITCH) * 4u,
             ((i / PER_SEG) * G + q) * F32_SEG + (i % PER_SEG) * BK, K);
  };
  auto load_x = [&](int i) {
#pragma unroll
    for (int q = 0; q < G; ++q)
      copy_x(base + (uint32_t)((i % STAGES) * STAGE + (G * BN + q * BM) * PITCH) * 4u,
             ((i / PER_SEG) * G + q) * F32_SEG + (i % PER_SEG) * BK, K);
  };
  pdl_launch_dependents();
  // W may be what the kernel before writes, so nothing of it is read ahead of that kernel's end; its lines are asked for as
  // far as L2, where that kernel's stores arrive too
  for (int i = threadIdx.x; i < (STAGES - 1) * G * BN; i += 128) {
    const int k = (i / BN % G) * F32_SEG + (i / (G * BN)) * BK, n = n0 + i % BN;
    if (n < N && k < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)n * ldw + k));
  }
  pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_steps) load_w(s), load_x(s);
    copy_commit();
  }
  unsigned long long acc[MT];
  float total[MT];                                         // (group 0 keeps the totals of its feature)
#pragma unroll
  for (int i = 0; i < MT; ++i) acc[i] = 0ull, total[i] = 0.f;
  auto join = [&](int round) {                             // the round's segments join the totals in their order
#pragma unroll
    for (int i = 0; i < MT; ++i) sums[(g * BM + 2 * i + h) * BN + f] = both(acc[i]), acc[i] = 0ull;
    __syncthreads();
    if (g == 0) {
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const float* t = sums + (2 * i + h) * BN + f;
        total[i] = round == 0 ? *t : __fadd_rn(total[i], *t);
        for (int q = 1; q < G && round * G + q < n_seg; ++q) total[i] = __fadd_rn(total[i], t[q * BM * BN]);
      }
    }
    __syncthreads();
  };
  constexpr int UNROLL = MT == 2 ? 1 : 2;                  // (by measurement: 16 tokens 13.5 us at N = 256, K = 2048, 15.3 without; 4 tokens 7.5, 8.8 with)
#pragma unroll UNROLL
  for (int step = 0; step < n_steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    if (step + STAGES - 1 < n_steps) load_w(step + STAGES - 1), load_x(step + STAGES - 1);
    copy_commit();
    const float* ws = tiles + (step % STAGES) * STAGE + (g * BN + f) * PITCH;
    const float* xs = tiles + (step % STAGES) * STAGE + (G * BN + g * BM + h) * PITCH;   // token i of this thread: row 2 i + h
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + k);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + 2 * i * PITCH + k);
        fma2(acc[i], a.x, b.x), fma2(acc[i], a.y, b.y);
      }
    }
    if ((step + 1) % PER_SEG == 0) join(step / PER_SEG);
  }
  if (n_steps % PER_SEG) join(n_rounds - 1);
  if (g == 0 && n0 + f < N) {
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const int m = m0 + 2 * i + h;
      if (m < M) Y[(size_t)m * ldy + n0 + f] = total[i];
    }
  }
}

// One launch of a kernel whose CTAs own BM tokens x BN features.
template <typename Shape, typename Kernel, typename... More>
static int launch_f32(Kernel kernel, bool& attr_set, const float* X, const float* W, float* Y, int M, int N, int K,
                      long long ldx, long long ldw, long long ldy, cudaStream_t stream, int cluster, More... more) {
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const long long n_tiles = (N + Shape::BN - 1) / Shape::BN, m_tiles = (M + Shape::BM - 1) / Shape::BM;
  if (n_tiles * m_tiles * cluster > 0x7fffffff) return LLMX_REFUSED(3);
  const dim3 grid((unsigned)(n_tiles * m_tiles * cluster));
  if (cluster > 1)
    launch_pdl_cluster(kernel, grid, dim3(128), Shape::SMEM, stream, (unsigned)cluster, X, W, Y, M, N, K, ldx, ldw, ldy,
                       (int)n_tiles, more...);
  else
    launch_pdl(kernel, grid, dim3(128), Shape::SMEM, stream, X, W, Y, M, N, K, ldx, ldw, ldy, (int)n_tiles, more...);
  return LLMX_LAUNCH_STATUS();
}

// The float32 product by a launch of the caller's choice (tests: every one gives the same bits); -1: by the rule.
// 0..3: rows kernel with 2, 4, 8, 16 tokens a CTA; 4: tiles of 32 x 64; 5: tiles of 64 x 128; 6, 7: the same, a cluster's
// CTAs with a segment of K each (2 to 8 segments).
#define F32_N_FORMS 8
LLMX_API int llmx_gemm_f32_form(int form, const float* X, const float* W, float* Y, int M, int N, int K, long long ldx,
                                long long ldw, long long ldy, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || ldx < K || ldw < K || ldy < N || form >= F32_N_FORMS) return LLMX_REFUSED(1);
  if ((M + 63) / 64 > 65535) return LLMX_REFUSED(3);
  const int n_seg = (K + F32_SEG - 1) / F32_SEG;
  if (form >= 6 && (n_seg < 2 || n_seg > 8)) return LLMX_REFUSED(1);
  if (form < 0) {
    // Rule: the cheapest by what was measured over K = 64 to 8192, N = 64 to 8192 and 1 to 2500 tokens (us beside a launch's
    // 1.5, on 148 SMs; CTAs are counted by the SM).  A step of 32 k in four segments costs a round of two CTAs of rows an SM 0.6,
    // 0.65, 0.75 or 1.1 (2, 4, 8, 16 tokens); 16 k cost a round of one tile of 32 x 64 an SM 0.26 (few tiles an SM cannot hide
    // their waits: 0.41, 0.6, 1.01 and 1.1 at one to four), one of 64 x 128 0.88 (1.17 at least).  Up to 512 k only one
    // segment's threads work in the rows kernel, so tiles win there from few tokens on: 16 tokens, N = 8192, K = 256: 18 us by
    // rows, 9.3 by tiles; N = 2048, K = 2048: 19 and 50.
    // Tiles that share K cost by the CTA, not by the round: their clusters are of all sizes.  32 x 64: 14 and 8.8 for every CTA an
    // SM, 20 at least (a round of rows that the rule puts at 17.6 takes 13, such tiles 16 to 18) and 40 beyond two an SM.  64 x 128:
    // 57 up to one an SM, 69 up to the 1.73 that run at once (clusters do not fill every GPC), then 32 and 32.9 for every
    // one; many clusters of four, which fill the GPCs better than three, six and eight do, 15 and 30.6.  What the fit puts less
    // than 3 % below another form is within its error and stays with that form (many clusters of four are taken as fitted).
    // Up to 16 tokens rows are cheaper than the rule thinks (9 tokens, N = 2048, K = 4096: 28 us, 35 by the rule, 31
    // shared).  64 tokens, N = 2048, K = 1024: 18.9 us shared, 26.6 not; 33 tokens, N = 8192, K = 2048: 64 and 91; 400 tokens,
    // N = 8192, K = 3000: 613 and 574.  Over 621 shapes the rule's choice took 1.007 times the best form's time.
    const auto rounds = [](long long n, int m) { return (double)((n + m - 1) / m); };
    const auto tiles = [&](int bm, int bn) { return (long long)rounds(M, bm) * (long long)rounds(N, bn); };
    const int sms = llmx_sm_count();
    const double steps = (n_seg / 4) * 16 + (n_seg % 4 == 1 ? (K - (n_seg - 1) * F32_SEG + 31) / 32 : n_seg % 4 ? 16 : 0);
    const double blocks = (K + 15) / 16;
    const int few = M <= 2 ? 0 : M <= 4 ? 1 : M <= 8 ? 2 : 3;
    const double a_step[4] = {0.6, 0.65, 0.75, 1.1};
    const double rows = a_step[few] * steps * rounds(tiles(2 << few, 16), 2 * sms);
    const double r = rounds(tiles(32, 64), sms);
    const double small = blocks * (r <= 1 ? 0.41 : r <= 2 ? 0.6 : fmax(0.26 * r, fmin(0.11 + 0.3 * r, 1.1)));
    const double large = blocks * fmax(0.88 * rounds(tiles(64, 128), sms), 1.17);
    double best = rows;
    form = few;
    const auto take = [&](int f, double us) {
      if (us < best) best = us, form = f;
    };
    take(4, small);
    take(5, large);
    if (M > 16 && n_seg >= 2 && n_seg <= 8) {
      const double fit = 1.03, c6 = (double)n_seg * (double)tiles(32, 64) / sms, c7 = (double)n_seg * (double)tiles(64, 128) / sms;
      take(6, fit * fmax(14.0 + 8.8 * c6, c6 > 2.0 ? 40.0 : 20.0));
      take(7, c7 > 6.76 && n_seg == 4 ? 15.0 + 30.6 * c7 : fit * (c7 <= 1.0 ? 57.0 : c7 <= 1.73 ? 69.0 : 32.0 + 32.9 * c7));
    }
  }
  // 16-byte copies where every row starts on a 16-byte boundary and K ends on one, else 4-byte copies
  const bool wide = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && !((uintptr_t)X & 15) && !((uintptr_t)W & 15);
#define GO(SHAPE, CLUSTER, KERNEL, ...)                                                                             \
  {                                                                                                                 \
    static bool set = false;                                                                                        \
    return launch_f32<SHAPE>(KERNEL, set, X, W, Y, M, N, K, ldx, ldw, ldy, stream, CLUSTER, ##__VA_ARGS__);          \
  }
#define ROWS(MT)                                                                                                    \
  {                                                                                                                 \
    using S = F32Rows<MT>;                                                                                          \
    if (wide) GO(S, 1, (gemm_f32_rows_kernel<MT, 4>)) else GO(S, 1, (gemm_f32_rows_kernel<MT, 1>))                    \
  }
#define TILE(TM, TN, SHARED)                                                                                        \
  {                                                                                                                 \
    using S = F32Tile<TM, TN>;                                                                                      \
    if (wide) GO(S, SHARED ? n_seg : 1, (gemm_f32_tile_kernel<TM, TN, 4, SHARED>), n_seg)                             \
    else GO(S, SHARED ? n_seg : 1, (gemm_f32_tile_kernel<TM, TN, 1, SHARED>), n_seg)                                  \
  }
  switch (form) {
    case 0: ROWS(1)
    case 1: ROWS(2)
    case 2: ROWS(4)
    case 3: ROWS(8)
    case 4: TILE(4, 4, false)
    case 5: TILE(8, 8, false)
    case 6: TILE(4, 4, true)
    case 7: TILE(8, 8, true)
  }
#undef TILE
#undef ROWS
#undef GO
  return LLMX_REFUSED(1);
}

// ---------------------------------------------------------------------------
// The other types: one chain per element, k = 0..K-1.
// ---------------------------------------------------------------------------
#define FMA_BM 64
#define FMA_BN 64
#define FMA_BK 16

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256)
gemm_fma_kernel(const TX* __restrict__ X, const TW* __restrict__ W, TY* __restrict__ Y, int M, int N, int K,
                long long ldx, long long ldw, long long ldy) {
  __shared__ float Xs[FMA_BK][FMA_BM + 4];
  __shared__ float Ws[FMA_BK][FMA_BN + 4];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * FMA_BM, n0 = blockIdx.x * FMA_BN;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += FMA_BK) {
    {
      const int m = m0 + lrow, n = n0 + lrow;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int k = k0 + lk + c;
        Xs[lk + c][lrow] = (m < M && k < K) ? to_f32(X[(size_t)m * ldx + k]) : 0.f;
        Ws[lk + c][lrow] = (n < N && k < K) ? to_f32(W[(size_t)n * ldw + k]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < FMA_BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = Xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) Y[(size_t)m * ldy + n] = from_f32<TY>(acc[i][j]);
    }
  }
}

LLMX_API int llmx_gemm_fma(const void* X, int x_dtype, const void* W, int w_dtype, void* Y, int y_dtype, int M,
                           int N, int K, long long ldx, long long ldw, long long ldy, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || ldx < K || ldw < K || ldy < N) return LLMX_REFUSED(1);
  dim3 grid((N + FMA_BN - 1) / FMA_BN, (M + FMA_BM - 1) / FMA_BM);
  if (grid.y > 65535) return LLMX_REFUSED(3);
#define CASE(TX, TW, TY) \
  launch_pdl(gemm_fma_kernel<TX, TW, TY>, grid, dim3(256), 0, stream, (const TX*)X, (const TW*)W, (TY*)Y, M, N, K, ldx, ldw, ldy)
  const int key = x_dtype * 4 + w_dtype * 2 + y_dtype;
  switch (key) {
    case 0: return llmx_gemm_f32_form(-1, (const float*)X, (const float*)W, (float*)Y, M, N, K, ldx, ldw, ldy, stream);
    case 1: CASE(float, float, bf16); break;
    case 2: CASE(float, bf16, float); break;
    case 3: CASE(float, bf16, bf16); break;
    case 4: CASE(bf16, float, float); break;
    case 5: CASE(bf16, float, bf16); break;
    case 6: CASE(bf16, bf16, float); break;
    case 7: CASE(bf16, bf16, bf16); break;
    default: return LLMX_REFUSED(2);
  }
#undef CASE
  return LLMX_LAUNCH_STATUS();
}
