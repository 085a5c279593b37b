// Recurrences over a matrix state walked in chunks of 64 tokens: what the kernels of state_space.cu and linear_attention.cu
// share.  Chunks of a sequence are counted from its first token of the step.
#pragma once

#include "common.cuh"

#define SS_CHUNK 64

__device__ __forceinline__ float4 ss_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void ss_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// Slots of sequence b in units of `unit` tokens start at seq_start[b] / unit + b: the last b whose first slot is <= slot.
__device__ __forceinline__ int ss_find_seq(const int* seq_start, int n_seqs, int slot, int unit) {
  int lo = 0, hi = n_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (seq_start[mid] / unit + mid <= slot) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// acc[r][c] += sum_k A[k][row r] B[k][col c]: K rows of 64 results in shared memory, 128 threads, 4 x 8 results each, on the
// tensor cores in float32 precision.  An operand is split in two 11-bit parts that TF32 holds, x = hi + lo up to 2^-23 of x,
// and lo hi, hi lo and hi hi are added (lo lo is below 2^-24 of the product), the small ones first; the tensor core adds eight
// k at a time from zero, and those sums join acc by float32 additions, so that what its adder cuts off (towards zero, the same
// way every time) is cut off once.  Sums over 32 k inside it were off by 1.6 times as much as the FMA units' chains.
// A warp owns 32 rows and 32 columns.  Which row and column of a fragment stands for which of the tile is free, so it is
// chosen such that a thread reads four neighbouring rows or columns at once and owns rows i0 .. i0+3 and columns j0 .. j0+7;
// with rows of shared memory SS_LD floats apart no read meets a bank twice.
// Rows of A and B are there, and zero, up to the next multiple of 8 behind K.
// An operand that is not finite has no such parts: it is left out, and joins by float32 multiply-adds, so that it reaches the
// results of its own row or column and leaves the others' bits alone.
// ---------------------------------------------------------------------------
#define SS_THREADS 128
#define SS_LD 72
__device__ __forceinline__ int ss_row0() { return (threadIdx.x >> 6) * 32 + ((threadIdx.x & 31) >> 2) * 4; }
__device__ __forceinline__ int ss_col0() { return ((threadIdx.x >> 5) & 1) * 32 + (threadIdx.x & 3) * 8; }
__device__ __forceinline__ void ss_split(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;     // (rounded: what lo then lacks has no preferred sign)
  lo = __float_as_uint(x - __uint_as_float(hi));         // (the tensor core takes the upper 19 bits)
}
__device__ __forceinline__ void ss_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ bool ss_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ float4 ss_finite4(float4 v) {
  return make_float4(ss_finite(v.x) ? v.x : 0.f, ss_finite(v.y) ? v.y : 0.f, ss_finite(v.z) ? v.z : 0.f, ss_finite(v.w) ? v.w : 0.f);
}
// first_row: row k of A is zero for results of rows below k + first_row, which do not see row k of B whatever it holds (a
// masked matrix, whose rows from 32 on are all that K rows behind first_row 32 reach; else -64: every row sees it).
__device__ __forceinline__ void ss_product(float (&acc)[4][8], const float* A, const float* B, int K, int first_row = -64) {
  if (first_row >= 32 && threadIdx.x < 64) return;       // (warps of the rows below 32)
  const float* ap = A + (threadIdx.x & 3) * SS_LD + ss_row0();
  const float* bp = B + (threadIdx.x & 3) * SS_LD + ((threadIdx.x >> 5) & 1) * 32 + ((threadIdx.x & 31) >> 2) * 4;
#pragma unroll 1
  for (int k = 0; k < K; k += 8) {
    uint32_t ah[2][4], al[2][4], bh[2][4], bl[2][4];
    float4 u[2], v[2];
    float zero = 0.f;                                    // (a part lo that is not finite makes it NaN)
#pragma unroll
    for (int q = 0; q < 2; ++q) u[q] = ss_load4(ap + (k + 4 * q) * SS_LD), v[q] = ss_load4(bp + (k + 4 * q) * SS_LD);
    auto split = [&]() {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        ss_split(u[q].x, ah[0][2 * q], al[0][2 * q]), ss_split(u[q].y, ah[0][2 * q + 1], al[0][2 * q + 1]);
        ss_split(u[q].z, ah[1][2 * q], al[1][2 * q]), ss_split(u[q].w, ah[1][2 * q + 1], al[1][2 * q + 1]);
        ss_split(v[q].x, bh[q][0], bl[q][0]), ss_split(v[q].y, bh[q][1], bl[q][1]);
        ss_split(v[q].z, bh[q][2], bl[q][2]), ss_split(v[q].w, bh[q][3], bl[q][3]);
      }
    };
    split();
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        zero = fmaf(__uint_as_float(al[i][e]), 0.f, zero);
        zero = fmaf(__uint_as_float(bl[i][e]), 0.f, zero);
      }
    const bool finite = __all_sync(0xffffffffu, zero == 0.f);
    if (!finite) {
#pragma unroll
      for (int q = 0; q < 2; ++q) u[q] = ss_finite4(u[q]), v[q] = ss_finite4(v[q]);
      split();
    }
    // rows i0 + 2 i + half are fragment rows g + 8 half of i, columns 4 n + j its column n of j
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float sum[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[j][e] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) ss_mma(sum[j], al[i], bh[0][j], bh[1][j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) ss_mma(sum[j], ah[i], bl[0][j], bl[1][j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) ss_mma(sum[j], ah[i], bh[0][j], bh[1][j]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float& to = acc[i * 2 + (e >> 1)][(e & 1) * 4 + j];
          to = __fadd_rn(to, sum[j][e]);
        }
    }
    if (!finite)
      for (int kk = k; kk < min(K, k + 8); ++kk)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float m = A[kk * SS_LD + ss_row0() + r];
          if (ss_row0() + r < kk + first_row) continue;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float x = B[kk * SS_LD + ss_col0() + c];
            if (!ss_finite(m) || !ss_finite(x)) acc[r][c] = fmaf(m, x, acc[r][c]);
          }
        }
  }
}
// ---------------------------------------------------------------------------
// The same on the FMA units (where a few products weigh most, one chain rounds less than the tensor core's sums cut off: the
// state of the state-space recurrence): K rows of 64 results in shared memory, 64 threads, 8 x 8 results each, so that
// the four 16-byte reads a thread makes per k (512 bytes a warp each, 128 a cycle) last as long as its 64 multiply-adds.
// A thread's rows are i0 .. i0+3 and i0+32 .. i0+35, its columns j0 .. j0+3 and j0+32 .. j0+35: neighbouring lanes read
// neighbouring 16 bytes.
// ---------------------------------------------------------------------------
#define SS_FMA_THREADS 64
__device__ __forceinline__ int ss_fma_row0() { return (threadIdx.x >> 3) * 4; }
__device__ __forceinline__ int ss_fma_col0() { return (threadIdx.x & 7) * 4; }
// Two multiply-adds in one instruction, each rounded like fmaf: (d.x, d.y) += a * (b.x, b.y).
__device__ __forceinline__ void ss_fma2(float& dx, float& dy, float a, float bx, float by) {
  asm("{\n.reg .b64 va, vb, vd;\nmov.b64 va, {%2, %2};\nmov.b64 vb, {%3, %4};\nmov.b64 vd, {%0, %1};\n"
      "fma.rn.f32x2 vd, va, vb, vd;\nmov.b64 {%0, %1}, vd;\n}"
      : "+f"(dx), "+f"(dy)
      : "f"(a), "f"(bx), "f"(by));
}
template <int UNROLL>
__device__ __forceinline__ void ss_product_fma(float (&acc)[8][8], const float* A, int lda, const float* B, int ldb, int K) {
  const float* ap = A + ss_fma_row0();
  const float* bp = B + ss_fma_col0();
#pragma unroll UNROLL
  for (int k = 0; k < K; ++k) {
    const float4 a0 = ss_load4(ap + k * lda), a1 = ss_load4(ap + k * lda + 32);
    const float4 b0 = ss_load4(bp + k * ldb), b1 = ss_load4(bp + k * ldb + 32);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 8; c += 2) ss_fma2(acc[r][c], acc[r][c + 1], av[r], bv[c], bv[c + 1]);
  }
}
__device__ __forceinline__ int ss_fma_row(int i0, int r) { return i0 + (r & 3) + ((r & 4) << 3); }   // the r-th of a thread's rows
__device__ __forceinline__ void ss_copy16(float* dst, const float* src, bool live) {             // 16 bytes, or zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(live ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void ss_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ss_copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The chunk of a slot: its sequence, first token, number of tokens (0: none) and number within the sequence.
struct SsChunk {
  int b, t0, n, index;
};
// Sequences that bring no more than `short_new` tokens have none.
__device__ __forceinline__ SsChunk ss_chunk_of(const int* seq_start, int n_seqs, int n_tokens, int slot, int short_new = 0) {
  SsChunk k;
  k.b = ss_find_seq(seq_start, n_seqs, slot, SS_CHUNK);
  const int row0 = seq_start[k.b], n_new = seq_start[k.b + 1] - row0;
  k.index = slot - (row0 / SS_CHUNK + k.b);
  k.t0 = row0 + k.index * SS_CHUNK;
  k.n = min(SS_CHUNK, n_new - k.index * SS_CHUNK);
  if (k.index < 0 || row0 < 0 || row0 + n_new > n_tokens || n_new <= short_new) k.n = 0;
  return k;
}
