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
// acc[r][c] += sum_k A[k][row r] B[k][col c]: K rows of 64 results in shared memory, 64 threads, 8 x 8 results each, so that
// the four 16-byte reads a thread makes per k (512 bytes a warp each, 128 a cycle) last as long as its 64 multiply-adds.
// A thread's rows are i0 .. i0+3 and i0+32 .. i0+35, its columns j0 .. j0+3 and j0+32 .. j0+35: neighbouring lanes read
// neighbouring 16 bytes.
// ---------------------------------------------------------------------------
#define SS_THREADS 64
__device__ __forceinline__ int ss_row0() { return (threadIdx.x >> 3) * 4; }
__device__ __forceinline__ int ss_col0() { return (threadIdx.x & 7) * 4; }
// Two multiply-adds in one instruction, each rounded like fmaf: (d.x, d.y) += a * (b.x, b.y).
__device__ __forceinline__ void ss_fma2(float& dx, float& dy, float a, float bx, float by) {
  asm("{\n.reg .b64 va, vb, vd;\nmov.b64 va, {%2, %2};\nmov.b64 vb, {%3, %4};\nmov.b64 vd, {%0, %1};\n"
      "fma.rn.f32x2 vd, va, vb, vd;\nmov.b64 {%0, %1}, vd;\n}"
      : "+f"(dx), "+f"(dy)
      : "f"(a), "f"(bx), "f"(by));
}
// LOW false: only the rows from 32 on (a triangle's lower half has nothing above).
template <int UNROLL, bool LOW = true>
__device__ __forceinline__ void ss_product(float (&acc)[8][8], const float* A, int lda, const float* B, int ldb, int K) {
  const float* ap = A + ss_row0();
  const float* bp = B + ss_col0();
#pragma unroll UNROLL
  for (int k = 0; k < K; ++k) {
    const float4 a0 = LOW ? ss_load4(ap + k * lda) : make_float4(0.f, 0.f, 0.f, 0.f), a1 = ss_load4(ap + k * lda + 32);
    const float4 b0 = ss_load4(bp + k * ldb), b1 = ss_load4(bp + k * ldb + 32);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int r = LOW ? 0 : 4; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 8; c += 2) ss_fma2(acc[r][c], acc[r][c + 1], av[r], bv[c], bv[c + 1]);
  }
}
__device__ __forceinline__ int ss_row(int i0, int r) { return i0 + (r & 3) + ((r & 4) << 3); }   // the r-th of a thread's rows
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
