// Linear attention with a fixed decay per head (no softmax, no denominator), as a recurrence over a
// per-sequence state, and the normalisation and gate that follow it.
//
//   S_t = decay_h * S_{t-1} + k_t v_t^T        S: [D, Dv] per (sequence, head), float32, kept from step to step
//   o_t = S_t^T q_t
//
// q, k and v come out of one fused projection (a row holds q heads, k heads, v heads and the gate's columns).
// What the design does to them before the recurrence is done by a kernel of its own, once per (token, head):
// an activation (none or SiLU), the rotation of q and k (pairs (i, i + n_rot/2) of a head's first n_rot dims,
// angle from float32 tables), a scale on k.  All of it, the state and the sums are float32.
//
// The recurrence is independent for every column of v, so a CTA owns `cols` columns of one (sequence, head)
// and walks that sequence's tokens of the step in order.  Within a CTA a warp owns 4 or 8 columns; the 8 lanes of
// a column (or of two neighbouring ones) split D among them in blocks of 4 dims (lane r owns dims 4 (r + 8 i) + 0..3),
// update their part of S and add up q . S by shuffles.  The order of every addition is fixed by (d, column) alone, and a
// token's update is the same arithmetic whether it arrives in a prompt, in a later portion of one or alone, so
// among steps that bring a sequence up to seg_len tokens a position's result does not depend on how tokens were cut into
// steps or batched, to the last bit.  Longer prompts go in segments or by chunks (below), whose sums are ordered by where
// those begin: the same for every batch, but rounded differently when a prompt is cut differently.
//
// The same kernels run a recurrence whose decay and input weight change from token to token (the matrix memory
// of an mLSTM layer, GATED below):
//
//   m_t = max(f_t + m_{t-1}, i_t)                            f, i: log forget and log input gate; m starts at 0
//   S_t = a_t S_{t-1} + b_t k_t v_t^T,  a_t = exp(f_t + m_{t-1} - m_t),  b_t = exp(i_t - m_t)
//   n_t = a_t n_{t-1} + b_t k_t
//   o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + den_eps)
//
// n is carried as one more column of S whose "value" is 1 for every token, so n_t . q_t comes out as one more
// output column; a small kernel of its own walks the gates of a (sequence, head) in order, keeps m, and leaves
// (a_t, b_t, exp(-m_t), the product of a over the token's segment so far) for every token.
//
// Work per token and head is 3 D Dv float32 operations (a multiply for k v, one fused multiply-add for the
// state, one for the output), which is what the FMA units are for; the state is read and written once per
// step, which is what bounds a decode step.
//
// A sequence that brings more than seg_len tokens under a fixed decay, with a state of at least 64 x 64, is walked in
// chunks of 64 tokens instead.  With E the state a chunk starts from,
//   o_i = decay^(i+1) E^T q_i + sum_(j<=i) decay^(i-j) (q_i . k_j) v_j,   E' = decay^n E + sum_j decay^(n-1-j) k_j v_j^T
// which is the recurrence written out as products of small matrices (chunk_products.cuh, as the state-space layers walk
// theirs): as many multiply-adds, but 8 x 8 results a thread share what they read from shared memory.
//   decay_chunk   per (chunk, head): the chunk's own part of E', and the 64 x 64 products q_i . k_j
//   decay_pass    walks a sequence's chunks in order: leaves every chunk its E and the sequence its new state
//   decay_out     per (chunk, head, 64 columns): the outputs
// Four prompts of 700 to 1300 tokens, 16 heads of 128 x 128: 255 us, where the recurrence in segments took 586 (two
// passes); off the 64-bit result by 2.7e-7 (3.4e-7).
#include "chunk_products.cuh"

#define LA_CHUNK 8           // tokens per staged chunk
#define LA_STAGES 3          // chunks in flight or in use
#define LA_SEG 128           // tokens per segment of a long prompt
#define LA_MAX_D 256

enum { LA_ACT_NONE = 0, LA_ACT_SILU = 1, LA_ACT_SIGMOID = 2 };

__device__ __forceinline__ float la_act(float x, int act) {
  if (act == LA_ACT_SILU) return x / (1.0f + expf(-x));
  if (act == LA_ACT_SIGMOID) return 1.0f / (1.0f + expf(-x));
  return x;
}

// value of column c of token row t: one tensor, or split partials added in order
template <typename TIN>
__device__ __forceinline__ float la_value(const TIN* row, int c, int n_split, size_t split_stride) {
  float v = to_f32(row[c]);
  for (int s = 1; s < n_split; ++s) v += to_f32(row[s * split_stride + c]);
  return v;
}

// Before the recurrence: what the design does to q, k and v, once per (token, head), into float32 rows
// prep[t][h] = (q[Dp], k[Dp], v[Dvp]) with Dp, Dvp the sizes rounded up to 4 (the padding is zero).
template <typename TIN>
__global__ void __launch_bounds__(128)
decay_prep_kernel(const TIN* __restrict__ proj, int n_split, size_t split_stride, size_t row_stride, int q_off,
                  int k_off, int v_off, float* __restrict__ prep, const int* __restrict__ token_pos,
                  const float* __restrict__ cos_t, const float* __restrict__ sin_t, int n_rot, int act, float k_scale,
                  float q_scale, int v_ones, int H, int D, int Dv) {
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y;
  const int Dp = (D + 3) & ~3, Dvp = (Dv + v_ones + 3) & ~3;   // v_ones: one more column of v that is 1
  const int pos = token_pos[t], half = n_rot >> 1;
  pdl_wait();
  const TIN* row = proj + (size_t)t * row_stride;
  const TIN* qrow = row + q_off + h * D;
  const TIN* krow = row + k_off + h * D;
  const TIN* vrow = row + v_off + h * Dv;
  float* out = prep + ((size_t)t * H + h) * (size_t)(2 * Dp + Dvp);
  for (int d = threadIdx.x; d < Dp; d += blockDim.x) {
    float qv = 0.f, kv = 0.f;
    if (d < D) {
      qv = la_act(la_value(qrow, d, n_split, split_stride), act);
      kv = la_act(la_value(krow, d, n_split, split_stride), act);
      if (d < n_rot) {
        const int i = d < half ? d : d - half;
        const float c = cos_t[(size_t)pos * half + i], s = sin_t[(size_t)pos * half + i];
        const int partner = d < half ? d + half : d - half;
        const float qp = la_act(la_value(qrow, partner, n_split, split_stride), act);
        const float kp = la_act(la_value(krow, partner, n_split, split_stride), act);
        // (u, v) -> (u cos - v sin, v cos + u sin) for the pair (i, i + half)
        qv = d < half ? qv * c - qp * s : qv * c + qp * s;
        kv = d < half ? kv * c - kp * s : kv * c + kp * s;
      }
      kv *= k_scale;
      qv *= q_scale;
    }
    out[d] = qv;
    out[Dp + d] = kv;
  }
  for (int c = threadIdx.x; c < Dvp; c += blockDim.x)
    out[2 * Dp + c] = c < Dv ? la_act(la_value(vrow, c, n_split, split_stride), act) : (c == Dv && v_ones) ? 1.f : 0.f;
}

// Four neighbouring elements, a vector a partial; partials are added in order, seven asked for together.
__device__ __forceinline__ void la_load(const float* p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
}
__device__ __forceinline__ void la_load(const bf16* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(u.x << 16), v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = __uint_as_float(u.y << 16), v[3] = __uint_as_float(u.y & 0xffff0000u);
}
template <typename TIN>
__device__ __forceinline__ void la_values(const TIN* p, int n_split, size_t split_stride, float (&v)[4]) {
  la_load(p, v);
  for (int s0 = 1; s0 < n_split; s0 += 7) {
    float t[7][4];
#pragma unroll
    for (int s = 0; s < 7; ++s)
      if (s0 + s < n_split) la_load(p + (size_t)(s0 + s) * split_stride, t[s]);
#pragma unroll
    for (int s = 0; s < 7; ++s)
      if (s0 + s < n_split)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += t[s][i];
  }
}

// The same by four neighbouring dims a thread (sizes, rotated dims halved, offsets and strides all multiples of 4, whole
// vectors, no column of ones): what decay_prep_kernel read and wrote an element at a time.  A thread takes the same piece of
// TOKS tokens (2 in prompts, whose loads are then under way together).  Bound by the rows it writes: 4100 tokens, 16 heads of
// 128: 72 us an element a thread, 36 like this (150 MB, 23 us at the copy's rate); with four tokens a thread and room for
// partials in the same instance 107 (registers).  Four tokens in a decode step: 4.4 -> 2.5 us.
template <typename TIN, int TOKS, bool SPLIT>
__global__ void __launch_bounds__(128)
decay_prep_vec_kernel(const TIN* __restrict__ proj, int n_split, size_t split_stride, size_t row_stride, int q_off, int k_off,
                      int v_off, float* __restrict__ prep, const int* __restrict__ token_pos, const float* __restrict__ cos_t,
                      const float* __restrict__ sin_t, int n_rot, int act, float k_scale, float q_scale, int n_tokens, int H,
                      int D, int Dv) {
  pdl_launch_dependents();
  // a head's pieces: of q and of k the pairs (i, i + half) of the rotated dims, then the other dims; then v
  const unsigned half = n_rot >> 1, pairs = half >> 2, per = pairs + ((D - n_rot) >> 2), pieces = 2 * per + (Dv >> 2);
  const unsigned idx = blockIdx.x * 128u + threadIdx.x, gh = idx / pieces, piece = idx - gh * pieces, t0 = gh / H * TOKS, h = gh % H;
  pdl_wait();
  if (t0 >= (unsigned)n_tokens) return;
  // where the piece comes from and goes to, in its token's row and its head's
  const bool is_v = piece >= 2 * per, is_k = !is_v && piece >= per;
  const unsigned q = is_v ? piece - 2 * per : is_k ? piece - per : piece;
  const bool rotated = !is_v && q < pairs;
  const unsigned d = is_v || rotated ? q * 4 : n_rot + (q - pairs) * 4;
  const TIN* src = proj + (is_v ? v_off + h * Dv : (is_k ? k_off : q_off) + h * D) + d;
  float* dst = prep + (size_t)h * (2 * D + Dv) + (is_v ? 2 * D : is_k ? D : 0) + d;
  const float scale = is_v ? 1.f : is_k ? k_scale : q_scale;
  const size_t to_step = (size_t)H * (2 * D + Dv);
  auto put = [](float* to, const float (&v)[4]) { *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]); };
  float x[TOKS][4], y[TOKS][4], c[TOKS][4], sn[TOKS][4];
#pragma unroll
  for (int j = 0; j < TOKS; ++j) {
    const unsigned t = min(t0 + j, (unsigned)n_tokens - 1);
    const TIN* from = src + (size_t)t * row_stride;
    if (SPLIT) la_values(from, n_split, split_stride, x[j]);
    else la_load(from, x[j]);
    if (rotated) {
      if (SPLIT) la_values(from + half, n_split, split_stride, y[j]);
      else la_load(from + half, y[j]);
      const size_t at = (size_t)token_pos[t] * half + d;
      la_load(cos_t + at, c[j]);
      la_load(sin_t + at, sn[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < TOKS; ++j) {
    if (t0 + j >= (unsigned)n_tokens) break;
    float* to = dst + (size_t)(t0 + j) * to_step;
    if (rotated) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float u = la_act(x[j][i], act), w = la_act(y[j][i], act);
        x[j][i] = (u * c[j][i] - w * sn[j][i]) * scale;
        y[j][i] = (w * c[j][i] + u * sn[j][i]) * scale;
      }
      put(to + half, y[j]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[j][i] = la_act(x[j][i], act) * scale;
    }
    put(to, x[j]);
  }
}

__device__ __forceinline__ void la_cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void la_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void la_cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The recurrence over the prepared rows.  Chunks of LA_CHUNK tokens come into a ring of LA_STAGES buffers by
// 16-byte asynchronous copies, two chunks ahead of the one being walked.
//
// A long prompt is cut into segments of seg_len tokens that run side by side (a sequence alone would keep only
// H * Dv / cols CTAs busy).  PASS 1: every segment runs the recurrence, the first from the stored state, the
// others from zero, and leaves its last state in `partial` (a sequence of one segment writes the state itself).
// PASS 2, for the segments after the first: the state the segment should have started from, E, is put together
// from the segments before it (E_0 = partial_0, E_s = decay^seg_len E_(s-1) + partial_s); a token i of the
// segment then lacks decay^(i+1) E^T q_i, which is added to its output; the last segment also writes the
// sequence's new state.  Segments are counted from the step's first token of a sequence, so a sum may be
// rounded differently when a prompt is cut differently; a step of up to seg_len tokens per sequence (every
// decode step) is the plain recurrence.
// DPT: dims of D per thread (a multiple of 4; 8 threads share a column, so D <= 8 DPT).
// GATED: decay and input weight per token from `gates` [T, H, 4] = (a, b, exp(-m), product of a over the segment
// up to and including the token) instead of the head's fixed decay.  head_stride: floats from one head's state to
// the next (a design may keep more than S there).
// C: neighbouring columns a thread owns.  Two (some prompts: the rule is at the launch): q and k then cost half as many
// shared-memory reads a multiply-add, which is what one column a thread waits for (the multiply-adds are packed in pairs of
// dims), and the shares of a chunk's eight tokens are added so that each of the eight lanes ends with one token's sum (7
// shuffles a column instead of 24).  Steps of few tokens stream the state and want the threads: one column.  Both, and a
// chunk cut short, make the same additions in the same order.
__device__ __forceinline__ void la_fma2(unsigned long long& d, unsigned long long a, unsigned long long b, unsigned long long c) {
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
}
__device__ __forceinline__ unsigned long long la_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long la_pair(float x, float y) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float la_lo(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float la_hi(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

template <int DPT, int PASS, bool GATED, int C>
__global__ void __launch_bounds__(256)
decay_scan_kernel(const float* __restrict__ prep, float* __restrict__ out, float* __restrict__ state,
                  float* __restrict__ partial, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                  const float* __restrict__ decay, const float* __restrict__ gates, size_t head_stride, int H, int D,
                  int Dv, int cols, int col_blocks, int seg_len, int n_seg_max, int by_chunks) {
  extern __shared__ __align__(16) float la_smem[];
  const int Dp = (D + 3) & ~3, Dvp = (Dv + 3) & ~3;
  const int row_len = 2 * Dp + Dvp;               // floats per (token, head) of prep
  const int tok_len = 2 * Dp + cols + (GATED ? 4 : 0);   // floats per staged token: q, k, this CTA's columns of v, gates
  pdl_launch_dependents();
  const int b = blockIdx.z, h = blockIdx.y;
  const int seg = blockIdx.x / col_blocks, c0 = (blockIdx.x - seg * col_blocks) * cols;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cw = (warp * 4 + (lane >> 3)) * C;    // this thread's first column of the CTA's
  const int col = c0 + cw;                        // and of v
  const int r = lane & 7;                         // its share of D
  const bool col_live = col < Dv;
  const int seq_t0 = seq_start[b], seq_new = seq_start[b + 1] - seq_t0;
  const int n_seg = (seq_new + seg_len - 1) / seg_len;        // this sequence's segments
  const float g = GATED ? 1.f : decay[h];
  float* S = state + ((size_t)seq_slot[b] * H + h) * head_stride;
  if (seg >= n_seg || (PASS == 2 && (n_seg == 1 || seg == 0)) || (by_chunks && n_seg > 1)) {       // (uniform over the CTA)
    pdl_wait();                        // (a kernel whose CTAs all leave must not end before the one ahead of it)
    return;
  }
  const int t0 = seq_t0 + seg * seg_len;                                      // the segment's first token
  const int n_new = min(seg_len, seq_new - seg * seg_len);
  float* part_seq = partial ? partial + ((size_t)b * H + h) * (size_t)n_seg_max * D * Dv : nullptr;
  if (PASS == 1 && seg == 0)           // this CTA's columns of the state, on their way to L2 while the kernel before runs
    for (int d = tid; d < D; d += blockDim.x) prefetch_l2(S + (size_t)d * Dv + c0);
  pdl_wait();

  auto own = [&](int i) { return 4 * (r + 8 * (i >> 2)) + (i & 3); };        // dim of this thread's i-th state value
  float s_reg[C == 1 ? DPT : 1];                                             // one column: its values
  unsigned long long s2[C][C == 1 ? 1 : DPT / 2];                            // two: their values in pairs of neighbouring dims
  if constexpr (C == 1) {
    if (PASS == 1) {
#pragma unroll
      for (int i = 0; i < DPT; ++i) s_reg[i] = (seg == 0 && col_live && own(i) < D) ? S[(size_t)own(i) * Dv + col] : 0.f;
    } else {
      // E_(seg-1): what the segments before left, each decayed over the segments after it
      float g_seg = 1.f;
      if (!GATED)
        for (int i = 0; i < seg_len; ++i) g_seg *= g;
#pragma unroll
      for (int i = 0; i < DPT; ++i) s_reg[i] = 0.f;
      for (int sp = 0; sp < seg; ++sp) {
        const float* ps = part_seq + (size_t)sp * D * Dv;
        if (GATED) g_seg = __ldcg(gates + ((size_t)(seq_t0 + (sp + 1) * seg_len - 1) * H + h) * 4 + 3);   // over all of segment sp
#pragma unroll
        for (int i = 0; i < DPT; ++i)
          if (col_live && own(i) < D) s_reg[i] = fmaf(g_seg, s_reg[i], __ldcg(ps + (size_t)own(i) * Dv + col));
      }
    }
  } else {
    if (PASS == 1) {
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int i = 0; i < DPT; i += 2) {
          const bool live = seg == 0 && col + c < Dv;
          s2[c][i >> 1] = la_pair(live && own(i) < D ? S[(size_t)own(i) * Dv + col + c] : 0.f,
                                  live && own(i + 1) < D ? S[(size_t)own(i + 1) * Dv + col + c] : 0.f);
        }
    } else {
      // E_(seg-1): what the segments before left, each decayed over the segments after it
      float g_seg = 1.f;
      if (!GATED)
        for (int i = 0; i < seg_len; ++i) g_seg *= g;
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int i = 0; i < DPT / 2; ++i) s2[c][i] = 0ull;
      for (int sp = 0; sp < seg; ++sp) {
        const float* ps = part_seq + (size_t)sp * D * Dv;
        if (GATED) g_seg = __ldcg(gates + ((size_t)(seq_t0 + (sp + 1) * seg_len - 1) * H + h) * 4 + 3);   // over all of segment sp
        const unsigned long long gg = la_pair(g_seg, g_seg);
#pragma unroll
        for (int i = 0; i < DPT; i += 2)
#pragma unroll
          for (int c = 0; c < C; ++c) {
            const bool live = col + c < Dv;
            la_fma2(s2[c][i >> 1], gg, s2[c][i >> 1],
                    la_pair(live && own(i) < D ? __ldcg(ps + (size_t)own(i) * Dv + col + c) : 0.f,
                            live && own(i + 1) < D ? __ldcg(ps + (size_t)own(i + 1) * Dv + col + c) : 0.f));
          }
      }
    }
  }

  const int n_chunks = (n_new + LA_CHUNK - 1) / LA_CHUNK;
  const int qk_pieces = (PASS == 1 ? 2 : 1) * Dp / 4, v_pieces = PASS == 1 ? cols / 4 : 0;
  const int pieces = qk_pieces + v_pieces + (GATED ? 1 : 0);
  const int tid_tok = tid / pieces, tid_pc = tid - tid_tok * pieces;              // where this thread's first piece lies
  const int step_tok = (int)blockDim.x / pieces, step_pc = (int)blockDim.x - step_tok * pieces;   // and its stride
  auto load_chunk = [&](int chunk) {
    float* buf = la_smem + (size_t)(chunk % LA_STAGES) * LA_CHUNK * tok_len;
    const int base = chunk * LA_CHUNK;
    const int n_tok = (n_new - base) < LA_CHUNK ? (n_new - base) : LA_CHUNK;
    // piece e of the chunk is piece (e % pieces) of token (e / pieces); a thread walks its pieces without dividing
    const float* src0 = prep + ((size_t)(t0 + base) * H + h) * row_len;
    const size_t tok_stride = (size_t)H * row_len;
    const float* gsrc0 = GATED ? gates + ((size_t)(t0 + base) * H + h) * 4 : nullptr;
    int tt = tid_tok, pc = tid_pc;
    for (int e = tid; e < n_tok * pieces; e += blockDim.x) {
      const float* src = src0 + tt * tok_stride;
      float* dst = buf + tt * tok_len;
      if (pc < qk_pieces) la_cp_async16(dst + 4 * pc, src + 4 * pc);
      else if (GATED && pc == pieces - 1) la_cp_async16(dst + 2 * Dp + cols, gsrc0 + (size_t)tt * H * 4);
      else if (c0 + 4 * (pc - qk_pieces) < Dvp) la_cp_async16(dst + 2 * Dp + 4 * (pc - qk_pieces), src + 2 * Dp + c0 + 4 * (pc - qk_pieces));
      tt += step_tok;
      pc += step_pc;
      if (pc >= pieces) pc -= pieces, ++tt;
    }
  };
  for (int c = 0; c < LA_STAGES - 1; ++c) {
    if (c < n_chunks) load_chunk(c);
    la_cp_async_commit();
  }
  float g_pow = g;                                 // PASS 2: decay^(i+1) for the token at hand
  const size_t out_stride = (size_t)H * Dv;
  float* out_col = out + (size_t)t0 * out_stride + (size_t)h * Dv + col;        // this thread's column of the segment's first token
  for (int chunk = 0; chunk < n_chunks; ++chunk) {
    if (chunk + LA_STAGES - 1 < n_chunks) load_chunk(chunk + LA_STAGES - 1);     // into the buffer walked last round
    la_cp_async_commit();
    la_cp_async_wait<LA_STAGES - 1>();            // this chunk's copies have landed
    __syncthreads();
    const float* buf = la_smem + (size_t)(chunk % LA_STAGES) * LA_CHUNK * tok_len;
    const int base = chunk * LA_CHUNK;
    const int n_tok = (n_new - base) < LA_CHUNK ? (n_new - base) : LA_CHUNK;
    // one token.  PASS 1: S = g S + k v, then this thread's share of q . S.  PASS 2: its share of q . E.  The
    // shares are added and stored afterwards, so that in a full chunk (the loop below unrolls) one token's
    // shuffles overlap the next token's arithmetic.
    if constexpr (C == 1) {
      auto one_token = [&](int tt) {
        const float* qrow = buf + tt * tok_len;
        const float* krow = qrow + Dp;
        float v = (PASS == 1 && col_live) ? qrow[2 * Dp + warp * 4 + (lane >> 3)] : 0.f;
        float gt = g;
        if (GATED && PASS == 1) gt = qrow[2 * Dp + cols], v *= qrow[2 * Dp + cols + 1];      // a_t; b_t rides on v
        float acc0 = 0.f, acc1 = 0.f, acc2 = 0.f, acc3 = 0.f;
#pragma unroll
        for (int i4 = 0; i4 < DPT / 4; ++i4) {
          const int d = 4 * (r + 8 * i4);
          if (d < Dp) {
            const float4 q4 = *reinterpret_cast<const float4*>(qrow + d);
            float* s4 = s_reg + 4 * i4;
            if (PASS == 1) {
              const float4 k4 = *reinterpret_cast<const float4*>(krow + d);
              s4[0] = fmaf(gt, s4[0], k4.x * v);
              s4[1] = fmaf(gt, s4[1], k4.y * v);
              s4[2] = fmaf(gt, s4[2], k4.z * v);
              s4[3] = fmaf(gt, s4[3], k4.w * v);
            }
            acc0 = fmaf(s4[0], q4.x, acc0);
            acc1 = fmaf(s4[1], q4.y, acc1);
            acc2 = fmaf(s4[2], q4.z, acc2);
            acc3 = fmaf(s4[3], q4.w, acc3);
          }
        }
        return (acc0 + acc1) + (acc2 + acc3);
      };
      const bool writer = r == 0 && col_live;
      float* out_chunk = out_col + (size_t)base * out_stride;
      auto out_at = [&](int tt) { return out_chunk + (size_t)tt * out_stride; };
      auto finish = [&](int tt, float acc, float before) {       // before: PASS 2, what the first pass left there
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if (PASS == 1) {
          if (writer) *out_at(tt) = acc;
        } else if (GATED) {
          if (writer) *out_at(tt) = before + buf[tt * tok_len + 2 * Dp + cols + 3] * acc;
        } else {
          if (writer) *out_at(tt) = before + g_pow * acc;
          g_pow *= g;
        }
      };
      if (n_tok == LA_CHUNK) {
        float part[LA_CHUNK], before[LA_CHUNK];
        if (PASS == 2) {                       // the chunk's outputs of the first pass, fetched together
#pragma unroll
          for (int tt = 0; tt < LA_CHUNK; ++tt) before[tt] = writer ? __ldcg(out_at(tt)) : 0.f;
        }
#pragma unroll
        for (int tt = 0; tt < LA_CHUNK; ++tt) part[tt] = one_token(tt);
#pragma unroll
        for (int tt = 0; tt < LA_CHUNK; ++tt) finish(tt, part[tt], PASS == 2 ? before[tt] : 0.f);
      } else {
        for (int tt = 0; tt < n_tok; ++tt) {
          const float before = (PASS == 2 && writer) ? __ldcg(out_at(tt)) : 0.f;
          finish(tt, one_token(tt), before);
        }
      }
    } else {
      auto one_token = [&](int tt, float (&share)[C]) {
        const float* qrow = buf + tt * tok_len;
        const float* krow = qrow + Dp;
        unsigned long long vv[C], acc01[C], acc23[C];
        const float gt = GATED && PASS == 1 ? qrow[2 * Dp + cols] : g;              // a_t
        const unsigned long long gg = la_pair(gt, gt);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          float v = (PASS == 1 && col + c < Dv) ? qrow[2 * Dp + cw + c] : 0.f;
          if (GATED && PASS == 1) v *= qrow[2 * Dp + cols + 1];                       // b_t rides on v
          vv[c] = la_pair(v, v);
          acc01[c] = acc23[c] = 0ull;
        }
#pragma unroll
        for (int i4 = 0; i4 < DPT / 4; ++i4) {
          const int d = 4 * (r + 8 * i4);
          if (d < Dp) {
            const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(qrow + d);
            if (PASS == 1) {
              const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(krow + d);
#pragma unroll
              for (int c = 0; c < C; ++c) {
                la_fma2(s2[c][2 * i4], gg, s2[c][2 * i4], la_mul2(k4.x, vv[c]));
                la_fma2(s2[c][2 * i4 + 1], gg, s2[c][2 * i4 + 1], la_mul2(k4.y, vv[c]));
              }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
              la_fma2(acc01[c], s2[c][2 * i4], q4.x, acc01[c]);
              la_fma2(acc23[c], s2[c][2 * i4 + 1], q4.y, acc23[c]);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) share[c] = (la_lo(acc01[c]) + la_hi(acc01[c])) + (la_lo(acc23[c]) + la_hi(acc23[c]));
      };
      float* out_chunk = out_col + (size_t)base * out_stride;
      // what token tt's sum is worth (PASS 2: added to what the first pass left there)
      auto result = [&](int tt, float acc, float before, float pow) {
        if (PASS == 1) return acc;
        return GATED ? before + buf[tt * tok_len + 2 * Dp + cols + 3] * acc : before + pow * acc;
      };
      if (n_tok == LA_CHUNK) {
        static_assert(LA_CHUNK == 8, "a token for each of a column's lanes");
        float part[LA_CHUNK][C], before[C], pow = 0.f;
        float* mine = out_chunk + (size_t)r * out_stride;        // lane r finishes token r
#pragma unroll
        for (int c = 0; c < C; ++c) before[c] = (PASS == 2 && col + c < Dv) ? __ldcg(mine + c) : 0.f;
#pragma unroll
        for (int tt = 0; tt < LA_CHUNK; ++tt) one_token(tt, part[tt]);
        if (PASS == 2 && !GATED) {
#pragma unroll
          for (int tt = 0; tt < LA_CHUNK; ++tt) {
            if (tt == r) pow = g_pow;
            g_pow *= g;
          }
        }
        // lanes r and r ^ 1 add their shares and keep every other token, then r ^ 2, then r ^ 4
#pragma unroll
        for (int c = 0; c < C; ++c) {
          float a4[4], a2[2];
#pragma unroll
          for (int j = 0; j < 4; ++j) {               // tokens 2 j (even lanes) and 2 j + 1 (odd lanes)
            const float give = (r & 1) ? part[2 * j][c] : part[2 * j + 1][c], keep = (r & 1) ? part[2 * j + 1][c] : part[2 * j][c];
            a4[j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float give = (r & 2) ? a4[2 * j] : a4[2 * j + 1], keep = (r & 2) ? a4[2 * j + 1] : a4[2 * j];
            a2[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
          }
          const float give = (r & 4) ? a2[0] : a2[1], keep = (r & 4) ? a2[1] : a2[0];
          const float acc = keep + __shfl_xor_sync(0xffffffffu, give, 4);
          if (col + c < Dv) mine[c] = result(r, acc, before[c], pow);
        }
      } else {
        for (int tt = 0; tt < n_tok; ++tt) {
          float* at = out_chunk + (size_t)tt * out_stride;
          float share[C];
          one_token(tt, share);
#pragma unroll
          for (int c = 0; c < C; ++c) {
            const bool writer = r == 0 && col + c < Dv;
            const float before = (PASS == 2 && writer) ? __ldcg(at + c) : 0.f;
            float acc = share[c];
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (writer) at[c] = result(tt, acc, before, g_pow);
          }
          if (PASS == 2 && !GATED) g_pow *= g;
        }
      }
    }
    __syncthreads();                              // the buffer is refilled by the next round's copies
  }
  auto value = [&](int c, int i) {
    if constexpr (C == 1) return s_reg[i];
    else return (i & 1) ? la_hi(s2[c][i >> 1]) : la_lo(s2[c][i >> 1]);
  };
  if (PASS == 1) {
    float* dst = n_seg == 1 ? S : part_seq + (size_t)seg * D * Dv;
#pragma unroll
    for (int i = 0; i < DPT; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (col + c < Dv && own(i) < D) dst[(size_t)own(i) * Dv + col + c] = value(c, i);
  } else if (seg == n_seg - 1) {
    // the sequence's new state: E_(n_seg-1) = decay^(its length) E_(n_seg-2) + partial_(n_seg-1)
    float g_len = 1.f;
    if (GATED) g_len = __ldcg(gates + ((size_t)(t0 + n_new - 1) * H + h) * 4 + 3);
    else
      for (int i = 0; i < n_new; ++i) g_len *= g;
    const float* ps = part_seq + (size_t)seg * D * Dv;
#pragma unroll
    for (int i = 0; i < DPT; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (col + c < Dv && own(i) < D)
          S[(size_t)own(i) * Dv + col + c] = fmaf(g_len, value(c, i), __ldcg(ps + (size_t)own(i) * Dv + col + c));
  }
}

// ---------------------------------------------------------------------------
// Long prompts under a fixed decay, by chunks.  prep as above; chunks of sequences with more than short_new tokens.
// st [slots][H][D][Dvp]: the chunk's own part of its last state, then (decay_pass) the state it starts from; at [slots][H]:
// decay to the power of its tokens; cb [slots][H][64][64]: q_i . k_j at row j, column i.
// Powers of the decay are taken in 64 bits: a product of equal float32 factors errs the same way every time, and the
// recurrence applies the decay itself, which is exact.  `at` keeps what its rounding to float32 left out beside it, for it
// is applied chunk after chunk.
// ---------------------------------------------------------------------------
struct LaDims {
  int H, D, Dv, short_new;
  size_t head_stride;                                   // of the state
  __host__ __device__ int Dp() const { return (D + 3) & ~3; }
  __host__ __device__ int Dvp() const { return (Dv + 3) & ~3; }
  __host__ __device__ int row() const { return 2 * Dp() + Dvp(); }
};

#define LA_FOLD 128              // dims whose products are added in one chain; more are added in two
__device__ __forceinline__ double la_power(double g, int n) {       // g^n, 0 <= n <= 64
  double p = 1.0;
#pragma unroll
  for (int bit = 0; bit < 7; ++bit) {
    if (n >> bit & 1) p *= g;
    g *= g;
  }
  return p;
}

__global__ void __launch_bounds__(SS_THREADS)
decay_chunk_kernel(const float* __restrict__ prep, const float* __restrict__ decay, float* __restrict__ st,
                   float2* __restrict__ at, float* __restrict__ cb, const int* __restrict__ seq_start, int n_seqs,
                   int n_tokens, const LaDims dm) {
  __shared__ __align__(16) float As[64 * 64];
  __shared__ __align__(16) float Bs[64 * 64];
  __shared__ float ws[SS_CHUNK];
  pdl_launch_dependents();
  const int Dp = dm.Dp(), Dvp = dm.Dvp();
  const size_t step = (size_t)dm.H * dm.row();          // from token to token
  const int p_tiles = (Dvp + 63) >> 6, tiles = ((dm.D + 63) >> 6) * p_tiles;
  const int tid = threadIdx.x, slot = blockIdx.x / (dm.H * (tiles + 1)), job = blockIdx.x - slot * dm.H * (tiles + 1);
  const SsChunk ck = ss_chunk_of(seq_start, n_seqs, n_tokens, slot, dm.short_new);
  pdl_wait();                                          // (ahead of any leaving: a kernel whose CTAs all leave must not end
  if (ck.n <= 0) return;                               // before the one ahead of it)
  float acc[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] = 0.f;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int i0 = ss_row0(), j0 = ss_col0();
  if (job < dm.H * tiles) {
    const int h = job / tiles, tl = job - h * tiles;
    const int n0 = (tl / p_tiles) * 64, c0 = (tl % p_tiles) * 64;
    const float g = decay[h];
    // 16 lanes a row: v goes straight to shared memory, k through registers, where it takes its token's weight
    const int lr = tid >> 4, lc = (tid & 15) * 4;
    const float* krow = prep + (size_t)ck.t0 * step + (size_t)h * dm.row() + Dp + n0 + lc;
    const float* vrow = prep + (size_t)ck.t0 * step + (size_t)h * dm.row() + 2 * Dp + c0 + lc;
    const bool k_live = n0 + lc < Dp, v_live = c0 + lc < Dvp;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = lr + 4 * m;
      const bool live = v_live && j < ck.n;
      ss_copy16(Bs + j * 64 + lc, live ? vrow + (size_t)j * step : prep, live);
    }
    ss_copy_commit();
    float4 kv[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = lr + 4 * m;
      kv[m] = k_live && j < ck.n ? ss_load4(krow + (size_t)j * step) : zero;
    }
    ws[tid] = (float)la_power(g, max(ck.n - 1 - tid, 0));        // (k past the chunk's tokens is zero)
    if (tid == 0 && tl == 0) {
      const double all = la_power(g, ck.n);
      at[(size_t)slot * dm.H + h] = make_float2((float)all, (float)(all - (double)(float)all));
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = lr + 4 * m;
      const float w = ws[j];
      ss_store4(As + j * 64 + lc, make_float4(kv[m].x * w, kv[m].y * w, kv[m].z * w, kv[m].w * w));
    }
    ss_copy_wait<0>();
    __syncthreads();
    ss_product<4>(acc, As, 64, Bs, 64, (ck.n + 3) & ~3);   // (rows past the chunk's tokens are zero)
    float* dst = st + ((size_t)slot * dm.H + h) * dm.D * Dvp + c0 + j0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int n = n0 + ss_row(i0, r);
      if (n >= dm.D) continue;
      if (c0 + j0 < Dvp) ss_store4(dst + (size_t)n * Dvp, make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]));
      if (c0 + j0 + 32 < Dvp) ss_store4(dst + (size_t)n * Dvp + 32, make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]));
    }
    return;
  }
  // ---- q_i . k_j: both operands are turned so that a row of shared memory holds one dim of all tokens
  const int h = job - dm.H * tiles;
  const float* qrow = prep + (size_t)(ck.t0 + tid) * step + (size_t)h * dm.row();
  const bool live = tid < ck.n;
  for (int kb = 0; kb < Dp; kb += 32) {
    float4 qv[8], kv[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      qv[m] = live && kb + 4 * m < Dp ? ss_load4(qrow + kb + 4 * m) : zero;
      kv[m] = live && kb + 4 * m < Dp ? ss_load4(qrow + Dp + kb + 4 * m) : zero;
    }
    __syncthreads();                                   // (the tiles of the block before have been read)
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      float* ap = As + 4 * m * 64 + tid;
      float* bp = Bs + 4 * m * 64 + tid;
      ap[0] = qv[m].x, ap[64] = qv[m].y, ap[128] = qv[m].z, ap[192] = qv[m].w;
      bp[0] = kv[m].x, bp[64] = kv[m].y, bp[128] = kv[m].z, bp[192] = kv[m].w;
    }
    __syncthreads();
    ss_product<4>(acc, As, 64, Bs, 64, min(32, Dp - kb));
    if (kb + 32 == LA_FOLD || kb + 32 >= Dp) {         // the first LA_FOLD dims' sums wait where the result goes
      float* dst = cb + ((size_t)slot * dm.H + h) * 4096;
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float* row = dst + ss_row(j0, c) * 64 + i0 + 32 * half;
          float4 v = make_float4(acc[4 * half][c], acc[4 * half + 1][c], acc[4 * half + 2][c], acc[4 * half + 3][c]);
          if (kb >= LA_FOLD) {
            const float4 w = ss_load4(row);
            v = make_float4(w.x + v.x, w.y + v.y, w.z + v.z, w.w + v.w);
          }
          ss_store4(row, v);
          acc[4 * half][c] = acc[4 * half + 1][c] = acc[4 * half + 2][c] = acc[4 * half + 3][c] = 0.f;
        }
    }
  }
}

// Every four elements of a sequence's state, one thread: E_0 is the stored state, E_(c+1) = at_c E_c + st_c; st_c becomes
// E_c, the stored state the last E.
__global__ void __launch_bounds__(256)
decay_pass_kernel(float* __restrict__ st, const float2* __restrict__ at, float* __restrict__ state,
                  const int* __restrict__ seq_start, const int* __restrict__ seq_slot, const LaDims dm) {
  pdl_launch_dependents();
  const int b = blockIdx.y, row0 = seq_start[b], n_new = seq_start[b + 1] - row0;
  pdl_wait();
  if (n_new <= dm.short_new) return;
  const int Dvp = dm.Dvp(), p4 = Dvp >> 2;
  const size_t per_head = (size_t)dm.D * p4, idx = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (idx >= per_head * dm.H) return;
  const int h = (int)(idx / per_head), d = (int)((idx - h * per_head) / p4), p = (int)(idx % p4) * 4;
  const int chunks = (n_new + SS_CHUNK - 1) / SS_CHUNK, slot0 = row0 / SS_CHUNK + b;
  float* sp = state + ((size_t)seq_slot[b] * dm.H + h) * dm.head_stride + (size_t)d * dm.Dv + p;
  const bool vec = (dm.Dv & 3) == 0 && (dm.head_stride & 3) == 0 && ((uintptr_t)state & 15) == 0;
  float4 e;
  if (vec) e = ss_load4(sp);
  else e = make_float4(sp[0], p + 1 < dm.Dv ? sp[1] : 0.f, p + 2 < dm.Dv ? sp[2] : 0.f, p + 3 < dm.Dv ? sp[3] : 0.f);
  const size_t step = (size_t)dm.H * dm.D * Dvp;
  float* cp = st + (size_t)slot0 * step + ((size_t)h * dm.D + d) * Dvp + p;
  const float2* ap = at + (size_t)slot0 * dm.H + h;
  for (int c0 = 0; c0 < chunks; c0 += 4) {              // four chunks' parts in flight
    float4 s[4];
    float2 a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u < chunks) s[u] = ss_load4(cp + (size_t)(c0 + u) * step), a[u] = ap[(size_t)(c0 + u) * dm.H];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u < chunks) {
        ss_store4(cp + (size_t)(c0 + u) * step, e);
        e = make_float4(fmaf(a[u].x, e.x, fmaf(a[u].y, e.x, s[u].x)), fmaf(a[u].x, e.y, fmaf(a[u].y, e.y, s[u].y)),
                        fmaf(a[u].x, e.z, fmaf(a[u].y, e.z, s[u].z)), fmaf(a[u].x, e.w, fmaf(a[u].y, e.w, s[u].w)));
      }
  }
  if (vec) {
    ss_store4(sp, e);
  } else {
    sp[0] = e.x;
    if (p + 1 < dm.Dv) sp[1] = e.y;
    if (p + 2 < dm.Dv) sp[2] = e.z;
    if (p + 3 < dm.Dv) sp[3] = e.w;
  }
}

#define LA_LDM 68                // row stride of the masked 64 x 64 matrix in shared memory: 16-byte stores meet no bank twice
__global__ void __launch_bounds__(SS_THREADS)
decay_out_kernel(const float* __restrict__ prep, const float* __restrict__ decay, const float* __restrict__ st,
                 const float* __restrict__ cb, float* __restrict__ out, const int* __restrict__ seq_start, int n_seqs,
                 int n_tokens, const LaDims dm) {
  __shared__ __align__(16) float Ms[64 * LA_LDM];      // row j: decay^(i-j) (q_i . k_j) over i; before that the turned q
  __shared__ __align__(16) float Bs[2][32 * 64];       // rows of E, then of v
  __shared__ float power[SS_CHUNK + 1];                // of the decay
  pdl_launch_dependents();
  const int Dp = dm.Dp(), Dvp = dm.Dvp(), p_tiles = (Dvp + 63) >> 6;
  const int tid = threadIdx.x, slot = blockIdx.x / (dm.H * p_tiles), job = blockIdx.x - slot * dm.H * p_tiles;
  const SsChunk ck = ss_chunk_of(seq_start, n_seqs, n_tokens, slot, dm.short_new);
  pdl_wait();
  if (ck.n <= 0) return;                               // (uniform)
  const int h = job / p_tiles, c0 = (job - h * p_tiles) * 64;
  const size_t step = (size_t)dm.H * dm.row();
  const float g = decay[h];
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int lr = tid >> 4, lc = (tid & 15) * 4;        // a row of E or v: 16 lanes
  const bool col_live = c0 + lc < Dvp;
  const float* e_base = st + ((size_t)slot * dm.H + h) * dm.D * Dvp + c0 + lc;
  const float* v_base = prep + (size_t)ck.t0 * step + (size_t)h * dm.row() + 2 * Dp + c0 + lc;
  const float* qrow = prep + (size_t)(ck.t0 + tid) * step + (size_t)h * dm.row();
  const int e_steps = (dm.D + 31) >> 5, steps = e_steps + ((ck.n + 31) >> 5);
  auto copy_rows = [&](int k0) {                        // step k0: 32 rows of E, then of v, into one of two buffers
    float* dst = Bs[k0 & 1] + lc;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int r = lr + 4 * m, k = (k0 < e_steps ? k0 : k0 - e_steps) * 32 + r;
      const bool live = col_live && (k0 < e_steps ? k < dm.D : k < ck.n);
      const float* src = k0 < e_steps ? e_base + (size_t)k * Dvp : v_base + (size_t)k * step;
      ss_copy16(dst + r * 64, live ? src : prep, live);
    }
    ss_copy_commit();
  };
  float4 qv[8];
  auto fetch_q = [&](int kb) {
#pragma unroll
    for (int m = 0; m < 8; ++m) qv[m] = tid < ck.n && kb + 4 * m < Dp ? ss_load4(qrow + kb + 4 * m) : zero;
  };
  copy_rows(0);
  fetch_q(0);
  // the rest is on its way to L2 meanwhile: rows of E and the products q . k
  for (int i = tid; i < 2 * dm.D; i += SS_THREADS)
    if (c0 + (i & 1) * 32 < Dvp) prefetch_l2(st + ((size_t)slot * dm.H + h) * dm.D * Dvp + (size_t)(i >> 1) * Dvp + c0 + (i & 1) * 32);
  for (int i = tid; i < 128; i += SS_THREADS) prefetch_l2(cb + ((size_t)slot * dm.H + h) * 4096 + i * 32);
  power[tid] = (float)la_power(g, tid);
  if (tid == 0) power[SS_CHUNK] = (float)la_power(g, SS_CHUNK);
  float acc[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] = 0.f;
  const int i0 = ss_row0(), j0 = ss_col0();
  auto each_result = [&](auto&& f) {                   // f(a result of this thread, where it goes)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = ss_row(i0, r);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int p = c0 + ss_row(j0, c);
        if (i < ck.n && p < dm.Dv) f(acc[r][c], out + ((size_t)(ck.t0 + i) * dm.H + h) * dm.Dv + p);
      }
    }
  };
  // ---- E^T q_i
  for (int s = 0; s < e_steps; ++s) {
    float* As = Ms + (s & 1) * 32 * 64;
#pragma unroll
    for (int m = 0; m < 8; ++m) {                      // q turned: a row of shared memory holds one dim of all tokens
      float* ap = As + 4 * m * 64 + tid;
      ap[0] = qv[m].x, ap[64] = qv[m].y, ap[128] = qv[m].z, ap[192] = qv[m].w;
    }
    ss_copy_wait<0>();
    __syncthreads();                                   // (and every thread is done with the tiles of the step before)
    copy_rows(s + 1);
    if (s + 1 < e_steps) fetch_q((s + 1) * 32);
    ss_product<2>(acc, As, 64, Bs[s & 1], 64, min(32, Dp - s * 32));      // (rows of E past D are zero)
    if ((s + 1) * 32 == LA_FOLD && s + 1 < e_steps)    // the first LA_FOLD dims' sums wait where the result goes
      each_result([](float& a, float* to) { *to = a, a = 0.f; });
  }
  if (dm.D > LA_FOLD) each_result([](float& a, float* to) { a += *to; });
  __syncthreads();                                     // the turned q has been read: its place takes the masked matrix
  {
    // a thread a column j; what lies above the diagonal is zero
    const float* cbj = cb + (((size_t)slot * dm.H + h) * 64 + tid) * 64;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 d[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) d[m] = 16 * q + 15 >= tid ? ss_load4(cbj + 16 * q + 4 * m) : zero;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float o[4] = {d[m].x, d[m].y, d[m].z, d[m].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = 16 * q + 4 * m + e;
          o[e] = i >= tid ? o[e] * power[i - tid] : 0.f;
        }
        ss_store4(Ms + tid * LA_LDM + 16 * q + 4 * m, make_float4(o[0], o[1], o[2], o[3]));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const float ga = power[ss_row(i0, r) + 1];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] *= ga;
  }
  // ---- + sum over the chunk's own tokens
  for (int s = e_steps; s < steps; ++s) {
    ss_copy_wait<0>();
    // A token's infinite or NaN value is not multiplied by the zeros above the diagonal: tokens before it do not see it.
    float zero_if_finite = 0.f;
#pragma unroll
    for (int m = 0; m < 8; ++m) {                      // (what this thread copied)
      const float4 v = ss_load4(Bs[s & 1] + (lr + 4 * m) * 64 + lc);
      zero_if_finite = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, zero_if_finite))));
    }
    const bool select = __syncthreads_or(!(zero_if_finite == 0.f));
    if (s + 1 < steps) copy_rows(s + 1);
    const int jb = (s - e_steps) * 32;
    if (select) {
      for (int k = 0; k < min(32, ck.n - jb); ++k)
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int i = ss_row(i0, r);
          if (jb + k > i) continue;
          const float m = Ms[(jb + k) * LA_LDM + i];
#pragma unroll
          for (int c = 0; c < 8; ++c) acc[r][c] = fmaf(m, Bs[s & 1][k * 64 + ss_row(j0, c)], acc[r][c]);
        }
    } else if (jb == 0) ss_product<2>(acc, Ms, LA_LDM, Bs[s & 1], 64, min(32, ck.n));
    else ss_product<2, false>(acc, Ms + jb * LA_LDM, LA_LDM, Bs[s & 1], 64, ck.n - jb);      // (they reach rows 32.. only)
  }
  const bool vec = (dm.Dv & 3) == 0 && ((uintptr_t)out & 15) == 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = ss_row(i0, r);
    if (i >= ck.n) continue;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int p = c0 + j0 + 32 * half;
      if (p >= dm.Dv) continue;
      const float* a = acc[r] + 4 * half;
      float* dst = out + ((size_t)(ck.t0 + i) * dm.H + h) * dm.Dv + p;
      if (vec) ss_store4(dst, make_float4(a[0], a[1], a[2], a[3]));
      else
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (p + c < dm.Dv) dst[c] = a[c];
    }
  }
}

// One warp per (sequence, head) walks the step's tokens of the sequence in order: the gates' pre-activations are
// columns i_off + h and f_off + h of the projected row (plus a bias), i = cap tanh(z_i / cap), f =
// logsigmoid(cap tanh(z_f / cap)); m is read from and written back to the sequence's state (m_off floats into the
// head's state).  Thirty-two tokens at a time: every lane prepares one token's (i, f), all lanes then run the chain
// m_t = max(f_t + m_(t-1), i_t) over the 32 values (two dependent operations a token), and lane j keeps what
// token j needs.  The sum of f over a segment (which the segments' second pass wants as a product of a) restarts
// wherever a segment of seg_len tokens starts, counted from the sequence's first token of the step.
template <typename TIN>
__global__ void __launch_bounds__(128)
gate_scan_kernel(const TIN* __restrict__ proj, int n_split, size_t split_stride, size_t row_stride, int i_off, int f_off,
                 const float* __restrict__ bias_i, const float* __restrict__ bias_f, float cap,
                 float* __restrict__ gates, float* __restrict__ state, size_t head_stride, int m_off,
                 const int* __restrict__ seq_start, const int* __restrict__ seq_slot, int H, int seg_len) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = blockIdx.x * 4 + warp, b = blockIdx.y;
  if (h >= H) return;
  const int t0 = seq_start[b], n_new = seq_start[b + 1] - t0;
  float* m_ptr = state + ((size_t)seq_slot[b] * H + h) * head_stride + m_off;
  const float bi = bias_i ? bias_i[h] : 0.f, bf = bias_f ? bias_f[h] : 0.f;
  pdl_wait();
  float m = *m_ptr, cum = 0.f, m_base = m;
  int in_seg = 0;                                    // (base + j) % seg_len, kept by counting
  for (int base = 0; base < n_new; base += 32) {
    const int n = min(32, n_new - base);
    float il = 0.f, fl = 0.f;
    if (lane < n) {
      const TIN* row = proj + (size_t)(t0 + base + lane) * row_stride;
      float zi = la_value(row, i_off + h, n_split, split_stride) + bi;
      float zf = la_value(row, f_off + h, n_split, split_stride) + bf;
      if (cap > 0.f) zi = cap * tanhf(zi / cap), zf = cap * tanhf(zf / cap);
      il = zi;
      fl = fminf(zf, 0.f) - log1pf(expf(-fabsf(zf)));           // log sigmoid(zf)
    }
    float my_prev = 0.f, my_m = 0.f, my_sum = 0.f;
    // every lane walks the chain m -> max(f + m, i); a whole block of 32 tokens is unrolled, so that the broadcasts
    // run ahead of the chain
    auto token = [&](int j) {
      const float f = __shfl_sync(0xffffffffu, fl, j), i = __shfl_sync(0xffffffffu, il, j);
      if (in_seg == 0) cum = 0.f, m_base = m;
      if (++in_seg == seg_len) in_seg = 0;
      const float m_new = fmaxf(f + m, i);
      cum += f;
      if (lane == j) my_prev = m, my_m = m_new, my_sum = cum + m_base;
      m = m_new;
    };
    if (n == 32) {
#pragma unroll
      for (int j = 0; j < 32; ++j) token(j);
    } else {
      for (int j = 0; j < n; ++j) token(j);
    }
    if (lane < n)
      *reinterpret_cast<float4*>(gates + ((size_t)(t0 + base + lane) * H + h) * 4) =
          make_float4(expf(fl + my_prev - my_m), expf(il - my_m), expf(-my_m), expf(my_sum - my_m));
  }
  if (lane == 0) *m_ptr = m;
}

// proj: [T, row_stride] (or split partials of it); gates: float32 [T, H, 4], 16-byte aligned; state: float32
// [slots, H, head_stride] with a head's m at m_off; bias_i, bias_f: float32 [H] or null; cap <= 0: no cap.
LLMX_API int llmx_gate_scan(const void* proj, int in_dtype, int n_split, long long split_stride, long long row_stride,
                            int i_off, int f_off, const float* bias_i, const float* bias_f, float cap, float* gates,
                            float* state, long long head_stride, int m_off, const int* seq_start, const int* seq_slot,
                            int n_seqs, int H, int seg_len, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (H <= 0 || n_split < 1 || head_stride <= m_off || m_off < 0 || n_seqs > 65535 || ((uintptr_t)gates & 15))
    return LLMX_REFUSED(1);
  if (seg_len <= 0) seg_len = LA_SEG;
  const dim3 grid((H + 3) / 4, n_seqs);
  if (in_dtype == LLMX_F32)
    launch_pdl(gate_scan_kernel<float>, grid, dim3(128), 0, stream, (const float*)proj, n_split, (size_t)split_stride,
               (size_t)row_stride, i_off, f_off, bias_i, bias_f, cap, gates, state, (size_t)head_stride, m_off,
               seq_start, seq_slot, H, seg_len);
  else if (in_dtype == LLMX_BF16)
    launch_pdl(gate_scan_kernel<bf16>, grid, dim3(128), 0, stream, (const bf16*)proj, n_split, (size_t)split_stride,
               (size_t)row_stride, i_off, f_off, bias_i, bias_f, cap, gates, state, (size_t)head_stride, m_off,
               seq_start, seq_slot, H, seg_len);
  else
    return LLMX_REFUSED(2);
  return LLMX_LAUNCH_STATUS();
}

// Whether prompts of more than one segment go by chunks: under a fixed decay, for states of at least 64 x 64 (v_size counts
// the extra column), which fill a tile.  16 heads, four prompts of 700 to 1300 tokens, chunks against the recurrence in
// segments: 291 / 586 us at 128 x 128, 139 / 212 at 64 x 64, 105 / 117 at 32 x 32, 87 / 81 at 16 x 16.  States below 64 have
// little to gain and keep the recurrence, whose sums for a whole prompt and for its tokens one by one lie closer together.
LLMX_API int llmx_decay_scan_by_chunks(int gated, int k_size, int v_size) { return !gated && k_size >= 64 && v_size >= 64; }

// proj: [T, row_stride] (or split partials of it); prep: float32 scratch of T * H * (2 Dp + Dvp) elements, 16-byte
// aligned; out: float32 [T, H*Dva]; state: float32 [slots, H, head_stride >= D*Dva], Dva = Dv + v_ones (v_ones:
// the values get one more column that is 1 for every token).  max_new: most tokens of one sequence; seg_len:
// tokens per segment (0: LA_SEG); partial: float32 scratch, 16-byte aligned, needed when max_new > seg_len:
// [n_seqs, H, ceil(max_new / seg_len), D, Dva], or where llmx_decay_scan_by_chunks says so C chunks, C = n_tokens / 64 +
// n_seqs, of H (D Dvap + 4098) floats (Dvap: Dva rounded up to 4).  gates: null (the heads' fixed `decay`), or float32 [T, H, 4] as gate_scan leaves them
// (made with the same seg_len).
LLMX_API int llmx_decay_scan(const void* proj, int in_dtype, int n_split, long long split_stride, long long row_stride,
                             int q_off, int k_off, int v_off, float* prep, float* out, float* state, float* partial,
                             const int* seq_start, const int* token_pos, const int* seq_slot, const float* decay,
                             const float* cos_t, const float* sin_t, int n_rot, int act, float k_scale, int n_tokens,
                             int n_seqs, int max_new, int seg_len, int H, int D, int Dv, int n_sm, const float* gates,
                             long long head_stride, float q_scale, int v_ones, cudaStream_t stream) {
  if (n_seqs <= 0 || n_tokens <= 0) return 0;
  if (H <= 0 || D <= 0 || D > LA_MAX_D || Dv <= 0 || n_split < 1 || n_rot < 0 || n_rot > D || (n_rot & 1))
    return LLMX_REFUSED(1);
  v_ones = v_ones ? 1 : 0;
  const int Dva = Dv + v_ones;
  if (head_stride <= 0) head_stride = (long long)D * Dva;
  if (head_stride < (long long)D * Dva || (!gates && !decay) || ((uintptr_t)gates & 15)) return LLMX_REFUSED(1);
  if (n_rot > 0 && (!cos_t || !sin_t)) return LLMX_REFUSED(4);
  if (act != LA_ACT_NONE && act != LA_ACT_SILU) return LLMX_REFUSED(1);
  if (n_seqs > 65535 || H > 65535 || ((uintptr_t)prep & 15)) return LLMX_REFUSED(3);
  if (seg_len <= 0) seg_len = LA_SEG;
  if (max_new <= 0 || max_new > n_tokens) max_new = n_tokens;
  const int n_seg = (max_new + seg_len - 1) / seg_len;
  const bool by_chunks = n_seg > 1 && llmx_decay_scan_by_chunks(gates != nullptr, D, Dva);
  if (n_seg > 1 && (!partial || (by_chunks && ((uintptr_t)partial & 15)))) return LLMX_REFUSED(4);
  const dim3 pgrid(n_tokens, H);
  const int esz = in_dtype == LLMX_F32 ? 4 : 2;
  const bool vec = !v_ones && ((D | Dv | (n_rot >> 1) | q_off | k_off | v_off) & 3) == 0 && ((row_stride | split_stride) & 3) == 0 &&
                   ((uintptr_t)proj & (4 * esz - 1)) == 0 &&
                   (((uintptr_t)cos_t | (uintptr_t)sin_t) & 15) == 0;
  const bool many = n_tokens > 64 && n_split == 1;
  const long long pieces = (long long)(many ? (n_tokens + 1) / 2 : n_tokens) * H * ((n_rot >> 2) + ((D - n_rot) >> 1) + (Dv >> 2));
  const dim3 vgrid((unsigned)((pieces + 127) / 128));
#define PREP_VEC(TIN, TOKS, SPLIT)                                                                                                 \
  launch_pdl(decay_prep_vec_kernel<TIN, TOKS, SPLIT>, vgrid, dim3(128), 0, stream, (const TIN*)proj, n_split, (size_t)split_stride, \
             (size_t)row_stride, q_off, k_off, v_off, prep, token_pos, cos_t, sin_t, n_rot, act, k_scale, q_scale, n_tokens, \
             H, D, Dv)
#define PREP(TIN)                                                                                                           \
  if (vec && many && pieces < (1ll << 32) - 128)                                                                            \
    PREP_VEC(TIN, 2, false);                                                                                                       \
  else if (vec && pieces < (1ll << 32) - 128)                                                                               \
    PREP_VEC(TIN, 1, true);                                                                                                       \
  else                                                                                                                      \
    launch_pdl(decay_prep_kernel<TIN>, pgrid, dim3(128), 0, stream, (const TIN*)proj, n_split, (size_t)split_stride,        \
               (size_t)row_stride, q_off, k_off, v_off, prep, token_pos, cos_t, sin_t, n_rot, act, k_scale, q_scale,        \
               v_ones, H, D, Dv)
  if (in_dtype == LLMX_F32) {
    PREP(float);
  } else if (in_dtype == LLMX_BF16) {
    PREP(bf16);
  } else {
    return LLMX_REFUSED(2);
  }
#undef PREP
#undef PREP_VEC
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  Dv = Dva;                                        // from here on the extra column is a column like the others
  if (by_chunks) {
    // (a sequence of up to seg_len tokens goes through the plain recurrence below, as it does without long ones beside it)
    const LaDims dm = {H, D, Dv, seg_len, (size_t)head_stride};
    const int slots = n_tokens / SS_CHUNK + n_seqs, p_tiles = (dm.Dvp() + 63) / 64, d_tiles = (D + 63) / 64;
    const long long per_state = (long long)H * D * (dm.Dvp() / 4), jobs = (long long)slots * H * (d_tiles * p_tiles + 1);
    if (jobs > 0x7fffffff) return LLMX_REFUSED(3);
    float* cb = partial + (size_t)slots * H * D * dm.Dvp();
    float2* at = reinterpret_cast<float2*>(cb + (size_t)slots * H * 4096);
    launch_pdl(decay_chunk_kernel, dim3((unsigned)jobs), dim3(SS_THREADS), 0, stream, (const float*)prep, decay, partial, at,
               cb, seq_start, n_seqs, n_tokens, dm);
    launch_pdl(decay_pass_kernel, dim3((unsigned)((per_state + 255) / 256), n_seqs), dim3(256), 0, stream, partial,
               (const float2*)at, state, seq_start, seq_slot, dm);
    launch_pdl(decay_out_kernel, dim3((unsigned)(slots * H * p_tiles)), dim3(SS_THREADS), 0, stream, (const float*)prep, decay,
               (const float*)partial, (const float*)cb, out, seq_start, n_seqs, n_tokens, dm);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
  }
  const int scan_segs = by_chunks ? 1 : n_seg;
  // Rule: two columns a thread where they were faster (H = 2 to 16, sizes of 16 to 256, 1 to 4000 tokens a sequence; one
  // column / two, us): long gated prompts (four of 700 to 1300 tokens: 855 / 657 at 16 heads of 128 x 128, 216 / 196 at
  // 64 x 64, 566 / 480 at 192 x 96), many prompts of up to a segment with keys of 65 to 128 (eight of 100, gated: 126 / 104),
  // and small ungated states in prompts up to about 1000 tokens (300 tokens, 32 x 32: 50 / 40; 4000: 82 / 95).  Not short
  // prompts with larger keys, whose registers halve the CTAs of an SM (100 tokens, 256 x 256, gated: 81 / 110), nor steps of
  // mostly single tokens (32 of them, 128 x 128, gated: 10 / 16) unless the states are small (31 and a prompt of 200, 32 x 32,
  // gated: 44 / 35).
  const bool prompts = !by_chunks && (n_tokens >= 32 * n_seqs || (D <= 32 && n_seg > 1));
  const bool two = prompts && ((gates && max_new > (D <= 32 ? 128 : D <= 128 ? 256 : 640)) ||
                               (D > 64 && D <= 128 && n_tokens >= 512 && max_new >= 64 && max_new <= 128) ||
                               (!gates && D <= 32 && max_new <= 1024));
  const int C = two ? 2 : 1;
  // columns per CTA: as many as still give every SM a CTA or two (a CTA with more columns stages q and k fewer times)
  int cols = 32 * C;
  while (cols > 8 * C && (long long)n_seqs * H * scan_segs * ((Dv + cols - 1) / cols) < 2LL * n_sm) cols >>= 1;
  while (cols > 4 * C && cols / 2 >= Dv) cols >>= 1;
  const int Dp = (D + 3) & ~3;
  const int col_blocks = (Dv + cols - 1) / cols;
  if ((long long)col_blocks * scan_segs > 0x7fffffff) return LLMX_REFUSED(3);
  dim3 grid(col_blocks * scan_segs, H, n_seqs), block(cols * 8 / C);
  const size_t smem = (size_t)LA_STAGES * LA_CHUNK * (2 * Dp + cols + (gates ? 4 : 0)) * sizeof(float);
#define GO2(DPT, PASS, GATED, C)                                                                                       \
  do {                                                                                                                 \
    static bool attr_set = false;                                                                                      \
    if (!attr_set && smem > 48 * 1024) {                                                                               \
      e = cudaFuncSetAttribute(decay_scan_kernel<DPT, PASS, GATED, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                               100 * 1024);                                                                            \
      if (e != cudaSuccess) return (int)e;                                                                             \
      attr_set = true;                                                                                                 \
    }                                                                                                                  \
    launch_pdl(decay_scan_kernel<DPT, PASS, GATED, C>, grid, block, smem, stream, (const float*)prep, out, state, partial, \
               seq_start, seq_slot, decay, gates, (size_t)head_stride, H, D, Dv, cols, col_blocks, seg_len, n_seg,     \
               (int)by_chunks);                                                                                        \
  } while (0)
// (the instances that the rule reaches)
#define GO1(DPT, PASS)                                                                       \
  do {                                                                                       \
    if (gates && C == 2) GO2(DPT, PASS, true, 2);                                            \
    else if (gates) GO2(DPT, PASS, true, 1);                                                 \
    else if (C == 2) GO2(DPT, PASS, false, (DPT == 4 || (DPT == 16 && PASS == 1) ? 2 : 1));  \
    else GO2(DPT, PASS, false, 1);                                                           \
  } while (0)
#define GO(DPT)                    \
  do {                             \
    GO1(DPT, 1);                   \
    if (scan_segs > 1) GO1(DPT, 2); \
  } while (0)
  if (Dp <= 32) GO(4);
  else if (Dp <= 64) GO(8);
  else if (Dp <= 128) GO(16);
  else GO(32);
#undef GO
#undef GO1
#undef GO2
  return LLMX_LAUNCH_STATUS();
}

// ---------------------------------------------------------------------------
// After the recurrence: y[t, j] = o[t, j] * r * gain[j] * act(gate[t, j]) with r = 1 / sqrt(mean(o^2) + eps), the
// mean taken over one head's Dv columns (per_head, usually without a gain) or over all H*Dv columns of the
// token.  One warp per (token, head), or one CTA per token.  float32 throughout; y in the activations' dtype.
// ---------------------------------------------------------------------------
// With `gates` (float32 [T, H, 4], exp(-m) third) a head's o has o_stride = Dv + 1 columns, the last one n . q,
// and o is first divided by max(|n . q|, exp(-m)) + den_eps.
template <typename TIN, typename TO>
__global__ void gated_norm_heads_kernel(const float* __restrict__ o, const TIN* __restrict__ proj, int n_split,
                                        size_t split_stride, size_t row_stride, int g_off,
                                        const float* __restrict__ gain, float eps, int gate_act,
                                        TO* __restrict__ y, int H, int Dv, int o_stride,
                                        const float* __restrict__ gates, float den_eps) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x, h = blockIdx.y * 4 + warp;
  if (h >= H) return;
  const float* orow = o + ((size_t)t * H + h) * o_stride;
  float den = 1.f;
  if (gates) den = fmaxf(fabsf(orow[Dv]), gates[((size_t)t * H + h) * 4 + 2]) + den_eps;
  float ss = 0.f;
  for (int i = lane; i < Dv; i += 32) {
    const float v = gates ? orow[i] / den : orow[i];
    ss += v * v;
  }
  const float r = 1.0f / sqrtf(warp_sum(ss) / (float)Dv + eps);
  const TIN* grow = proj + (size_t)t * row_stride + g_off + h * Dv;
  for (int i = lane; i < Dv; i += 32) {
    float v = (gates ? orow[i] / den : orow[i]) * r;
    if (gain) v *= gain[h * Dv + i];
    y[((size_t)t * H + h) * Dv + i] = from_f32<TO>(v * la_act(la_value(grow, i, n_split, split_stride), gate_act));
  }
}

template <typename TIN, typename TO>
__global__ void __launch_bounds__(256)
gated_norm_row_kernel(const float* __restrict__ o, const TIN* __restrict__ proj, int n_split, size_t split_stride,
                      size_t row_stride, int g_off, const float* __restrict__ gain, float eps, int gate_act,
                      TO* __restrict__ y, int n) {
  __shared__ float red[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const float* orow = o + (size_t)t * n;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) ss += orow[i] * orow[i];
  const float r = 1.0f / sqrtf(block_sum(ss, red) / (float)n + eps);
  const TIN* grow = proj + (size_t)t * row_stride + g_off;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    float v = orow[i] * r;
    if (gain) v *= gain[i];
    y[(size_t)t * n + i] = from_f32<TO>(v * la_act(la_value(grow, i, n_split, split_stride), gate_act));
  }
}

// The same by four neighbouring elements a thread, U times (sizes, offsets and strides multiples of 4, no gates), everything
// asked for ahead of the reduction.  The squares are added in the chains of the kernels above, a row's by way of shared memory,
// so that the bits are theirs.  By elements and like this: four rows of 2048 with five partials (a decode step) 6.8 and 2.2 us,
// of 8192 23.6 and 5.0; 4100 rows of 8192 140 and 93.  U 0: a warp per (token, head) of up to 128 columns: 4 and 4100 tokens
// of 16 heads 3.7 and 1.7, 28.8 and 23.8.
template <typename TIN, typename TO, int U>
__global__ void __launch_bounds__(U ? 512 : 128)
gated_norm_vec_kernel(const float* __restrict__ o, const TIN* __restrict__ proj, int n_split, size_t split_stride,
                      size_t row_stride, int g_off, const float* __restrict__ gain, float eps, int gate_act,
                      TO* __restrict__ y, int n_rows, int n, int H) {
  __shared__ float red[32];
  constexpr int PARTS = U ? U : 1, LANES = U ? 512 : 32;
  pdl_launch_dependents();
  const int lane = U ? threadIdx.x : threadIdx.x & 31, r = U ? blockIdx.x : blockIdx.x * 4 + (threadIdx.x >> 5);
  const int t = U ? r : r / H, h = U ? 0 : r - t * H;                  // row r of n elements: a token, or a head of one
  float w[PARTS][4];
#pragma unroll
  for (int u = 0; u < PARTS; ++u) {
    const int i = (u * LANES + lane) * 4;
    if (gain && i < n) la_load(gain + h * n + i, w[u]);
  }
  pdl_wait();
  if (!U && r >= n_rows) return;                                       // (uniform over a warp)
  const float* orow = o + (size_t)r * n;
  const TIN* grow = proj + (size_t)t * row_stride + g_off + h * n;
  float v[PARTS][4], z[PARTS][4], ss = 0.f;
#pragma unroll
  for (int u = 0; u < PARTS; ++u) {
    const int i = (u * LANES + lane) * 4;
    if (i < n) la_load(orow + i, v[u]);
    else v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
  }
#pragma unroll
  for (int u = 0; u < PARTS; ++u) {
    const int i = (u * LANES + lane) * 4;
    if (i < n) la_values(grow + i, n_split, split_stride, z[u]);
  }
  if constexpr (U == 0) {
    ss = head_sumsq<4, 32>(v[0], 0xffffffffu);
  } else {                                                             // a thread's squares are columns 256 apart
    __shared__ __align__(16) float squared[U * 2048];
#pragma unroll
    for (int u = 0; u < U; ++u) *reinterpret_cast<float4*>(squared + (u * 512 + lane) * 4) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    __syncthreads();
    if (lane < 256)
#pragma unroll
      for (int k = 0; k < 8 * U; ++k) ss = fmaf(squared[k * 256 + lane], squared[k * 256 + lane], ss);
    ss = block_sum(ss, red);
  }
  const float rs = 1.0f / sqrtf(ss / (float)n + eps);
#pragma unroll
  for (int u = 0; u < PARTS; ++u) {
    const int i = (u * LANES + lane) * 4;
    if (i >= n) continue;
    float f[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[e] = v[u][e] * rs;
      if (gain) f[e] *= w[u][e];
      f[e] *= la_act(z[u][e], gate_act);
    }
    TO* dst = y + (size_t)r * n + i;
    if constexpr (sizeof(TO) == 4) {
      *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
    } else {
      const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
  }
}

// per_head != 0: the mean of squares is a head's; else the token's.  gain: float32 [H*Dv] or null.  gates (per_head
// only): see the kernel; o is then [T, H, Dv + 1].
LLMX_API int llmx_gated_norm(const float* o, const void* proj, int in_dtype, int n_split, long long split_stride,
                             long long row_stride, int g_off, const float* gain, float eps, int gate_act, int per_head,
                             void* y, int out_dtype, int n_tokens, int H, int Dv, const float* gates, float den_eps,
                             cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (H <= 0 || Dv <= 0 || n_split < 1 || (gates && !per_head)) return LLMX_REFUSED(1);
  const int o_stride = gates ? Dv + 1 : Dv;
  if (gate_act != LA_ACT_SILU && gate_act != LA_ACT_SIGMOID && gate_act != LA_ACT_NONE) return LLMX_REFUSED(1);
  // four elements a thread where every row, gate and gain is whole vectors, and a row fits a CTA (a head a warp)
  const int n = per_head ? Dv : H * Dv, in_size = in_dtype == LLMX_F32 ? 4 : 2, out_size = out_dtype == LLMX_F32 ? 4 : 2;
  // Where that is faster.  Heads: a warp needs more than half its lanes, or all warps run at once (seven CTAs of four an SM):
  // 4800 and 3200 heads of 64, by vectors and by elements 3.5 and 3.3, 2.7 and 2.8 us; of 32 the line is two heads an SM.  Rows: a
  // CTA is 512 threads whatever n is, and one or two share an SM: 64 rows of 512 2.2 and 2.5 us, of 256 2.1 and 2.0 (with partials
  // 2.3 and 2.4); 300 rows of 2048 4.9 and 5.2, 1200 12.8 and 9.5, 1200 of 8192 29.7 and 44.
  const long long rows = per_head ? (long long)n_tokens * H : n_tokens, sms = llmx_sm_count();
  const bool fits = per_head ? n > 64 || rows <= (n == 64 ? 28 : 2) * sms
                             : rows <= sms ? n >= 512 || n_split > 1 : n > 6144 || (n >= 2048 && rows <= 2 * sms);
  const bool vec = fits && !gates && n % 4 == 0 && g_off % 4 == 0 && row_stride % 4 == 0 && split_stride % 4 == 0 &&
                   n <= (per_head ? 128 : 8192) && (long long)n_tokens * H < (1ll << 31) && !((uintptr_t)o & 15) &&
                   !((uintptr_t)gain & 15) && !((uintptr_t)proj & (4 * in_size - 1)) && !((uintptr_t)y & (4 * out_size - 1));
#define VEC(TIN, TO, U)                                                                                              \
  launch_pdl(gated_norm_vec_kernel<TIN, TO, U>, dim3(U ? n_tokens : (n_tokens * H + 3) / 4), dim3(U ? 512 : 128), 0, \
             stream, o, (const TIN*)proj, n_split, (size_t)split_stride, (size_t)row_stride, g_off, gain, eps, gate_act, \
             (TO*)y, per_head ? n_tokens * H : n_tokens, n, H)
#define GO(TIN, TO)                                                                                                  \
  do {                                                                                                               \
    if (vec) {                                                                                                       \
      if (per_head) VEC(TIN, TO, 0);                                                                                 \
      else if (n <= 2048) VEC(TIN, TO, 1);                                                                           \
      else if (n <= 4096) VEC(TIN, TO, 2);                                                                           \
      else VEC(TIN, TO, 4);                                                                                          \
    } else if (per_head)                                                                                                    \
      launch_pdl(gated_norm_heads_kernel<TIN, TO>, dim3(n_tokens, (H + 3) / 4), dim3(128), 0, stream, o,             \
                 (const TIN*)proj, n_split, (size_t)split_stride, (size_t)row_stride, g_off, gain, eps, gate_act,    \
                 (TO*)y, H, Dv, o_stride, gates, den_eps);                                                                                  \
    else                                                                                                             \
      launch_pdl(gated_norm_row_kernel<TIN, TO>, dim3(n_tokens), dim3(256), 0, stream, o, (const TIN*)proj, n_split, \
                 (size_t)split_stride, (size_t)row_stride, g_off, gain, eps, gate_act, (TO*)y, H * Dv);              \
  } while (0)
  const int key = in_dtype * 2 + out_dtype;
  switch (key) {
    case 0: GO(float, float); break;
    case 1: GO(float, bf16); break;
    case 2: GO(bf16, float); break;
    case 3: GO(bf16, bf16); break;
    default: return LLMX_REFUSED(2);
  }
#undef GO
#undef VEC
  return LLMX_LAUNCH_STATUS();
}
