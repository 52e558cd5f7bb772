// Prompts through the recurrent mixers in chunks of 16 tokens: the delta rule (a decay per head or per key
// channel), the selective state space, and linear attention with a decay per key channel (read before or
// after the write).  recurrent.cu walks a sequence token by token; there a prompt of one sequence is bound by
// the chain from one token's state to the next (0.6 us a token at heads of 128 x 128).  Here the chain is from
// chunk to chunk, and what a chunk does to the state is three small matrix products on the tensor cores.
//
// With S the state before a chunk, and for its tokens i the decay products G_i (up to and with token i, a number
// per key channel, or one for all), K~ and Q~ rows that carry them, all four recurrences are
//     U  = T V - W S                  (what the tokens write; the state space and linear attention: U = V)
//     Y  = Q~ S + P U                 P[i, j], j <= i: what token i reads of token j's write
//     S <- G_16 S + Kd^T U            Kd[j]: k of token j, decayed to the chunk's end
// where for the delta rule A[i, j] = beta_i k_i . (G_i / G_j) k_j (j < i), T = (1 + A)^-1 diag(beta) and
// W = (1 + A)^-1 diag(beta) (G K).  Ratios of decays are products over the tokens between, never quotients, so a
// decay of zero is no exception.
//
// chunk_prepare_kernel makes Q~, Kd, W, P, T and G of every (chunk, head): all chunks side by side, nothing of it
// depends on the state.  chunk_scan_kernel walks the chunks: a warp holds 16 columns of the state, transposed,
// as accumulators of mma.sync m16n8k8, which are at the same time the next product's left operand (the inner
// index may be taken in any order, and lane t's two neighbouring columns of an accumulator stand for inner
// indexes t and t + 4).
//
// Numbers: everything is float32.  A product's operands are split into two tf32 halves, hi + lo, hi rounded to nearest (lo at
// most 2^-11 of the number, of either sign), and hi hi + hi lo + lo hi is summed in float32.  Left out: lo lo, at most 2^-22 of a
// product, and what the instruction cuts off a lo (it reads 11 bits: at most 2^-23 of the number), both of either sign.
// The tensor core's own sums are cut towards zero; see whole().  The state's own sum, S <- G S + (chunk's part), is a
// float32 fused multiply-add outside the tensor cores.  Relative errors against 64 bits, token by token / so (1,024 tokens,
// outputs and state, 1e-7): delta rule 2.2 / 2.5 and 3.6 / 3.5, with a decay per channel 1.9 / 1.8 and 2.2 / 1.9, state space
// 1.0 / 1.4 and 1.8 / 1.8, read before 2.4 / 2.2 and 2.5 / 2.0, read after 1.9 / 1.9 and 1.7 / 1.6; of a layer's states,
// whose inputs come from bfloat16 products, 54 / 54, 67 / 66 and 80 / 79 (delta rule, state space, read before).
// A number that is not finite reaches what it reaches token by token: see mend_lower().
#include <type_traits>
#include "common.cuh"

namespace {

constexpr int CT = 16;      // tokens of a chunk
enum { DELTA = 0, CHANNEL_DELTA = 1, STATE_SPACE = 2, READ_BEFORE = 3, READ_AFTER = 4 };
__host__ __device__ constexpr bool is_delta(int mode) { return mode == DELTA || mode == CHANNEL_DELTA; }
__host__ __device__ constexpr bool per_channel(int mode) { return mode == CHANNEL_DELTA || mode == READ_BEFORE || mode == READ_AFTER; }

// A (chunk, head)'s block in memory, in floats: Q~, Kd (, W), P (, T) as the scan's lanes read them, G.
template <int DP, bool HAS_W>
struct Block {
  static constexpr int Q = 0, K = DP * CT, W = 2 * DP * CT, P = (HAS_W ? 3 : 2) * DP * CT, T = P + CT * CT,
                       G = T + (HAS_W ? CT * CT : 0), FLOATS = G + DP;
};

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

__device__ __forceinline__ void split(float v, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(v - __uint_as_float(hi));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two neighbouring numbers in one instruction.
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void mul2(uint64_t& d, uint64_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ float both(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
// d += a b in three parts: hi hi into d, the two cross parts into x.
__device__ __forceinline__ void mma3(float (&d)[4], float (&x)[4], const uint32_t (&ahi)[4], const uint32_t (&alo)[4], float b0, float b1) {
  uint32_t h0, l0, h1, l1;
  split(b0, h0, l0);
  split(b1, h1, l1);
  mma(d, ahi, h0, h1);
  mma(x, ahi, l0, l1);
  mma(x, alo, h0, h1);
}
// The same with hi hi added outside the tensor core (rounded, not cut): for long sums whose partial sums say little of the whole.
__device__ __forceinline__ void mma3_apart(float (&d)[4], float (&x)[4], const uint32_t (&ahi)[4], const uint32_t (&alo)[4], float b0, float b1) {
  float f[4] = {};
  mma3(f, x, ahi, alo, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) d[e] += f[e];
}
// A sum of hi hi over `links` products added one onto the other, and its cross parts.  The tensor core cuts its sums to float32
// towards zero: every link loses 2^-25 to 2^-24 of what has been summed so far (0.72 x 2^-24 on the mean over numbers' leading
// digits; measured as a state that was 4e-8 too small), always the same way, and losses of one sign add up over the chunks
// where roundings do not.  That mean is given back, for partial sums that on the mean grow evenly.
__device__ __forceinline__ float whole(float d, float x, float links) { return d + fmaf(d, 4.3e-8f * (0.5f * (links + 1.f)), x); }

// Over a chunk's tokens, by weights below a diagonal (T, P): d = (columns of V or U) x (weights of the eight tokens 8 nt ..), token i
// from tokens up to i.
__device__ __forceinline__ void mma_lower(float (&d)[4], const uint32_t (&hi)[2][4], const uint32_t (&lo)[2][4], float4 w, int nt) {
  float x[4] = {};
  d[0] = d[1] = d[2] = d[3] = 0.f;
  mma3(d, x, hi[0], lo[0], w.x, w.y);
  if (nt) mma3(d, x, hi[1], lo[1], w.z, w.w);
#pragma unroll
  for (int e = 0; e < 4; ++e) d[e] = whole(d[e], x[e], nt ? 2.f : 1.f);
}
// Above the diagonal the weights are zeros, and what they multiply must not reach the result where it is not finite: a column's
// tokens before the first such one take the product without it.  For operands that are not all finite.
__device__ __forceinline__ void mend_lower(float (&d)[4], const uint32_t (&hi)[2][4], const uint32_t (&lo)[2][4], float4 w, int nt, int lane) {
  uint32_t h[2][4], l[2][4];
  int first[2] = {CT, CT};                      // of columns gr and gr + 8
#pragma unroll
  for (int half = 1; half >= 0; --half)
#pragma unroll
    for (int e = 3; e >= 0; --e) {              // entry e: column e & 1, token 2 t + (e >> 1) of the half
      const bool bad = !isfinite(__uint_as_float(lo[half][e]));
      h[half][e] = bad ? 0u : hi[half][e];
      l[half][e] = bad ? 0u : lo[half][e];
      if (bad) first[e & 1] = 8 * half + 2 * (lane & 3) + (e >> 1);
    }
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
    for (int c = 0; c < 2; ++c) first[c] = min(first[c], __shfl_xor_sync(0xffffffffu, first[c], o));
  float f[4];
  mma_lower(f, h, l, w, nt);
#pragma unroll
  for (int e = 0; e < 4; ++e)                   // result e: column e >> 1, token 2 t + (e & 1)
    if (8 * nt + 2 * (lane & 3) + (e & 1) < first[e >> 1]) d[e] = f[e];
}
// Whether all of a warp's numbers in such an operand are finite (a low half is not finite where its number, or the high half, is not).
__device__ __forceinline__ bool all_finite(const uint32_t (&lo)[2][4]) {
  float z = 0.f;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 4; ++e) z = fmaf(__uint_as_float(lo[h][e]), 0.f, z);
  return __all_sync(0xffffffffu, z == 0.f);
}

// Chunks are numbered over the whole step: sequence b's are cu[b] / 16 + b and those after it, which leaves room
// for every sequence's last, partly filled one.
__host__ __device__ inline int chunk_slots(int ntok, int nseq) { return ntok / CT + nseq; }

struct Prepare {
  const float *q, *k;                   // rows of ldqk floats, head group g at g * D
  long long ldqk;
  const float *first, *second;          // delta: logits of beta (and of the decay); state space: dt
  long long ldg;
  const float* decay;                   // per channel: rows of ldd floats, head h at h * D
  long long ldd;
  const float *A_log, *dt_bias, *skip, *bonus;
  const int* cu;
  int nseq, H, G, D, head0;
  float qscale;
  float* blocks;
  int slots, wide;
};

template <int DP, int MODE>
__global__ void __launch_bounds__(128, DP == 64 ? 8 : 6) chunk_prepare_kernel(const Prepare a) {
  constexpr bool HAS_W = is_delta(MODE), CH = per_channel(MODE);
  using B = Block<DP, HAS_W>;
  // A head's decay stands before whole rows, so that the roundings of its products do not average out over a row's channels
  using Product = std::conditional_t<MODE == STATE_SPACE, double, float>;
  constexpr int LD = DP + 4;
  __shared__ __align__(16) float ks[CT][LD], qs[CT][LD], extra[HAS_W || CH ? CT : 1][LD];    // extra: the decays, then W
  __shared__ __align__(16) float at[CT][CT + 4];        // A transposed: what row i takes of w_j, at [j][i]
  __shared__ float qk[CT][CT + 1], tb[HAS_W ? CT : 1][CT + 1];
  __shared__ float gate[CT], beta[CT];
  pdl_release_next();
  pdl_wait_prior();
  const int slot = blockIdx.x, head = a.head0 + blockIdx.y, g = head / (a.H / a.G), tid = threadIdx.x, D = a.D;
  int b = 0;
  // The last sequence whose chunks start at or before this one.  From the highest bit that a sequence's number can have:
  // from 1 << 30 the rounds before the first load cost a delta rule of 2,048 tokens 75 -> 69 us, a state space of four prompts 47 -> 41.
  for (int step = a.nseq > 1 ? 1 << (31 - __clz(a.nseq - 1)) : 0; step > 0; step >>= 1)
    if (b + step < a.nseq && a.cu[b + step] / CT + b + step <= slot) b += step;
  const int first = a.cu[b] + (slot - (a.cu[b] / CT + b)) * CT, n = min(CT, a.cu[b + 1] - first);
  if (n <= 0) return;
  auto load = [&](const float* base, long long ld, float (*to)[LD], float beyond) {
    if (a.wide) {                       // D fills the block's columns and rows start at 16-byte boundaries
      float4 v[DP * CT / 512];
#pragma unroll
      for (int u = 0; u < DP * CT / 512; ++u) {
        const int e = tid + 128 * u, i = e / (DP / 4), d = e % (DP / 4) * 4;
        v[u] = i < n ? *(const float4*)(base + (size_t)(first + i) * ld + d) : make_float4(beyond, beyond, beyond, beyond);
      }
#pragma unroll
      for (int u = 0; u < DP * CT / 512; ++u) {
        const int e = tid + 128 * u;
        *(float4*)&to[e / (DP / 4)][e % (DP / 4) * 4] = v[u];
      }
      return;
    }
#pragma unroll 8
    for (int e = tid; e < CT * DP; e += 128) {
      const int i = e / DP, d = e % DP;
      to[i][d] = i < n && d < D ? base[(size_t)(first + i) * ld + d] : beyond;
    }
  };
  load(a.k + (size_t)g * D, a.ldqk, ks, 0.f);
  load(a.q + (size_t)g * D, a.ldqk, qs, 0.f);
  if (CH) load(a.decay + (size_t)head * D, a.ldd, extra, 1.f);
  if (tid < CT) {          // tokens beyond the end write nothing and keep everything
    float bt = 0.f, gt = 1.f;
    if (tid < n) {
      const size_t row = (size_t)(first + tid) * a.ldg + head;
      if (HAS_W) bt = sigmoid_f(a.first[row]);
      if (MODE == DELTA) gt = expf(-expf(a.A_log[head]) * softplus_f(a.second[row] + a.dt_bias[head]));
      if (MODE == STATE_SPACE) {
        bt = softplus_f(a.first[row] + a.dt_bias[head]);
        gt = expf(-expf(a.A_log[head]) * bt);
      }
    }
    beta[tid] = bt;
    gate[tid] = gt;
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  if (HAS_W) {             // unit vectors
    for (int i = warp; i < CT; i += 4) {
      float k2 = 0.f, q2 = 0.f;
#pragma unroll
      for (int d = lane; d < DP; d += 32) k2 = fmaf(ks[i][d], ks[i][d], k2), q2 = fmaf(qs[i][d], qs[i][d], q2);
      const float ik = 1.0f / sqrtf(warp_sum(k2) + 1e-6f), iq = a.qscale / sqrtf(warp_sum(q2) + 1e-6f);
#pragma unroll
      for (int d = lane; d < DP; d += 32) ks[i][d] *= ik, qs[i][d] *= iq;
    }
    __syncthreads();
  }
  if (!CH) {
    // k_i . k_j and q_i . k_j on the tensor cores, a warp 16 x 8 of either; the decays between come after
    const int gr = lane >> 2, t = lane & 3, nt = warp & 1, which = warp >> 1;
    if (which == 0 || HAS_W) {
      const float(*rows)[LD] = which ? ks : qs;
      float d[4] = {}, x[4] = {};
#pragma unroll 4
      for (int s = 0; s < DP / 8; ++s) {
        uint32_t hi[4], lo[4];
        split(rows[gr][8 * s + t], hi[0], lo[0]);
        split(rows[gr + 8][8 * s + t], hi[1], lo[1]);
        split(rows[gr][8 * s + t + 4], hi[2], lo[2]);
        split(rows[gr + 8][8 * s + t + 4], hi[3], lo[3]);
        mma3_apart(d, x, hi, lo, ks[8 * nt + gr][8 * s + t], ks[8 * nt + gr][8 * s + t + 4]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = gr + 8 * (e >> 1), j = 8 * nt + 2 * t + (e & 1);
        if (which) at[j][i] = whole(d[e], x[e], 1.f);
        else qk[i][j] = whole(d[e], x[e], 1.f);
      }
    }
    __syncthreads();
    const int j = tid >> 3, i0 = (tid & 7) * 2;       // two neighbouring rows of a column
    Product between = 1;
#pragma unroll
    for (int l = 1; l < CT; ++l)
      if (l > j && l <= i0) between *= gate[l];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + u;
      if (u && i > j) between *= gate[i];
      const float r = (float)between;
      float p = i >= j ? qk[i][j] * r : 0.f;
      if (MODE == STATE_SPACE && i >= j) p = p * beta[j] + (i == j ? a.skip[head] : 0.f);
      qk[i][j] = p;
      if (HAS_W) at[j][i] = i > j ? beta[i] * (at[j][i] * r) : 0.f;
    }
  } else {
    // a decay per channel stands inside the sums: eight lanes take a column j's sums, DP / 8 channels each, and carry
    // k_j times the decays since j from row to row; a warp's four columns walk the rows together,
    // bound by instructions: two channels in one (99 -> 94 us with the search above, heads of 128, 2,048 tokens)
    constexpr int E = DP / 8;
    const int j = tid >> 3, part = (tid & 7) * 4;      // four channels of every 32: eight lanes' 16 bytes side by side
    auto dim = [&](int e) { return part + (e & 3) + 8 * (e & ~3); };
    uint64_t kr[E / 2];                   // two neighbouring channels a register pair: half the instructions
#pragma unroll
    for (int e = 0; e < E; e += 2) kr[e / 2] = *(const uint64_t*)&ks[j][dim(e)];
    if (MODE == READ_BEFORE) {            // a token's own write, which it reads through the bonus
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (dim(e) < D) s = fmaf(qs[j][dim(e)] * a.bonus[(size_t)head * D + dim(e)], ks[j][dim(e)], s);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((tid & 7) == 0) qk[j][j] = s;
    }
#pragma unroll 1
    for (int i = warp * 4; i < CT; ++i) {
      uint64_t sq2 = 0, sk2 = 0;          // sums over the even and the odd channels
#pragma unroll
      for (int e = 0; e < E; e += 4) {
        const ulonglong2 q4 = *(const ulonglong2*)&qs[i][dim(e)], g4 = *(const ulonglong2*)&extra[i][dim(e)];
        ulonglong2 k4;
        if (HAS_W) k4 = *(const ulonglong2*)&ks[i][dim(e)];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint64_t& k2 = kr[e / 2 + u];
          if (MODE == READ_BEFORE) fma2(sq2, u ? q4.y : q4.x, k2);     // token i reads before its own decay
          if (i > j) mul2(k2, u ? g4.y : g4.x);
          if (MODE != READ_BEFORE) fma2(sq2, u ? q4.y : q4.x, k2);
          if (HAS_W) fma2(sk2, u ? k4.y : k4.x, k2);
        }
      }
      float sq = both(sq2), sk = HAS_W ? both(sk2) : 0.f;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (HAS_W) sk += __shfl_xor_sync(0xffffffffu, sk, o);
      }
      if ((tid & 7) == 0) {
        if (MODE != READ_BEFORE || i != j) qk[i][j] = i >= j ? sq : 0.f;
        if (HAS_W) at[j][i] = i > j ? beta[i] * sk : 0.f;
      }
    }
    for (int i = tid & 7; i < warp * 4; i += 8) {        // the rows that no column of this warp reaches
      qk[i][j] = 0.f;
      if (HAS_W) at[j][i] = 0.f;
    }
  }
  __syncthreads();
  // a thread a channel: Q~, Kd and G, and W by forward substitution; then T's columns in the same way
  auto solve = [&](float (&w)[CT]) {        // w <- (1 + A)^-1 w, a column at a time
#pragma unroll
    for (int j = 0; j < CT - 1; ++j) {
      asm volatile("" ::: "memory");        // A is read a column at a time: all of it at once would not fit the registers
#pragma unroll
      for (int i4 = (j + 1) / 4 * 4; i4 < CT; i4 += 4) {
        const float4 c = *(const float4*)&at[j][i4];
        if (i4 > j) w[i4] = fmaf(-c.x, w[j], w[i4]);
        if (i4 + 1 > j) w[i4 + 1] = fmaf(-c.y, w[j], w[i4 + 1]);
        if (i4 + 2 > j) w[i4 + 2] = fmaf(-c.z, w[j], w[i4 + 2]);
        if (i4 + 3 > j) w[i4 + 3] = fmaf(-c.w, w[j], w[i4 + 3]);
      }
    }
  };
  constexpr bool APART = !HAS_W && DP == 64;       // Kd by the other 64 threads
  if (tid < DP) {
    Product c = 1;
    float w[CT];
#pragma unroll
    for (int i = 0; i < CT; ++i) {
      const float gi = CH ? extra[i][tid] : gate[i];
      if (MODE == READ_BEFORE) {
        qs[i][tid] *= (float)c;
        c *= gi;
      } else {
        c *= gi;
        qs[i][tid] *= (float)c;
      }
      if (HAS_W) w[i] = beta[i] * ((float)c * ks[i][tid]);
    }
    a.blocks[((size_t)blockIdx.y * a.slots + slot) * B::FLOATS + B::G + tid] = (float)c;
    if (HAS_W) {
      solve(w);
#pragma unroll
      for (int i = 0; i < CT; ++i)
        if (!CH) extra[i][tid] = w[i];
    }
    if (HAS_W || !APART) {
      Product r = 1;
#pragma unroll
      for (int i = CT - 1; i >= 0; --i) {
        const float gi = CH ? extra[i][tid] : gate[i];
        ks[i][tid] *= MODE == STATE_SPACE ? (float)r * beta[i] : (float)r;
        r *= gi;
      }
    }
    if (HAS_W && CH) {
#pragma unroll
      for (int i = 0; i < CT; ++i) extra[i][tid] = w[i];
    }
  } else if (APART) {
    Product r = 1;
#pragma unroll
    for (int i = CT - 1; i >= 0; --i) {
      const float gi = CH ? extra[i][tid - 64] : gate[i];
      ks[i][tid - 64] *= MODE == STATE_SPACE ? (float)r * beta[i] : (float)r;
      r *= gi;
    }
  }
  if (HAS_W && tid >= 128 - CT) {
    const int c = tid - (128 - CT);
    float t[CT];
#pragma unroll
    for (int i = 0; i < CT; ++i) t[i] = i == c ? beta[i] : 0.f;
    solve(t);
#pragma unroll
    for (int i = 0; i < CT; ++i) tb[HAS_W ? i : 0][c] = t[i];
  }
  __syncthreads();
  float4* out = (float4*)(a.blocks + ((size_t)blockIdx.y * a.slots + slot) * B::FLOATS);
  for (int e = tid; e < DP * CT / 4; e += 128) {
    const int l = e & 31, gr = l >> 2, t = l & 3;
    const int row = 8 * ((e >> 5) & 1) + gr, col = 16 * (e >> 6) + 2 * t;
    out[B::Q / 4 + e] = make_float4(qs[row][col], qs[row][col + 1], qs[row][col + 8], qs[row][col + 9]);
    if (HAS_W) out[B::W / 4 + e] = make_float4(extra[row][col], extra[row][col + 1], extra[row][col + 8], extra[row][col + 9]);
    const int dim = 8 * (e >> 5) + gr;
    out[B::K / 4 + e] = make_float4(ks[2 * t][dim], ks[2 * t + 1][dim], ks[8 + 2 * t][dim], ks[9 + 2 * t][dim]);
  }
  if (tid < CT * CT / 4) {
    const int l = tid & 31, gr = l >> 2, t = l & 3, row = 8 * (tid >> 5) + gr;
    out[B::P / 4 + tid] = make_float4(qk[row][2 * t], qk[row][2 * t + 1], qk[row][8 + 2 * t], qk[row][9 + 2 * t]);
    if (HAS_W) out[B::T / 4 + tid] = make_float4(tb[row][2 * t], tb[row][2 * t + 1], tb[row][8 + 2 * t], tb[row][9 + 2 * t]);
  }
}

struct Scan {
  const float* blocks;
  int slots;
  const float* v;                       // rows of ldv floats, head h at h * V
  long long ldv;
  float* state;                         // [slots, H, 8 V lanes 4]: the order of recurrent.cu
  const int *cu, *seq_slot;
  float* y;                             // [ntok, H * V]
  int H, head0, V, lanes;               // lanes: 32 channels of a column each, as the state lies in memory
  float yscale;
  int wide;
};

// NV groups of 16 columns a CTA; a group's channels are shared by DS warps (their parts of U and Y meet in shared
// memory, added in one order).  One more warp brings the blocks of coming chunks by asynchronous copies, STAGES - 1
// ahead.
template <int DP, int DS, int NV, bool HAS_W, int STAGES>
__global__ void __launch_bounds__(32 * DS * NV + 32) chunk_scan_kernel(const Scan a) {
  using B = Block<DP, HAS_W>;
  constexpr int DW = DP / DS, NJ = DW / 8;
  constexpr int LV = 16 * NV + 4, STAGE = B::FLOATS + CT * LV;      // a chunk's block, then its rows of V
  extern __shared__ __align__(16) float smem[];
  float* exch = smem + STAGES * STAGE;             // [2][warps][16][32], with DS over 1
  pdl_wait_prior();
  const int b = blockIdx.x, head = a.head0 + blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gr = lane >> 2, t = lane & 3, part = warp % DS, V = a.V;
  const int col0 = (blockIdx.z * NV + warp / DS) * 16, d0 = part * DW;
  const int t0 = a.cu[b], t1 = a.cu[b + 1], chunks = (t1 - t0 + CT - 1) / CT;
  const float* blocks = a.blocks + ((size_t)blockIdx.y * a.slots + t0 / CT + b) * B::FLOATS;
  const int vcol0 = blockIdx.z * NV * 16;
  const float* vbase = a.v + (size_t)t0 * a.ldv + (size_t)head * V + vcol0;
  if (warp == DS * NV) {
    auto bring = [&](int c) {
      if (c < chunks) {
        const float* src = blocks + (size_t)c * B::FLOATS + 4 * lane;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem + (c % STAGES) * STAGE);
#pragma unroll 8
        for (int e = lane; e < B::FLOATS / 4; e += 32)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + 4 * (e - lane)) : "memory");
        if (a.wide) {                     // rows of V at 16-byte boundaries, whole groups of 16 columns; zeros beyond the end
          for (int e = lane; e < CT * NV * 4; e += 32) {
            const int i = e / (NV * 4), col = e % (NV * 4) * 4, in = c * CT + i < t1 - t0 && vcol0 + col < V;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 4 * (B::FLOATS + i * LV + col)),
                         "l"(in ? vbase + (size_t)(c * CT + i) * a.ldv + col : a.v), "r"(in ? 16 : 0)
                         : "memory");
          }
        } else {
          for (int e = lane; e < CT * NV * 16; e += 32) {
            const int i = e / (NV * 16), col = e % (NV * 16), in = c * CT + i < t1 - t0 && vcol0 + col < V;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * (B::FLOATS + i * LV + col)),
                         "l"(in ? vbase + (size_t)(c * CT + i) * a.ldv + col : a.v), "r"(in ? 4 : 0)
                         : "memory");
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) bring(c);
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    asm volatile("bar.sync 0;" ::: "memory");             // block 0 is there
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 3) : "memory");
      asm volatile("bar.sync 0;" ::: "memory");           // block c + 1 is there; all have left block c - 1
      bring(c + STAGES - 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    pdl_release_next();
    return;
  }
  const bool in0 = col0 + gr < V, in1 = col0 + gr + 8 < V;
  float* st = a.state + ((size_t)a.seq_slot[b] * a.H + head) * 32 * V * a.lanes;
  auto place = [&](int j, int col) {   // of channels d0 + 8 j + 2 t and the next
    const int d = d0 + 8 * j + 2 * t;
    return ((size_t)((d & 31) >> 2) * V + col) * a.lanes * 4 + (d >> 5) * 4 + (d & 3);
  };
  float S[NJ][4];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const bool in = d0 + 8 * j < 32 * a.lanes;
    const float2 x = in && in0 ? *(const float2*)(st + place(j, col0 + gr)) : make_float2(0.f, 0.f);
    const float2 z = in && in1 ? *(const float2*)(st + place(j, col0 + gr + 8)) : make_float2(0.f, 0.f);
    S[j][0] = x.x; S[j][1] = x.y; S[j][2] = z.x; S[j][3] = z.y;
  }
  // Y = Q~ S + P U of a chunk, of the tokens that this warp finishes (the first warp the first half, the second the second).
  // LATE: made under the next chunk's products with S, off the chain from chunk to chunk.  A delta rule's (2, 2) 200 -> 187 us
  // (2,048 tokens, 32 heads of 128 x 128), linear attention at heads of 64 90.6 -> 89.1; four warps a group, whose chains
  // are shorter, gain nothing.
  constexpr bool LATE = DS == 2;
  const bool finishes = DS == 1 || part < 2;
  constexpr int HALF = DS == 1 ? 2 : 1;           // halves of the tokens that a warp finishes
  float* yrow = a.y + ((size_t)t0 * a.H + head) * V + col0 + gr;
  uint32_t uhi[2][4] = {}, ulo[2][4] = {};        // the chunk before: what was written, Q~ S, its weights, whether all is finite
  float ykept[HALF][4] = {}, pu[HALF][4];
  const float4* pblk = (const float4*)smem + B::P / 4 + lane;
  bool u_clean = true;
  int left = 0;                                   // its rows that exist; none before the first
  auto reads = [&]() {
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const int nt = DS == 1 ? i : part & 1;
      if constexpr (LATE) {                       // without a branch: the first half takes zeros for the second's numbers
        const uint32_t second = nt ? ~0u : 0u;
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = uhi[1][e] & second, l[e] = ulo[1][e] & second;
        const float4 w = pblk[32 * nt];
        float x[4] = {};
        pu[i][0] = pu[i][1] = pu[i][2] = pu[i][3] = 0.f;
        mma3(pu[i], x, uhi[0], ulo[0], w.x, w.y);
        mma3(pu[i], x, h, l, w.z, w.w);
#pragma unroll
        for (int e = 0; e < 4; ++e) pu[i][e] = whole(pu[i][e], x[e], nt ? 2.f : 1.f);
      } else if (finishes) {
        mma_lower(pu[i], uhi, ulo, pblk[32 * nt], nt);
      }
    }
  };
  auto leaves = [&]() {
    if (!finishes) return;
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const int nt = DS == 1 ? i : part, row = 8 * nt + 2 * t;
      if (!u_clean) mend_lower(pu[i], uhi, ulo, pblk[32 * nt], nt, lane);
      float* to = yrow + (size_t)row * a.H * V;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (row + (e & 1) < left && (e < 2 ? in0 : in1))
          to[(size_t)(e & 1) * a.H * V + 8 * (e >> 1)] = (ykept[i][e] + pu[i][e]) * a.yscale;
    }
    if (left) yrow += (size_t)CT * a.H * V;
  };
  asm volatile("bar.sync 0;" ::: "memory");
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    const float4* blk = (const float4*)(smem + (c % STAGES) * STAGE);
    const float* vs = (const float*)blk + B::FLOATS + 2 * t * LV + warp / DS * 16 + gr;
    uint32_t vhi[2][4], vlo[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e)        // a left operand: columns gr, gr + 8 of tokens 2 t, 2 t + 1 of each half
        split(vs[(8 * h + (e >> 1)) * LV + 8 * (e & 1)], vhi[h][e], vlo[h][e]);
    if (LATE) reads();
    // W S and Q~ S over this warp's channels, transposed: 16 columns by 16 tokens
    float y[2][4] = {}, yx[2][4] = {}, u[2][4] = {}, ux[2][4] = {};
#pragma unroll
    for (int jp = 0; jp < NJ / 2; ++jp) {
      const int at = (d0 / 16 + jp) * 64 + lane;
      float4 qf[2], wf[2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        qf[nt] = blk[B::Q / 4 + at + 32 * nt];
        if (HAS_W) wf[nt] = blk[B::W / 4 + at + 32 * nt];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float(&s)[4] = S[2 * jp + h];
        uint32_t hi[4], lo[4];
        split(s[0], hi[0], lo[0]);
        split(s[2], hi[1], lo[1]);
        split(s[1], hi[2], lo[2]);
        split(s[3], hi[3], lo[3]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          if (HAS_W) mma3(u[nt], ux[nt], hi, lo, h ? wf[nt].z : wf[nt].x, h ? wf[nt].w : wf[nt].y);
          mma3(y[nt], yx[nt], hi, lo, h ? qf[nt].z : qf[nt].x, h ? qf[nt].w : qf[nt].y);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        y[nt][e] = whole(y[nt][e], yx[nt][e], NJ);
        if (HAS_W) u[nt][e] = -whole(u[nt][e], ux[nt][e], NJ);
      }
    if (LATE) leaves();
    // + T V: the last warp's work, or the last two's, a half of the tokens each
    if (HAS_W && part >= DS - (DS == 4 ? 2 : 1)) {
      const bool v_clean = all_finite(vlo);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        if (DS == 4 && nt != (part & 1)) continue;
        float d[4];
        const float4 w = blk[B::T / 4 + 32 * nt + lane];
        mma_lower(d, vhi, vlo, w, nt);
        if (!v_clean) mend_lower(d, vhi, vlo, w, nt, lane);
#pragma unroll
        for (int e = 0; e < 4; ++e) u[nt][e] += d[e];
      }
    }
    if (DS > 1) {
      float4* mine = (float4*)(exch + ((c & 1) * DS * NV + warp) * 512) + lane;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        if (HAS_W) mine[32 * nt] = make_float4(u[nt][0], u[nt][1], u[nt][2], u[nt][3]);
        mine[32 * (2 + nt)] = make_float4(y[nt][0], y[nt][1], y[nt][2], y[nt][3]);
      }
    }
    asm volatile("bar.sync 0;" ::: "memory");     // the warps' parts are there, and block c + 1; block c - 1 may go
    // the warps' parts, in their order: four numbers of part q (u of either half of the tokens, then y)
    auto gather = [&](int q, float (&to)[4]) {
      const float4* group = (const float4*)(exch + ((c & 1) * DS * NV + warp - part) * 512) + 32 * q + lane;
      float4 sum = group[0];
#pragma unroll
      for (int o = 1; o < DS; ++o) {
        const float4 v = group[128 * o];
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
      }
      to[0] = sum.x; to[1] = sum.y; to[2] = sum.z; to[3] = sum.w;
    };
    if (DS > 1 && HAS_W) {
      gather(0, u[0]);
      gather(1, u[1]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (HAS_W) {
        split(u[h][0], uhi[h][0], ulo[h][0]);
        split(u[h][2], uhi[h][1], ulo[h][1]);
        split(u[h][1], uhi[h][2], ulo[h][2]);
        split(u[h][3], uhi[h][3], ulo[h][3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) uhi[h][e] = vhi[h][e], ulo[h][e] = vlo[h][e];
      }
    }
    // S <- G S + Kd^T U
    const float* gs = (const float*)blk + B::G + d0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float4 kf = blk[B::K / 4 + (d0 / 8 + j) * 32 + lane];
      const float2 gf = *(const float2*)(gs + 8 * j + 2 * t);
      float d[4] = {}, x[4] = {};
      mma3(d, x, uhi[0], ulo[0], kf.x, kf.y);
      mma3(d, x, uhi[1], ulo[1], kf.z, kf.w);
      S[j][0] = fmaf(gf.x, S[j][0], whole(d[0], x[0], 2.f));
      S[j][1] = fmaf(gf.y, S[j][1], whole(d[1], x[1], 2.f));
      S[j][2] = fmaf(gf.x, S[j][2], whole(d[2], x[2], 2.f));
      S[j][3] = fmaf(gf.y, S[j][3], whole(d[3], x[3], 2.f));
    }
    if (DS > 1) {
      if (finishes) gather(2 + part, ykept[0]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) ykept[0][e] = y[0][e], ykept[HALF - 1][e] = y[1][e];
    }
    u_clean = !finishes || all_finite(ulo);
    pblk = blk + B::P / 4 + lane;
    left = t1 - t0 - c * CT;
    if (!LATE) {
      reads();
      leaves();
    }
  }
  if (LATE) {
    reads();
    leaves();
  }
  pdl_release_next();
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    if (d0 + 8 * j >= 32 * a.lanes) continue;
    if (in0) *(float2*)(st + place(j, col0 + gr)) = make_float2(S[j][0], S[j][1]);
    if (in1) *(float2*)(st + place(j, col0 + gr + 8)) = make_float2(S[j][2], S[j][3]);
  }
}

template <int DP, int DS, int NV, bool HAS_W, int STAGES>
static void launch_scan(const Scan& s, int nseq, int heads, cudaStream_t stream) {
  static_assert(STAGES >= 3, "a chunk's block is asked for before the one ahead of it is read");
  constexpr size_t smem = (STAGES * (Block<DP, HAS_W>::FLOATS + CT * (16 * NV + 4)) + (DS > 1 ? 2 * DS * NV * 512 : 0)) * sizeof(float);
  auto kernel = chunk_scan_kernel<DP, DS, NV, HAS_W, STAGES>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const dim3 grid(nseq, heads, (s.V + 16 * NV - 1) / (16 * NV));
  // without the attribute that lets it start under the kernel before it, so that its few, long blocks spread one to
  // an SM (see launch_scan in recurrent.cu)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = 32 * DS * NV + 32;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchKernelEx(&cfg, kernel, s);
}

template <int DP, int MODE>
static int run(Prepare p, Scan s, int ntok, int heads_at_once, cudaStream_t stream) {
  constexpr bool HAS_W = is_delta(MODE);
  p.slots = s.slots = chunk_slots(ntok, p.nseq);
  const bool ch = per_channel(MODE);
  p.wide = p.D == DP && p.ldqk % 4 == 0 && (!ch || p.ldd % 4 == 0) &&
           !(((uintptr_t)p.q | (uintptr_t)p.k | (ch ? (uintptr_t)p.decay : 0)) & 15);
  s.wide = s.V % 4 == 0 && s.ldv % 4 == 0 && ((uintptr_t)s.v & 15) == 0;
  for (int h = 0; h < p.H; h += heads_at_once) {
    const int heads = p.H - h < heads_at_once ? p.H - h : heads_at_once;
    p.head0 = s.head0 = h;
    gb_launch(chunk_prepare_kernel<DP, MODE>, dim3(p.slots, heads), 128, 0, stream, p);
    // us for a delta rule at heads of 128 x 128, preparation and all, by (DS, NV): 64 groups of 16 columns, 1,218 tokens:
    // (4, 1) 96, (2, 2) 137, (1, 4) 236; 256 groups, 2,048 tokens: 287, 278, 434; eight sequences of 113 to 910 tokens in two
    // launches of 1,024 groups: 609, 632, 684; sixteen of 3,200 tokens in all, 2,048 groups a launch: 473, 491, 451; twelve of
    // 1,500, 3,072 groups: 232, 242, 203.
    // Few groups leave the chain to itself and want it short (more warps a group); many fill the SMs either way and
    // want the least that a group costs.  Without W (the scan alone, us, 1,600 tokens, (4, 1) / (2, 2)): 64 groups of a state
    // space 86 / 117, 128 groups 100 / 117, four sequences' 512 groups 71 / 74, but sixteen's 2,048 groups 81 / 77.  Heads of
    // up to 64 (linear attention, (2, 1) / (2, 2) / (4, 1)): 64 groups 73 / 71 / 71, 256 groups 99 / 72 / 102 (256 CTAs of
    // two warps put two chains on most SMs and one on the rest), four sequences' 1,024 82 / 67 / 85.
    const long long groups = (long long)p.nseq * heads * ((s.V + 15) / 16);
    if constexpr (DP == 64)
      launch_scan<DP, 2, HAS_W ? 1 : 2, HAS_W, 4>(s, p.nseq, heads, stream);
    else if (groups <= (HAS_W ? 1 : 4) * 148)
      launch_scan<DP, 4, 1, HAS_W, 3>(s, p.nseq, heads, stream);
    else if (!HAS_W || groups <= 8 * 148)
      launch_scan<DP, 2, 2, HAS_W, 4>(s, p.nseq, heads, stream);
    else
      launch_scan<DP, 1, 4, HAS_W, 3>(s, p.nseq, heads, stream);
  }
  return gb_launch_status();
}

template <int MODE>
static int run_any(const Prepare& p, const Scan& s, int ntok, long long scratch_floats, cudaStream_t stream) {
  constexpr bool HAS_W = is_delta(MODE);
  if (p.nseq <= 0 || ntok <= 0) return 0;
  if (p.D <= 0 || p.D > 128 || s.V <= 0 || p.H <= 0 || p.G <= 0 || p.H % p.G || ((uintptr_t)s.state & 15) ||
      ((uintptr_t)p.blocks & 15))
    return GB_ERR_SIZE;
  const long long head = (long long)chunk_slots(ntok, p.nseq) * (p.D <= 64 ? Block<64, HAS_W>::FLOATS : Block<128, HAS_W>::FLOATS);
  const long long most = scratch_floats / head;
  if (most < 1) return GB_ERR_SIZE;
  const int heads = most < p.H ? (int)most : p.H;
  return p.D <= 64 ? run<64, MODE>(p, s, ntok, heads, stream) : run<128, MODE>(p, s, ntok, heads, stream);
}

static int lanes_for(int dims) { return dims <= 32 ? 1 : (dims <= 64 ? 2 : 4); }

}  // namespace

// Floats of scratch that one head of a step needs (delta: the two forms of the delta rule); the entry points below
// take as many heads at once as their scratch holds.
GB_EXPORT long long gb_chunk_floats(int ntok, int nseq, int dims, int delta) {
  const int per = dims <= 64 ? (delta ? Block<64, true>::FLOATS : Block<64, false>::FLOATS)
                             : (delta ? Block<128, true>::FLOATS : Block<128, false>::FLOATS);
  return (long long)chunk_slots(ntok, nseq) * per;
}

// The arguments are those of the entry points of recurrent.cu, with the step's tokens and the scratch; D up to 128.
// decay null: the delta rule with a decay per head (a_logit, A_log, dt_bias); else with a decay per channel.
GB_EXPORT int gb_chunk_delta_rule(const float* q, const float* k, const float* v, long long ld, const float* beta_logit,
                                  const float* a_logit, long long ldg, const float* A_log, const float* dt_bias, const float* decay,
                                  long long ldd, float* state, const int* cu, const int* seq_slot, float* y, int ntok, int nseq, int H,
                                  int G, int D, int V, float qscale, float* scratch, long long scratch_floats, cudaStream_t stream) {
  Prepare p = {q, k, ld, beta_logit, a_logit, ldg, decay, ldd, A_log, dt_bias, nullptr, nullptr, cu, nseq, H, G, D, 0, qscale, scratch, 0, 0};
  Scan s = {scratch, 0, v, ld, state, cu, seq_slot, y, H, 0, V, lanes_for(D), 1.0f, 0};
  return decay ? run_any<CHANNEL_DELTA>(p, s, ntok, scratch_floats, stream) : run_any<DELTA>(p, s, ntok, scratch_floats, stream);
}

GB_EXPORT int gb_chunk_ssd_scan(const float* x, const float* Bm, const float* Cm, long long ld, const float* dt_raw, long long ldd,
                                const float* A_log, const float* dt_bias, const float* skip, float* state, const int* cu,
                                const int* seq_slot, float* y, int ntok, int nseq, int H, int G, int N, int V, float* scratch,
                                long long scratch_floats, cudaStream_t stream) {
  Prepare p = {Cm, Bm, ld, dt_raw, nullptr, ldd, nullptr, 0, A_log, dt_bias, skip, nullptr, cu, nseq, H, G, N, 0, 1.0f, scratch, 0, 0};
  Scan s = {scratch, 0, x, ld, state, cu, seq_slot, y, H, 0, V, lanes_for(N), 1.0f, 0};
  return run_any<STATE_SPACE>(p, s, ntok, scratch_floats, stream);
}

GB_EXPORT int gb_chunk_wkv_scan(const float* r, const float* k, const float* w, long long ld, long long ldw, const float* v, long long ldv,
                                const float* bonus, float* state, const int* cu, const int* seq_slot, float* y, int ntok, int nseq,
                                int H, int D, int V, float yscale, float* scratch, long long scratch_floats, cudaStream_t stream) {
  Prepare p = {r, k, ld, nullptr, nullptr, 0, w, ldw, nullptr, nullptr, nullptr, bonus, cu, nseq, H, H, D, 0, 1.0f, scratch, 0, 0};
  Scan s = {scratch, 0, v, ldv, state, cu, seq_slot, y, H, 0, V, lanes_for(D), yscale, 0};
  return bonus ? run_any<READ_BEFORE>(p, s, ntok, scratch_floats, stream) : run_any<READ_AFTER>(p, s, ntok, scratch_floats, stream);
}
