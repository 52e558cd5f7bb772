// Plain causal grouped-query attention over the paged cache, for prompts and for decoding alike.
//
// One block per (TOKENS tokens, up to HEADS query heads of one kv head).  The query at position p of head h
// uses kv head h / (nh / nkv) and the keys lo..p, lo = max(0, p + 1 - window) with a window, else 0
// (src/model.rs:1187-1226).  Softmax is m = max, e = exp(s - m), e / sum (src/kernels.rs:1550-1561),
// computed online over chunks of 128 keys that start at lo.  The arithmetic for one
// (token, head) is a function of its position and of the cache contents alone, so whole
// prompts, single tokens and any batch give the same bits.  Everything is float32 arithmetic;
// it is the attention of the float32 engine and the plain reference of the faster kernels.
//
// A chunk's keys come into shared memory with neighbouring threads on neighbouring dims, a thread then
// walks the dims of its own key for all of the block's queries; its values take the same place with
// neighbouring threads on neighbouring positions, a thread then walks the positions of its own dim.  What
// bounds it: the shared-memory reads of those walks.  (Read from memory by the walking threads themselves,
// 32 lines a load, a query a block, the kernel was bound by its requests: 301 tokens of three prompts, 16
// heads of 128 over 8 kv heads, took 336 us a layer; in this form 55, the same sums in the same order.)
#include "common.cuh"

constexpr int CHUNK = 128;

// Rows of the chunk in shared memory: a key's dims, or a dim's positions, a multiple of 4 and 4 more.
static __host__ __device__ inline int quads(int n) { return (n + 3) & ~3; }
static __host__ __device__ inline size_t tile_floats(int hd) {
  const size_t keys = (size_t)CHUNK * (quads(hd) + 4), values = (size_t)hd * (CHUNK + 4);
  return keys > values ? keys : values;
}

__device__ __forceinline__ float dot4(float d, float4 a, float4 b) {      // one sum, in order
  d = fmaf(a.x, b.x, d);
  d = fmaf(a.y, b.y, d);
  d = fmaf(a.z, b.z, d);
  return fmaf(a.w, b.w, d);
}

// One or four neighbouring elements into shared memory as float32: copies in flight for float32 (waited for by
// copies_done), loads and conversions for bfloat16.
__device__ __forceinline__ void bring1(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void bring4(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void bring1(float* dst, const bf16* src) { *dst = to_f32(*src); }
__device__ __forceinline__ void bring4(float* dst, const bf16* src) {
#pragma unroll
  for (int e = 0; e < 4; ++e) dst[e] = to_f32(src[e]);
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T, int TOKENS, int HEADS>
__global__ void __launch_bounds__(CHUNK) attention_ref_kernel(
    const T* __restrict__ q, long long q_stride, T* __restrict__ out, long long out_stride,
    const T* __restrict__ kcache, const T* __restrict__ vcache, PagedKV kv, const int* __restrict__ tok_pos,
    const int* __restrict__ tok_seq, const int* __restrict__ seq_slot, int ntok, int nh, int window, int wide) {
  constexpr int NQ = TOKENS * HEADS, WARPS = CHUNK / 32;
  extern __shared__ __align__(16) float smem[];
  pdl_release_next();
  pdl_wait_prior();
  const int hd = kv.head_dim, hq = quads(hd), ld = hq + 4;
  float* qs = smem;                          // [NQ][hq], zeros beyond hd
  float* p = qs + NQ * hq;                   // [NQ][CHUNK]
  float* sums = p + NQ * CHUNK;              // [2][NQ][WARPS] the warps' maxima and sums
  float* tile = sums + 2 * NQ * WARPS;       // keys [CHUNK][ld], then values [hd][CHUNK + 4]
  size_t* rows = (size_t*)(tile + tile_floats(hd));   // [2][CHUNK] where a position's key and value lie
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rep = nh / kv.num_kv_heads, parts = (rep + HEADS - 1) / HEADS;
  const int g = blockIdx.y / parts, h0 = g * rep + blockIdx.y % parts * HEADS;
  const int live = min(HEADS, (g + 1) * rep - h0);
  const int last = min(ntok, (int)(blockIdx.x + 1) * TOKENS);
  // the block's tokens that read the same keys from the same first one on are worked together
  for (int t = blockIdx.x * TOKENS, together; t < last; t += together) {
    const int seq = tok_seq[t], slot = seq_slot[seq];
    const int lo = window > 0 ? max(0, tok_pos[t] + 1 - window) : 0;
    int hi[TOKENS], most = 0, fewest = 0x7fffffff;
    together = 0;
#pragma unroll
    for (int i = 0; i < TOKENS; ++i) {
      const bool in = together == i && t + i < last && tok_seq[t + i] == seq &&
                      (window > 0 ? max(0, tok_pos[t + i] + 1 - window) : 0) == lo;
      hi[i] = in ? tok_pos[t + i] + 1 : lo;
      most = max(most, hi[i]);
      if (in) fewest = min(fewest, hi[i]);
      together += in;
    }
    __syncthreads();                         // the tokens before have been worked
    for (int e = tid; e < NQ * hq; e += CHUNK) {
      const int c = e / hq, i = e % hq, tok = c / HEADS, h = c % HEADS;
      qs[e] = tok < together && h < live && i < hd ? to_f32(q[(size_t)(t + tok) * q_stride + (size_t)(h0 + h) * hd + i]) : 0.f;
    }
    float m[NQ], l[NQ], acc[NQ][2];
#pragma unroll
    for (int c = 0; c < NQ; ++c) m[c] = -INFINITY, l[c] = 0.f, acc[c][0] = acc[c][1] = 0.f;
    for (int c0 = lo; c0 < most; c0 += CHUNK) {
      const int n = min(CHUNK, most - c0);
      __syncthreads();                       // the chunk before has been read
      if (tid < n) {
        rows[tid] = kv.row(slot, c0 + tid, g);
        rows[CHUNK + tid] = kv.vcol(slot, c0 + tid, g);
      }
      __syncthreads();
      if (wide) {                            // hd is a multiple of 4 and rows start at 16-byte boundaries
        for (int e = tid; e < n * (hd / 4); e += CHUNK) {
          const int j = e / (hd / 4), i = e % (hd / 4) * 4;
          bring4(tile + j * ld + i, kcache + rows[j] + i);
        }
      } else {
        for (int j = warp; j < n; j += WARPS)
          for (int i = lane; i < hq; i += 32)
            if (i < hd) bring1(tile + j * ld + i, kcache + rows[j] + i);
            else tile[j * ld + i] = 0.f;
      }
      copies_done();
      __syncthreads();
      float s[NQ];
#pragma unroll
      for (int c = 0; c < NQ; ++c) s[c] = 0.f;
      if (tid < n) {
        const float4* kr = (const float4*)(tile + tid * ld);
#pragma unroll 2
        for (int i = 0; i < hq / 4; ++i) {
          const float4 kd = kr[i];
#pragma unroll
          for (int c = 0; c < NQ; ++c) s[c] = dot4(s[c], ((const float4*)(qs + c * hq))[i], kd);
        }
      }
      // maxima and sums of all queries meet over the four warps at once, in the order of block_max and block_sum
#pragma unroll
      for (int c = 0; c < NQ; ++c) {
        s[c] = c0 + tid < hi[c / HEADS] ? s[c] : -INFINITY;
        const float v = warp_max(s[c]);
        if (lane == 0) sums[c * WARPS + warp] = v;
      }
      __syncthreads();                       // also: every thread is past its own key
      const bool whole = wide && kv.page_size % 4 == 0 && c0 % 4 == 0;     // four positions side by side in one page
      if (whole) {
        for (int e = tid; e < (n / 4) * hd; e += CHUNK) {
          const int d = e / (n / 4), j = e % (n / 4) * 4;
          bring4(tile + d * (CHUNK + 4) + j, vcache + rows[CHUNK + j] + (size_t)d * kv.page_size);
        }
      }
      for (int j0 = whole ? n / 4 * 4 : 0; j0 < n; j0 += 32)
        for (int d = warp; d < hd; d += WARPS)
          if (j0 + lane < n) bring1(tile + d * (CHUNK + 4) + j0 + lane, vcache + rows[CHUNK + j0 + lane] + (size_t)d * kv.page_size);
      float alpha[NQ];
#pragma unroll
      for (int c = 0; c < NQ; ++c) {
        const float* w = sums + c * WARPS;
        const float m_new = fmaxf(m[c], fmaxf(fmaxf(w[0], w[2]), fmaxf(w[1], w[3])));
        // a token none of whose keys lie in this chunk keeps what it has
        const bool any = c0 < hi[c / HEADS];
        const float pj = c0 + tid < hi[c / HEADS] ? expf(s[c] - m_new) : 0.f;
        p[c * CHUNK + tid] = pj;
        const float v = warp_sum(pj);
        if (lane == 0) sums[(NQ + c) * WARPS + warp] = v;
        alpha[c] = any ? expf(m[c] - m_new) : 1.f;
        if (any) m[c] = m_new;
      }
      copies_done();
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NQ; ++c) {
        const float* w = sums + (NQ + c) * WARPS;
        if (c0 < hi[c / HEADS]) l[c] = l[c] * alpha[c] + ((w[0] + w[2]) + (w[1] + w[3]));
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int d = tid + u * CHUNK;
        if (d >= hd) continue;
        const float4* vr = (const float4*)(tile + d * (CHUNK + 4));
#pragma unroll
        for (int c = 0; c < NQ; ++c) acc[c][u] *= alpha[c];
        // positions that every query of the group sees, four at a time, then each query's own last ones
        const int least = min(CHUNK, max(0, fewest - c0)) / 4 * 4;
#pragma unroll 2
        for (int j = 0; j < least / 4; ++j) {
          const float4 vd = vr[j];
#pragma unroll
          for (int c = 0; c < NQ; ++c) acc[c][u] = dot4(acc[c][u], ((const float4*)(p + c * CHUNK))[j], vd);
        }
        for (int j = least; j < n; ++j) {
          const float vd = tile[d * (CHUNK + 4) + j];
#pragma unroll
          for (int c = 0; c < NQ; ++c)
            if (c0 + j < hi[c / HEADS]) acc[c][u] = fmaf(p[c * CHUNK + j], vd, acc[c][u]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < NQ; ++c) {
      if (c / HEADS >= together || c % HEADS >= live) continue;
      T* orow = out + (size_t)(t + c / HEADS) * out_stride + (size_t)(h0 + c % HEADS) * hd;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int d = tid + u * CHUNK;
        if (d < hd) orow[d] = from_f32<T>(acc[c][u] / l[c]);
      }
    }
  }
}

// Prompts: the same sums in the same order with more of them in registers.  A block is TOKENS tokens and up to HEADS heads, 16
// queries in all, four a warp; a lane works four keys (lane, + 32, + 64, + 96: what four warps' lanes are above) for its warp's
// queries, then four dims: eight 16-byte reads feed 64 multiply-adds where a key a thread for eight queries reads nine for 32.
// Keys up to 128 wide.  301 tokens of three prompts, 16 heads of 128 over 8: 55 -> 43 us a layer (two rounds of loads, walks and
// sums a chunk, one after the other, are most of that).
template <typename T, int TOKENS, int HEADS>
__global__ void __launch_bounds__(CHUNK) attention_ref_tile_kernel(
    const T* __restrict__ q, long long q_stride, T* __restrict__ out, long long out_stride,
    const T* __restrict__ kcache, const T* __restrict__ vcache, PagedKV kv, const int* __restrict__ tok_pos,
    const int* __restrict__ tok_seq, const int* __restrict__ seq_slot, int ntok, int nh, int window, int wide) {
  constexpr int NQ = TOKENS * HEADS, WARPS = CHUNK / 32, QW = NQ / WARPS, KL = CHUNK / 32;   // QW queries a warp, KL keys or dims a lane
  static_assert(NQ == 16 && QW == 4 && KL == 4, "four queries by four keys a lane");
  extern __shared__ __align__(16) float smem[];
  pdl_release_next();
  pdl_wait_prior();
  const int hd = kv.head_dim, hq = quads(hd), ld = hq + 4;
  float* qs = smem;                          // [NQ][hq], zeros beyond hd
  float* p = qs + NQ * hq;                   // [NQ][CHUNK]
  float* tile = p + NQ * CHUNK;              // keys [CHUNK][ld], then values [hd][CHUNK + 4]
  size_t* rows = (size_t*)(tile + tile_floats(hd));   // [2][CHUNK] where a position's key and value lie
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rep = nh / kv.num_kv_heads, parts = (rep + HEADS - 1) / HEADS;
  const int g = blockIdx.y / parts, h0 = g * rep + blockIdx.y % parts * HEADS;
  const int live = min(HEADS, (g + 1) * rep - h0);
  // from the last tokens, which see the most keys, to the first: what the last round of blocks holds is short
  const int bx = gridDim.x - 1 - blockIdx.x, last = min(ntok, (bx + 1) * TOKENS);
  for (int t = bx * TOKENS, together; t < last; t += together) {
    const int seq = tok_seq[t], slot = seq_slot[seq];
    const int lo = window > 0 ? max(0, tok_pos[t] + 1 - window) : 0;
    int hi[QW], most = 0, fewest = 0x7fffffff;
    together = 0;
#pragma unroll
    for (int e = 0; e < QW; ++e) hi[e] = lo;
    for (int i = 0; i < TOKENS; ++i) {
      if (t + i >= last || tok_seq[t + i] != seq || (window > 0 ? max(0, tok_pos[t + i] + 1 - window) : 0) != lo) break;
      const int end = tok_pos[t + i] + 1;
      most = max(most, end);
      fewest = min(fewest, end);
      ++together;
#pragma unroll
      for (int e = 0; e < QW; ++e)
        if ((warp * QW + e) / HEADS == i) hi[e] = end;
    }
    __syncthreads();                         // the tokens before have been worked
    for (int e = tid; e < NQ * hq; e += CHUNK) {
      const int c = e / hq, i = e % hq, tok = c / HEADS, h = c % HEADS;
      qs[e] = tok < together && h < live && i < hd ? to_f32(q[(size_t)(t + tok) * q_stride + (size_t)(h0 + h) * hd + i]) : 0.f;
    }
    float m[QW], l[QW], acc[QW][KL];
#pragma unroll
    for (int c = 0; c < QW; ++c) {
      m[c] = -INFINITY;
      l[c] = 0.f;
#pragma unroll
      for (int u = 0; u < KL; ++u) acc[c][u] = 0.f;
    }
    const float* myq = qs + warp * QW * hq;
    float* myp = p + warp * QW * CHUNK;
    for (int c0 = lo; c0 < most; c0 += CHUNK) {
      const int n = min(CHUNK, most - c0);
      __syncthreads();                       // the chunk before has been read
      if (tid < n) {
        rows[tid] = kv.row(slot, c0 + tid, g);
        rows[CHUNK + tid] = kv.vcol(slot, c0 + tid, g);
      }
      __syncthreads();
      if (wide) {
        for (int e = tid; e < n * (hd / 4); e += CHUNK) {
          const int j = e / (hd / 4), i = e % (hd / 4) * 4;
          bring4(tile + j * ld + i, kcache + rows[j] + i);
        }
      } else {
        for (int j = warp; j < n; j += WARPS)
          for (int i = lane; i < hq; i += 32)
            if (i < hd) bring1(tile + j * ld + i, kcache + rows[j] + i);
            else tile[j * ld + i] = 0.f;
      }
      copies_done();
      __syncthreads();
      float s[QW][KL];
#pragma unroll
      for (int c = 0; c < QW; ++c)
#pragma unroll
        for (int u = 0; u < KL; ++u) s[c][u] = 0.f;
#pragma unroll 2
      for (int i = 0; i < hq / 4; ++i) {     // rows beyond n hold what was there: their scores are not used
        float4 kd[KL];
#pragma unroll
        for (int u = 0; u < KL; ++u) kd[u] = ((const float4*)(tile + (lane + 32 * u) * ld))[i];
#pragma unroll
        for (int c = 0; c < QW; ++c) {
          const float4 qd = ((const float4*)(myq + c * hq))[i];
#pragma unroll
          for (int u = 0; u < KL; ++u) s[c][u] = dot4(s[c][u], qd, kd[u]);
        }
      }
      __syncthreads();                       // every warp is past the keys
      const bool whole = wide && kv.page_size % 4 == 0 && c0 % 4 == 0;     // four positions side by side in one page
      if (whole) {
        for (int e = tid; e < (n / 4) * hd; e += CHUNK) {
          const int d = e / (n / 4), j = e % (n / 4) * 4;
          bring4(tile + d * (CHUNK + 4) + j, vcache + rows[CHUNK + j] + (size_t)d * kv.page_size);
        }
      }
      for (int j0 = whole ? n / 4 * 4 : 0; j0 < n; j0 += 32)
        for (int d = warp; d < hd; d += WARPS)
          if (j0 + lane < n) bring1(tile + d * (CHUNK + 4) + j0 + lane, vcache + rows[CHUNK + j0 + lane] + (size_t)d * kv.page_size);
#pragma unroll
      for (int c = 0; c < QW; ++c) {
        float top = -INFINITY;
#pragma unroll
        for (int u = 0; u < KL; ++u) {
          s[c][u] = c0 + lane + 32 * u < hi[c] ? s[c][u] : -INFINITY;
          top = fmaxf(top, s[c][u]);
        }
        const float m_new = fmaxf(m[c], warp_max(top));
        const bool any = c0 < hi[c];         // a token none of whose keys lie in this chunk keeps what it has
        float w[KL];
#pragma unroll
        for (int u = 0; u < KL; ++u) {
          const float pj = c0 + lane + 32 * u < hi[c] ? expf(s[c][u] - m_new) : 0.f;
          myp[c * CHUNK + lane + 32 * u] = pj;
          w[u] = warp_sum(pj);
        }
        const float alpha = any ? expf(m[c] - m_new) : 1.f;
        if (any) {
          m[c] = m_new;
          l[c] = l[c] * alpha + ((w[0] + w[2]) + (w[1] + w[3]));
        }
#pragma unroll
        for (int u = 0; u < KL; ++u) acc[c][u] *= alpha;
      }
      copies_done();
      __syncthreads();
      // positions that every query of the group sees, four at a time, then each query's own last ones
      const int least = min(CHUNK, max(0, fewest - c0)) / 4 * 4;
      const float* vr[KL];
#pragma unroll
      for (int u = 0; u < KL; ++u) vr[u] = tile + min(lane + 32 * u, hd - 1) * (CHUNK + 4);      // dims beyond the head's go nowhere
#pragma unroll 2
      for (int j = 0; j < least; j += 4) {
        float4 vd[KL];
#pragma unroll
        for (int u = 0; u < KL; ++u) vd[u] = *(const float4*)(vr[u] + j);
#pragma unroll
        for (int c = 0; c < QW; ++c) {
          const float4 pd = *(const float4*)(myp + c * CHUNK + j);
#pragma unroll
          for (int u = 0; u < KL; ++u) acc[c][u] = dot4(acc[c][u], pd, vd[u]);
        }
      }
      for (int j = least; j < n; ++j) {
#pragma unroll
        for (int c = 0; c < QW; ++c)
          if (c0 + j < hi[c]) {
            const float pj = myp[c * CHUNK + j];
#pragma unroll
            for (int u = 0; u < KL; ++u) acc[c][u] = fmaf(pj, vr[u][j], acc[c][u]);
          }
      }
    }
#pragma unroll
    for (int e = 0; e < QW; ++e) {
      const int c = warp * QW + e;
      if (c / HEADS >= together || c % HEADS >= live) continue;
      T* orow = out + (size_t)(t + c / HEADS) * out_stride + (size_t)(h0 + c % HEADS) * hd;
#pragma unroll
      for (int u = 0; u < KL; ++u)
        if (lane + 32 * u < hd) orow[lane + 32 * u] = from_f32<T>(acc[e][u] / l[e]);
    }
  }
}

template <typename T, int TOKENS, int HEADS, typename... Args>
static int launch_ref_tile(int ntok, int rep, const PagedKV& kv, cudaStream_t stream, Args... args) {
  constexpr int NQ = TOKENS * HEADS;
  const size_t smem = (NQ * (size_t)(quads(kv.head_dim) + CHUNK) + tile_floats(kv.head_dim)) * sizeof(float) + 2 * CHUNK * sizeof(size_t);
  auto kernel = attention_ref_tile_kernel<T, TOKENS, HEADS>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const dim3 grid((ntok + TOKENS - 1) / TOKENS, kv.num_kv_heads * ((rep + HEADS - 1) / HEADS));
  gb_launch(kernel, grid, CHUNK, smem, stream, args...);
  return gb_launch_status();
}

template <typename T, int TOKENS, int HEADS, typename... Args>
static int launch_ref(int ntok, int rep, const PagedKV& kv, cudaStream_t stream, Args... args) {
  constexpr int NQ = TOKENS * HEADS;
  const size_t smem = (NQ * (size_t)(quads(kv.head_dim) + CHUNK + 2 * CHUNK / 32) + tile_floats(kv.head_dim)) * sizeof(float) +
                      2 * CHUNK * sizeof(size_t);
  auto kernel = attention_ref_kernel<T, TOKENS, HEADS>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const dim3 grid((ntok + TOKENS - 1) / TOKENS, kv.num_kv_heads * ((rep + HEADS - 1) / HEADS));
  gb_launch(kernel, grid, CHUNK, smem, stream, args...);
  return gb_launch_status();
}

// Query heads of a kv head that a block works.
static int block_heads(int rep) { return rep >= 3 ? 4 : rep; }

// The form for a step whose neighbouring tokens share their sequence and first key, by its size: 16 (sixteen queries a block), 4
// (four tokens) or 1 (one).  The larger forms read a chunk's keys for more queries but leave fewer blocks.  us, one / four tokens /
// sixteen queries, heads of 128: 16 heads over 8: 100 tokens 25 / 18 / 18, 150 43 / 39 / 29, 301 110 / 79 / 49, 1,024 868 / 553 / 285; 32 over
// 8: 64 tokens 22 / 17 / 16, 100 29 / 21 / 21, 301 128 / 91 / 78; 8 over 8: 200 tokens 51 / 27 / 32, 301 92 / 50 / 46; 16 over 16: 100 tokens
// 35 / 16 / 21, 150 60 / 34 / 33, 200 89 / 45 / 36.  Sixteen queries want a block an SM (147 blocks: 145 tokens, 73, 289, 145 of those),
// and heads of up to 128; four tokens two.  With two or four heads a block the second line lies at or beyond the first: four tokens
// are then for wider heads, and for steps whose tokens share less (see the caller's rule).
static int form_by_size(int ntok, int nh, int nkv, int hd) {
  const int heads = block_heads(nh / nkv), columns = nkv * ((nh / nkv + heads - 1) / heads), tile_tokens = 16 / heads;
  if (hd <= CHUNK && (long long)((ntok + tile_tokens - 1) / tile_tokens) * columns >= 148) return 16;
  return (long long)ntok * columns >= 4 * 2 * 148 ? 4 : 1;
}
GB_EXPORT int gb_attention_ref_form(int ntok, int nh, int nkv, int hd) {
  return ntok > 0 && nkv > 0 && nh >= nkv && nh % nkv == 0 ? form_by_size(ntok, nh, nkv, hd) : 1;
}

// q: [ntok, nh, hd] rows q_stride apart (already normed, rotated, scaled); out likewise.  form: 1, 4 or 16 as above, or 0: by size.
// Tokens of a block that do not share their sequence and first key are worked one after the other.  The same bits whatever it is.
GB_EXPORT int gb_attention_ref(const void* q, long long q_stride, void* out, long long out_stride, int dtype,
                               const void* kcache, const void* vcache, const int* page_table, int table_width,
                               int page_size, int nkv, int hd, const int* tok_pos, const int* tok_seq,
                               const int* seq_slot, int ntok, int nh, int window, int form, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  if (hd <= 0 || hd > 2 * CHUNK || nkv <= 0 || nh % nkv) return GB_ERR_SIZE;
  if (form != 0 && form != 1 && form != 4 && form != 16) return GB_ERR_ARG;
  if (form == 16 && hd > CHUNK) return GB_ERR_SIZE;
  PagedKV kv{page_table, table_width, page_size, nkv, hd};
  const int rep = nh / nkv, heads = block_heads(rep);
  if (form == 0) form = form_by_size(ntok, nh, nkv, hd);
  const bool four = form == 4, tiles = form == 16;
  const int wide = hd % 4 == 0 && (((uintptr_t)kcache | (uintptr_t)vcache) & 15) == 0;
#define REF(T, TOKENS, HEADS)                                                                                              \
  launch_ref<T, TOKENS, HEADS>(ntok, rep, kv, stream, (const T*)q, q_stride, (T*)out, out_stride, (const T*)kcache, (const T*)vcache, \
                               kv, tok_pos, tok_seq, seq_slot, ntok, nh, window, wide)
#define REF_TILE(T, TOKENS, HEADS)                                                                                          \
  launch_ref_tile<T, TOKENS, HEADS>(ntok, rep, kv, stream, (const T*)q, q_stride, (T*)out, out_stride, (const T*)kcache, (const T*)vcache, \
                                    kv, tok_pos, tok_seq, seq_slot, ntok, nh, window, wide)
#define REF_TILES(T) (heads == 1 ? REF_TILE(T, 16, 1) : heads == 2 ? REF_TILE(T, 8, 2) : REF_TILE(T, 4, 4))
#define REF_HEADS(T) (heads == 1 ? (four ? REF(T, 4, 1) : REF(T, 1, 1)) : heads == 2 ? (four ? REF(T, 4, 2) : REF(T, 1, 2)) \
                                                                                   : (four ? REF(T, 4, 4) : REF(T, 1, 4)))
  if (dtype == GB_F32) return tiles ? REF_TILES(float) : REF_HEADS(float);
  if (dtype == GB_BF16) return tiles ? REF_TILES(bf16) : REF_HEADS(bf16);
#undef REF_HEADS
#undef REF_TILES
#undef REF_TILE
#undef REF
  return GB_ERR_DTYPE;
}
