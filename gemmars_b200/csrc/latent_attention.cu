// Latent attention: the plain kernels.
//
// A latent attention layer caches, per position, one row  [c (rank dims) | k_rot (rot dims)]
// shared by all heads: c is the RMS-normed low-rank projection of the layer's input and k_rot a
// rotated key part.  A head's unrotated key is  W_uk[h] c  and its value  W_uv[h] c.  Both
// matrices are moved to the query side, so attention runs on the cached rows as they are:
//
//   qa[t, h, :rank] = W_uk[h]^T q_nope[t, h]      (gb_heads_gemm, w = W_uk[h] transposed)
//   qa[t, h, rank:] = rotate(q_rot[t, h])
//   s[t, h, j]      = qa[t, h] . row[j]           (q already carries the score scale)
//   p               = softmax_j over j <= pos(t)  (float32)
//   ol[t, h]        = sum_j p[j] row[j, :rank]
//   o[t, h]         = gate[t, h] * W_uv[h] ol[t, h]   (gb_heads_gemm with a row scale), or with a gate per
//                    output number  sigmoid(z[t, h, :]) * W_uv[h] ol[t, h]
//
// This unit holds what every precision and size can use: the kernel that norms, rotates and
// writes the cache row (gb_latent_prepare), the per-head products (gb_heads_gemm, FFMA), the
// attention itself one (token, head) per block (gb_latent_attention_ref), and the stand-alone
// rotation of interleaved pairs (gb_rope_pairs).  The arithmetic for one (token, head) depends on
// its position and the cache alone, so prompts, single tokens and any batch give the same bits.
#include "mma.cuh"

// Rotation of a pair (u, v) -> (u cos - v sin, v cos + u sin), angle = float(pos) * inv_freq[i], all in
// float32, cosine and sine times `mag`.  Pair i < rot/2 is dims (2i, 2i+1), or with the half layout (i, i + rot/2).
__device__ __forceinline__ float2 cos_sin(float angle, float mag) {
  float s, c;
  sincosf(angle, &s, &c);
  return make_float2(c * mag, s * mag);
}
__device__ __forceinline__ void rotate_pair(float u, float v, float2 cs, float& ou, float& ov) {
  ou = u * cs.x - v * cs.y;
  ov = v * cs.x + u * cs.y;
}

// A second copy of the cache rows (latents null: not wanted): latents and rotated key parts, rows ldl and ldr apart, token
// by token.  With `cu` it is for keys and values that a prompt expands per head: sequence b's rows then start at
// (cu[b] / 8 + b) * 8 (a multiple of 8, with room for every sequence's last, partly filled eight), the queries lie
// head by head as [dim | rd], and the `rows` rows that no token fills are written as zeros.
template <typename T>
struct Copy {
  T *latents, *rotated;
  long long ldl, ldr;
  const int* cu;
  long long rows;
  __device__ __forceinline__ long long row(int b, int t) const { return (long long)(cu[b] / 8 + b) * 8 + (t - cu[b]); }
};

template <typename T> __device__ __forceinline__ void store4(T* to, float a, float b, float c, float d);
template <> __device__ __forceinline__ void store4<float>(float* to, float a, float b, float c, float d) { *(float4*)to = make_float4(a, b, c, d); }
template <> __device__ __forceinline__ void store4<bf16>(bf16* to, float a, float b, float c, float d) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b), q = __floats2bfloat162_rn(c, d);
  *(uint2*)to = make_uint2(*(const uint32_t*)&p, *(const uint32_t*)&q);
}

// A warp per token for its cache row, and a thread for every QUADS quads of its queries (or, where those are no quads, dims or
// pairs): one where few tokens leave the chip idle, two loads in flight a thread for prompts.  Inputs are the float32 results of the layer's projections.  What bounds it is a chain of loads (position,
// slot, page, the row), so nothing waits for a block: a warp holds a token's row and sums it alone, and a query's angles are
// taken where they are used.  `wide`: interleaved pairs, everything in fours.  16 heads of 128 + 64 over rows of 512 + 64, with
// the wait for the kernel before (us; a block a token, its row twice through memory, its angles through shared memory / so):
// 2,048 tokens 20.9 / 16.6, 16 tokens 10.6 / 8.5; the layer of 2,048 tokens, with the rows' zeros written here and not by two fills,
// 145.5 / 132.0 where one side's runs differ by up to a fifth; of 16 single tokens 65.7 / 65.4.
constexpr int PREPARE_THREADS = 128, PREPARE_QUADS = 2, ROW_HELD = 16;
template <typename T, int QUADS>
__global__ void __launch_bounds__(PREPARE_THREADS) latent_prepare_kernel(
    const float* __restrict__ q_in, long long ldq, const float* __restrict__ kv_in, long long ldkv,
    const float* __restrict__ g_in, long long ldg, const float* __restrict__ norm_w, float eps,
    const float* __restrict__ inv_freq, int rot, float q_scale, T* __restrict__ q_nope, long long ldqn,
    T* __restrict__ q_lat, long long ldql, float* __restrict__ gate, T* __restrict__ cache,
    const int* __restrict__ page_table, int table_width, int page_size, const int* __restrict__ tok_pos,
    const int* __restrict__ tok_seq, const int* __restrict__ seq_slot, int ntok, int H, int dim, int rd, int rank,
    Copy<T> ex, int half_layout, float rot_mag, int wide, int row_blocks, int token_blocks) {
  pdl_release_next();
  pdl_wait_prior();
  const int halves = rd / 2 + (rd & 1);
  if ((int)blockIdx.x >= row_blocks) {
    // queries: the unrotated dims go to the absorbing product and the rotated ones straight into qa, or both into the
    // head's own row
    const int qd = dim + rd, rot_at = ex.cu ? dim : rank, nope_head = ex.cu ? qd : dim, lat_head = rot_at + rd;
    const int block = (int)blockIdx.x - row_blocks, t = block / token_blocks;
    const float* q = q_in + (size_t)t * ldq;
    const float fpos = (float)tok_pos[t];
    const int first = (block - t * token_blocks) * (QUADS * PREPARE_THREADS) + threadIdx.x;
    if (wide) {       // four neighbouring dims at a time
      const int quads = qd / 4, total = H * quads;
      float4 v[QUADS];
      int h[QUADS], d[QUADS];
#pragma unroll
      for (int u = 0; u < QUADS; ++u) {
        const int e = first + u * PREPARE_THREADS;
        h[u] = e < total ? e / quads : -1;
        d[u] = (e - h[u] * quads) * 4;
        if (h[u] >= 0) v[u] = *(const float4*)(q + h[u] * qd + d[u]);
      }
#pragma unroll
      for (int u = 0; u < QUADS; ++u) {
        if (h[u] < 0) continue;
        float o[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
        const bool turned = d[u] >= dim;
        if (turned) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = (d[u] - dim) / 2 + e;
            if (2 * i < rot) rotate_pair(o[2 * e], o[2 * e + 1], cos_sin(fpos * inv_freq[i], rot_mag), o[2 * e], o[2 * e + 1]);
          }
        }
        T* dst = turned ? q_lat + (size_t)t * ldql + (size_t)h[u] * lat_head + rot_at + d[u] - dim
                        : q_nope + (size_t)t * ldqn + (size_t)h[u] * nope_head + d[u];
        store4(dst, o[0] * q_scale, o[1] * q_scale, o[2] * q_scale, o[3] * q_scale);
      }
      return;
    }
    const int units = dim + halves;
    for (int u = 0; u < QUADS; ++u) {
      const int e = first + u * PREPARE_THREADS;
      if (e >= H * units) return;
      const int h = e / units, unit = e - h * units;
      const float* src = q + h * qd;
      if (unit < dim) {
        q_nope[(size_t)t * ldqn + (size_t)h * nope_head + unit] = from_f32<T>(src[unit] * q_scale);
        continue;
      }
      const int i = unit - dim;
      const bool turns = 2 * i < rot;
      const int a = turns && half_layout ? i : 2 * i, b = turns && half_layout ? i + rot / 2 : 2 * i + 1;
      T* dst = q_lat + (size_t)t * ldql + (size_t)h * lat_head + rot_at;
      float x = src[dim + a], y = b < rd ? src[dim + b] : 0.f;
      if (turns) rotate_pair(x, y, cos_sin(fpos * inv_freq[i], rot_mag), x, y);
      dst[a] = from_f32<T>(x * q_scale);
      if (b < rd) dst[b] = from_f32<T>(y * q_scale);
    }
    return;
  }
  const int t = (int)blockIdx.x * (PREPARE_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= ntok) return;
  const int pos = tok_pos[t];
  const float* kv = kv_in + (size_t)t * ldkv;
  float x[ROW_HELD];                        // the row's first 512 numbers stay in registers
#pragma unroll
  for (int u = 0; u < ROW_HELD; ++u) x[u] = lane + 32 * u < rank ? kv[lane + 32 * u] : 0.f;
  // the row goes into the paged cache and, when asked for, into the rows to be expanded as well
  T *lat0 = nullptr, *lat1 = nullptr, *key0 = nullptr, *key1 = nullptr;
  if (cache != nullptr) {
    const int slot = seq_slot[tok_seq[t]];
    const int page = page_table[(size_t)slot * table_width + (pos / page_size) % table_width];
    lat0 = cache + ((size_t)page * page_size + pos % page_size) * (size_t)(rank + rd);
    key0 = lat0 + rank;
  }
  if (ex.latents != nullptr) {
    const long long row = ex.cu ? ex.row(tok_seq[t], t) : t;
    lat1 = ex.latents + row * ex.ldl;
    key1 = ex.rotated + row * ex.ldr;
    if (ex.cu) {                            // rows from this token's to the next one's, and before the first
      const long long next = t + 1 < ntok ? ex.row(tok_seq[t + 1], t + 1) : ex.rows;
      for (long long r = t > 0 ? row + 1 : 0; r < next; ++r) {
        if (r == row) continue;
        for (int i = lane; i < rank; i += 32) ex.latents[r * ex.ldl + i] = from_f32<T>(0.f);
        for (int i = lane; i < rd; i += 32) ex.rotated[r * ex.ldr + i] = from_f32<T>(0.f);
      }
    }
  }
  // the shared rotated key part: pairs below `rot` turn, the rest passes
  for (int i = lane; i < halves; i += 32) {
    const bool turns = 2 * i < rot;
    const int a = turns && half_layout ? i : 2 * i, b = turns && half_layout ? i + rot / 2 : 2 * i + 1;
    float u = kv[rank + a], v = b < rd ? kv[rank + b] : 0.f;
    if (turns) rotate_pair(u, v, cos_sin((float)pos * inv_freq[i], rot_mag), u, v);
    for (int copy = 0; copy < 2; ++copy) {
      T* key = copy ? key1 : key0;
      if (!key) continue;
      key[a] = from_f32<T>(u);
      if (b < rd) key[b] = from_f32<T>(v);
    }
  }
  // the latent: x / sqrt(mean(x^2) + eps) * w
  float ss = 0.f;
#pragma unroll
  for (int u = 0; u < ROW_HELD; ++u) ss = fmaf(x[u], x[u], ss);
  for (int i = lane + 32 * ROW_HELD; i < rank; i += 32) ss = fmaf(kv[i], kv[i], ss);
  ss = warp_sum(ss);
  const float rstd = 1.0f / sqrtf(ss / (float)rank + eps);
  auto put = [&](int i, float v) {
    const T o = from_f32<T>(v * rstd * norm_w[i]);
    if (lat0) lat0[i] = o;
    if (lat1) lat1[i] = o;
  };
#pragma unroll
  for (int u = 0; u < ROW_HELD; ++u)
    if (lane + 32 * u < rank) put(lane + 32 * u, x[u]);
  for (int i = lane + 32 * ROW_HELD; i < rank; i += 32) put(i, kv[i]);
  if (g_in != nullptr)
    for (int h = lane; h < H; h += 32) gate[(size_t)t * H + h] = 1.0f / (1.0f + expf(-g_in[(size_t)t * ldg + h]));
}

// latents, rotated, cu, rows: see Copy; with cu, q_nope and q_lat are one buffer of rows [H, dim + rd].
GB_EXPORT int gb_latent_prepare(const float* q_in, long long ldq, const float* kv_in, long long ldkv, const float* g_in,
                                long long ldg, const float* norm_w, float eps, const float* inv_freq, int rot,
                                float q_scale, void* q_nope, long long ldqn, void* q_lat, long long ldql, float* gate,
                                void* cache, int dtype, const int* page_table, int table_width, int page_size,
                                const int* tok_pos, const int* tok_seq, const int* seq_slot, int ntok, int H, int dim,
                                int rd, int rank, void* latents, long long ldl, void* rotated, long long ldr, const int* cu, long long rows,
                                int half_layout, float rot_mag, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  if (H <= 0 || dim < 0 || rd < 0 || rank <= 0 || rot < 0 || rot > rd || (rot & 1) || rot > 8192) return GB_ERR_SIZE;
  if (rot > 0 && inv_freq == nullptr) return GB_ERR_ARG;
  if (cu != nullptr && (latents == nullptr || rows < ntok)) return GB_ERR_ARG;
  const int qd = dim + rd, head_end = (cu ? dim : rank) + rd;
  const int elem = dtype == GB_F32 ? 16 : 8;          // bytes of four results
  const int wide = (rot == 0 || !half_layout) && dim % 4 == 0 && rd % 4 == 0 && rank % 4 == 0 && ldq % 4 == 0 && ldqn % 4 == 0 &&
                   ldql % 4 == 0 && head_end % 4 == 0 && ((uintptr_t)q_in & 15) == 0 &&
                   ((uintptr_t)q_nope % elem) == 0 && ((uintptr_t)q_lat % elem) == 0 && qd > 0;
  const int units = H * (wide ? qd / 4 : dim + rd / 2 + (rd & 1));          // of a token
  const int row_blocks = (ntok + PREPARE_THREADS / 32 - 1) / (PREPARE_THREADS / 32);
  // Two quads a thread where there are more than a chip of threads.  us, one / two, by units of 148 threads: 996 (8 heads, 768 tokens)
  // 5.9 / 5.6, 1,328 (16 heads, 256) 6.0 / 6.1, 1,328 (32 heads, 128) 5.9 / 5.9, 1,992 6.1 / 6.1 and 6.8 / 6.3, 2,656 6.6 / 6.6 and 6.3 / 6.4,
  // 3,985 7.9 / 6.9, 10,627 (16 heads, 2,048) 17.6 / 14.7.
  const int quads = (long long)ntok * units > 2048LL * 148 ? PREPARE_QUADS : 1;
  const int token_blocks = (units + PREPARE_THREADS * quads - 1) / (PREPARE_THREADS * quads);
  const long long blocks = row_blocks + (long long)ntok * token_blocks;
  if (blocks > 0x7fffffffLL) return GB_ERR_SIZE;
#define LAUNCH_QUADS(T, QUADS)                                                                                        \
  gb_launch(latent_prepare_kernel<T, QUADS>, dim3((unsigned)blocks), dim3(PREPARE_THREADS), 0, stream, q_in, ldq, kv_in, ldkv, \
            g_in, ldg, norm_w, eps, inv_freq, rot, q_scale, (T*)q_nope, ldqn, (T*)q_lat, ldql, gate, (T*)cache, page_table, \
            table_width, page_size, tok_pos, tok_seq, seq_slot, ntok, H, dim, rd, rank, Copy<T>{(T*)latents, (T*)rotated, ldl, ldr, cu, rows}, \
            half_layout, rot_mag, wide, row_blocks, token_blocks)
#define LAUNCH(T)                        \
  do {                                              \
    if (quads > 1) LAUNCH_QUADS(T, PREPARE_QUADS);  \
    else LAUNCH_QUADS(T, 1);                        \
  } while (0)
  if (dtype == GB_F32) LAUNCH(float);
  else if (dtype == GB_BF16) LAUNCH(bf16);
  else return GB_ERR_DTYPE;
#undef LAUNCH
#undef LAUNCH_QUADS
  return gb_launch_status();
}

// ---------------------------------------------------------------------------------------------
// y[t, h, n] = scale[t, h] * sum_k x[t, h, k] * w[h, n, k]: one product per head, FFMA with
// float32 accumulation in ascending k (a row's result does not depend on the other rows).  With `gate`
// (rows ldg apart, head h's numbers from h * N) the result is multiplied by sigmoid(gate[t, h * N + n]).
constexpr int HB = 64, HK = 16;

template <typename TI, typename TO>
__global__ void __launch_bounds__(256) heads_gemm_kernel(const TI* __restrict__ x, long long ldx_t, long long ldx_h,
                                                         const TI* __restrict__ w, TO* __restrict__ y, long long ldy_t,
                                                         long long ldy_h, const float* __restrict__ scale, int M, int H,
                                                         int N, int K, const float* __restrict__ gate, long long ldg) {
  pdl_release_next();
  pdl_wait_prior();
  __shared__ float xs[HK][HB + 4];
  __shared__ float ws[HK][HB + 4];
  const int tid = threadIdx.x, h = blockIdx.z;
  const int m0 = blockIdx.y * HB, n0 = blockIdx.x * HB;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  const TI* xh = x + (size_t)h * ldx_h;
  const TI* wh = w + (size_t)h * N * K;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += HK) {
    for (int e = tid; e < HB * HK; e += 256) {
      const int r = e / HK, c = e % HK;
      const int gm = m0 + r, gk = k0 + c, gn = n0 + r;
      xs[c][r] = (gm < M && gk < K) ? to_f32(xh[(size_t)gm * ldx_t + gk]) : 0.f;
      ws[c][r] = (gn < N && gk < K) ? to_f32(wh[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < HK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[kk][tm + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[kk][tn + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + tm + i;
    if (gm >= M) continue;
    const float s = scale ? scale[(size_t)gm * H + h] : 1.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tn + j;
      if (gn >= N) continue;
      const float open = gate ? 1.0f / (1.0f + expf(-gate[(size_t)gm * ldg + (size_t)h * N + gn])) : 1.f;
      y[(size_t)gm * ldy_t + (size_t)h * ldy_h + gn] = from_f32<TO>(acc[i][j] * s * open);
    }
  }
}

// The same in bfloat16 for a few rows (a step of single tokens): mma.sync on operands straight from memory.  A CTA is one
// head and 16 NSP columns; its eight warps deal the inner dimension, in blocks of 32, to KSP of them (a lane's 16 bytes are
// its share of a block in both operands), and their sums meet in shared memory in warp order.  The first blocks of the
// matrices are asked for before the kernel before this one has ended.  Bound by one round trip for the matrices and one for
// the rows: 16 tokens, 16 heads, 128 -> 512 and 512 -> 128: 8.3 us each on the grouped product's tiles of 128 rows, 2.8 and 2.6 so.
template <int KSP>
__global__ void __launch_bounds__(256) heads_few_kernel(const bf16* __restrict__ x, long long ldx_t, long long ldx_h,
                                                        const bf16* __restrict__ w, bf16* __restrict__ y, long long ldy_t, long long ldy_h,
                                                        const float* __restrict__ scale, int M, int H, int N, int K,
                                                        const float* __restrict__ gate, long long ldg) {
  constexpr int NSP = 8 / KSP, AHEAD = 2;
  __shared__ float sums[8][16][17];
  pdl_release_next();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int h = blockIdx.y, n0 = (blockIdx.x * NSP + warp / KSP) * 16, kw = warp % KSP, blocks = K / 32;
  const bf16* wrow = w + ((size_t)h * N + n0 + g) * K + 8 * c;
  const bool in0 = n0 + g < N, in1 = n0 + 8 + g < N;
  auto weights = [&](int kb, uint4 (&v)[2]) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    v[0] = in0 && kb < blocks ? *(const uint4*)(wrow + kb * 32) : zero;
    v[1] = in1 && kb < blocks ? *(const uint4*)(wrow + (size_t)8 * K + kb * 32) : zero;
  };
  uint4 first[AHEAD][2];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) weights(kw + i * KSP, first[i]);
  pdl_wait_prior();
  for (int m0 = 0; m0 < M; m0 += 16) {
    const bool a0 = m0 + g < M, a1 = m0 + g + 8 < M;
    const bf16* r0 = x + (size_t)(a0 ? m0 + g : 0) * ldx_t + (size_t)h * ldx_h + 8 * c;
    const bf16* r1 = x + (size_t)(a1 ? m0 + g + 8 : 0) * ldx_t + (size_t)h * ldx_h + 8 * c;
    float acc[2][4] = {};
    auto block = [&](int kb, const uint4 (&v)[2]) {
      const uint4 p = *(const uint4*)(r0 + kb * 32), q = *(const uint4*)(r1 + kb * 32);     // rows beyond M are not stored
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        mma16816(acc[j], p.x, q.x, p.y, q.y, v[j].x, v[j].y);
        mma16816(acc[j], p.z, q.z, p.w, q.w, v[j].z, v[j].w);
      }
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (kw + i * KSP < blocks) block(kw + i * KSP, first[i]);
    for (int kb = kw + AHEAD * KSP; kb < blocks; kb += KSP) {
      uint4 v[2];
      weights(kb, v);
      block(kb, v);
    }
    __syncthreads();                    // the rows before have left
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) sums[warp][g + 8 * (e >> 1)][8 * j + 2 * c + (e & 1)] = acc[j][e];
    __syncthreads();
    for (int e = tid; e < 256 * NSP; e += 256) {
      const int part = e >> 8, r = (e >> 4) & 15, col = e & 15, m = m0 + r, n = (blockIdx.x * NSP + part) * 16 + col;
      if (m >= M || n >= N) continue;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < KSP; ++k) v += sums[part * KSP + k][r][col];
      if (scale) v *= scale[(size_t)m * H + h];
      if (gate) v *= 1.0f / (1.0f + expf(-gate[(size_t)m * ldg + (size_t)h * N + n]));
      y[(size_t)m * ldy_t + (size_t)h * ldy_h + n] = __float2bfloat16_rn(v);
    }
  }
}

// x: [M, H, K], w: [H, N, K], y: [M, H, N] bfloat16; K a multiple of 32, x and w rows at 16-byte boundaries.
GB_EXPORT int gb_heads_few(const void* x, long long ldx_t, long long ldx_h, const void* w, void* y, long long ldy_t, long long ldy_h,
                           const float* scale, int M, int H, int N, int K, const float* gate, long long ldg, cudaStream_t stream) {
  if (M <= 0 || H <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 32 || H > 65535 || ldx_t % 8 || ldx_h % 8 || (((uintptr_t)x | (uintptr_t)w) & 15)) return GB_ERR_SIZE;
#define HEADS_FEW(KSP)                                                                                                \
  gb_launch(heads_few_kernel<KSP>, dim3((N + 16 * (8 / KSP) - 1) / (16 * (8 / KSP)), H), dim3(256), 0, stream, (const bf16*)x, ldx_t, \
            ldx_h, (const bf16*)w, (bf16*)y, ldy_t, ldy_h, scale, M, H, N, K, gate, ldg)
  if (K >= 256) HEADS_FEW(8);
  else if (K >= 128) HEADS_FEW(4);
  else HEADS_FEW(2);
#undef HEADS_FEW
  return gb_launch_status();
}

GB_EXPORT int gb_heads_gemm(const void* x, long long ldx_t, long long ldx_h, const void* w, void* y, long long ldy_t,
                            long long ldy_h, const float* scale, int dtype, int M, int H, int N, int K,
                            const float* gate, long long ldg, cudaStream_t stream) {
  if (M <= 0 || H <= 0 || N <= 0) return 0;
  if (K <= 0 || H > 65535) return GB_ERR_SIZE;
  dim3 grid((N + HB - 1) / HB, (M + HB - 1) / HB, H);
  if (dtype == GB_F32)
    gb_launch(heads_gemm_kernel<float, float>, grid, dim3(256), 0, stream, (const float*)x, ldx_t, ldx_h, (const float*)w,
              (float*)y, ldy_t, ldy_h, scale, M, H, N, K, gate, ldg);
  else if (dtype == GB_BF16)
    gb_launch(heads_gemm_kernel<bf16, bf16>, grid, dim3(256), 0, stream, (const bf16*)x, ldx_t, ldx_h, (const bf16*)w,
              (bf16*)y, ldy_t, ldy_h, scale, M, H, N, K, gate, ldg);
  else
    return GB_ERR_DTYPE;
  return gb_launch_status();
}

// ---------------------------------------------------------------------------------------------
// Attention over the cached rows, one block per (token, head); online softmax over chunks of
// 128 keys from the window's first key (key 0 without a window).
constexpr int CHUNK = 128;
constexpr int MAX_U = 8;      // rank <= MAX_U * CHUNK

template <typename T>
__global__ void __launch_bounds__(CHUNK) latent_attention_ref_kernel(
    const T* __restrict__ qa, long long ldq, T* __restrict__ out, long long ldo, const T* __restrict__ cache,
    const int* __restrict__ page_table, int table_width, int page_size, const int* __restrict__ tok_pos,
    const int* __restrict__ tok_seq, const int* __restrict__ seq_slot, int rank, int rd, int window) {
  extern __shared__ float smem[];
  pdl_release_next();
  pdl_wait_prior();
  const int kd = rank + rd;
  float* qs = smem;                    // [kd]
  float* p = qs + kd;                  // [CHUNK]
  float* scratch = p + CHUNK;          // [34]
  size_t* rows = (size_t*)(((uintptr_t)(scratch + 34) + 7) & ~(uintptr_t)7);   // [CHUNK]
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int pos = tok_pos[t];
  const int slot = seq_slot[tok_seq[t]];
  const int hi = pos + 1;
  const int lo = window > 0 ? max(0, hi - window) : 0;
  const T* qrow = qa + (size_t)t * ldq + (size_t)h * kd;
  for (int i = tid; i < kd; i += CHUNK) qs[i] = to_f32(qrow[i]);
  __syncthreads();
  float m = -INFINITY, l = 0.f, acc[MAX_U];
#pragma unroll
  for (int u = 0; u < MAX_U; ++u) acc[u] = 0.f;
  for (int c0 = lo; c0 < hi; c0 += CHUNK) {
    const int j = c0 + tid;
    float s = -INFINITY;
    if (j < hi) {
      const int page = page_table[(size_t)slot * table_width + (j / page_size) % table_width];
      const size_t r = ((size_t)page * page_size + j % page_size) * (size_t)kd;
      rows[tid] = r;
      const T* kr = cache + r;
      float d = 0.f;
      for (int i = 0; i < kd; ++i) d = fmaf(qs[i], to_f32(kr[i]), d);
      s = d;
    }
    const float m_new = fmaxf(m, block_max(s, scratch));
    const float pj = j < hi ? expf(s - m_new) : 0.f;
    p[tid] = pj;
    const float csum = block_sum(pj, scratch);   // also orders the writes of p and rows
    const float alpha = expf(m - m_new);
    l = l * alpha + csum;
    const int n = min(CHUNK, hi - c0);
#pragma unroll
    for (int u = 0; u < MAX_U; ++u) {
      const int d = tid + u * CHUNK;
      if (d < rank) {
        float a = acc[u] * alpha;
        for (int jj = 0; jj < n; ++jj) a = fmaf(p[jj], to_f32(cache[rows[jj] + d]), a);
        acc[u] = a;
      }
    }
    m = m_new;
    __syncthreads();
  }
  T* orow = out + (size_t)t * ldo + (size_t)h * rank;
#pragma unroll
  for (int u = 0; u < MAX_U; ++u) {
    const int d = tid + u * CHUNK;
    if (d < rank) orow[d] = from_f32<T>(acc[u] / l);
  }
}

// qa: [ntok, H, rank + rd] rows ldq apart; out: [ntok, H, rank] rows ldo apart;
// cache: [pages, page_size, rank + rd].
GB_EXPORT int gb_latent_attention_ref(const void* qa, long long ldq, void* out, long long ldo, int dtype, const void* cache,
                                      const int* page_table, int table_width, int page_size, const int* tok_pos,
                                      const int* tok_seq, const int* seq_slot, int ntok, int H, int rank, int rd,
                                      int window, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  if (rank <= 0 || rank > MAX_U * CHUNK || rd < 0 || H <= 0 || H > 65535) return GB_ERR_SIZE;
  const size_t smem = (size_t)(rank + rd + CHUNK + 34) * sizeof(float) + CHUNK * sizeof(size_t) + 8;
  if (smem > 48 * 1024) return GB_ERR_SIZE;
  dim3 grid(ntok, H);
#define LAUNCH(T)                                                                                                      \
  gb_launch(latent_attention_ref_kernel<T>, grid, dim3(CHUNK), smem, stream, (const T*)qa, ldq, (T*)out, ldo,          \
            (const T*)cache, page_table, table_width, page_size, tok_pos, tok_seq, seq_slot, rank, rd, window)
  if (dtype == GB_F32) LAUNCH(float);
  else if (dtype == GB_BF16) LAUNCH(bf16);
  else return GB_ERR_DTYPE;
#undef LAUNCH
  return gb_launch_status();
}

// ---------------------------------------------------------------------------------------------
// Stand-alone rotation of interleaved pairs, in place: x [ntok, heads, hd], the first `rot` dims
// of every head.
template <typename T>
__global__ void rope_pairs_kernel(T* __restrict__ x, long long ldx, const int* __restrict__ tok_pos,
                                  const float* __restrict__ inv_freq, int heads, int hd, int rot, float mag) {
  pdl_release_next();
  pdl_wait_prior();
  const int t = blockIdx.x;
  const float fpos = (float)tok_pos[t];
  const int half = rot / 2;
  for (int e = threadIdx.x; e < heads * half; e += blockDim.x) {
    const int h = e / half, i = e % half;
    T* v = x + (size_t)t * ldx + (size_t)h * hd + 2 * i;
    float a, b;
    rotate_pair(to_f32(v[0]), to_f32(v[1]), cos_sin(fpos * inv_freq[i], mag), a, b);
    v[0] = from_f32<T>(a);
    v[1] = from_f32<T>(b);
  }
}

GB_EXPORT int gb_rope_pairs(void* x, long long ldx, int dtype, const int* tok_pos, const float* inv_freq, int ntok,
                            int heads, int hd, int rot, float mag, cudaStream_t stream) {
  if (ntok <= 0 || rot <= 0) return 0;
  if (rot > hd || (rot & 1)) return GB_ERR_SIZE;
  if (dtype == GB_F32)
    gb_launch(rope_pairs_kernel<float>, dim3(ntok), dim3(128), 0, stream, (float*)x, ldx, tok_pos, inv_freq, heads, hd, rot, mag);
  else if (dtype == GB_BF16)
    gb_launch(rope_pairs_kernel<bf16>, dim3(ntok), dim3(128), 0, stream, (bf16*)x, ldx, tok_pos, inv_freq, heads, hd, rot, mag);
  else
    return GB_ERR_DTYPE;
  return gb_launch_status();
}
