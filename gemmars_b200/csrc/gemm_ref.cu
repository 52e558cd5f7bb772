// Plain CUDA-core matrix product  y[t, o] = sum_i W[o, i] * x[t, i] (+ bias[o])
// (src/kernels.rs:54-57), for float32 and for bfloat16 inputs, accumulating in float32 with
// FFMA only: no tensor-core or reduced-precision matrix mode is compiled into this unit.
//
// It is the whole matrix path of the float32 engine (gemm_f32_kernel) and the plain reference of the
// bfloat16 tensor-core kernels (gemm_ref_kernel).  The order in which an output element is summed depends
// on K alone, so a row's result does not depend on how many rows the call has (the property the
// reference tests as batch invariance, src/qwen_mtp.rs:748-776), nor on the tile that the launcher picks.
#include <type_traits>

#include "common.cuh"

enum { OUT_STORE = 0, OUT_ACCUMULATE_F32 = 1 };
enum { ACT_NONE = 0, ACT_GELU = 1, ACT_RELU2 = 2 };   // the exact (erf) GELU; the square of relu

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TI, typename TO, int MODE>
__global__ void __launch_bounds__(256) gemm_ref_kernel(const TI* __restrict__ x, const TI* __restrict__ w,
                                                       const float* __restrict__ bias, TO* __restrict__ y, int M,
                                                       int N, int K, long long ldx, long long ldy, int act,
                                                       const float* __restrict__ col_scale) {
  pdl_release_next();
  pdl_wait_prior();
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int e = tid; e < BM * BK; e += 256) {
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gk = k0 + c;
      xs[c][r] = (gm < M && gk < K) ? to_f32(x[(size_t)gm * ldx + gk]) : 0.f;
      const int gn = n0 + r;
      ws[c][r] = (gn < N && gk < K) ? to_f32(w[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
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
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tn + j;
      if (gn >= N) continue;
      float v = acc[i][j] + (bias ? bias[gn] : 0.f);
      if (act == ACT_GELU) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
      else if (act == ACT_RELU2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
      if (col_scale) v *= col_scale[gn];
      TO* dst = y + (size_t)gm * ldy + gn;
      if (MODE == OUT_ACCUMULATE_F32)
        *dst = from_f32<TO>(to_f32(*dst) + v);
      else
        *dst = from_f32<TO>(v);
    }
  }
}

// ------------------------------------------------------------------ float32
// The float32 product: four warps, each a part of the inner dimension of one tile of 4 TM rows of x by 8 TN rows of W, TM x TN
// results a lane.  Every result is the sum of PARTS parts, added in their order; a part's length depends on the inner dimension
// alone, and in a part the even and the odd inner elements have a sum each (two multiply-adds in one instruction).  So the bits
// depend neither on the tile nor on the number of rows, and the error is smaller than one long sum's (distance from 64 bits of
// 1,024 / 4,096 inner elements: 2.1e-7 / 4.1e-7, one sum 5.7e-7 / 1.2e-6).
// A warp brings its own rows, KB of K side by side and a row 4 floats longer so that the 16-byte reads of eight neighbouring
// rows touch all banks once, by asynchronous copies STAGES - 1 blocks ahead, and waits for no other warp until the parts are
// added: no barrier in the main loop, and four warps on a tile where one thread for every result's whole sum would leave an SM
// two (301 rows by 1,024 features are 2,082 results an SM).  What bounds it: the 16-byte reads, TM + TN for 4 TM TN
// multiply-adds (2,048 x 4,096 x 4,096 at 45.9 of some 70 TFLOP/s; 43.7 with KB of 16, 40 with a multiply-add an instruction), the last round of tiles, and the stream of W for a few
// rows.  The first blocks of W are asked for before the kernel before this one has ended.
constexpr int PARTS = 4;
__host__ __device__ constexpr int part_length(int K) { return ((K + PARTS - 1) / PARTS + 31) / 32 * 32; }

__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float even_and_odd(uint64_t v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

template <int TM, int TN, int KB, int STAGES>
struct F32Tile {
  static constexpr int BM = 4 * TM, BN = 8 * TN, LD = KB + 4;
  static constexpr int STAGE_FLOATS = (BM + BN) * LD, WARP_FLOATS = STAGES * STAGE_FLOATS;
  static_assert(WARP_FLOATS >= BM * BN, "a part's results go where its stages were");
  static_assert(TM * TN % PARTS == 0 && KB == 32, "whole shares; a part is a multiple of KB");
  static constexpr size_t SMEM = (size_t)PARTS * WARP_FLOATS * sizeof(float);
};

// VEC: rows of both operands start at 16-byte boundaries and K is a multiple of 4.  The grid's CTAs run over the rows first.
template <int TM, int TN, int KB, int STAGES, bool VEC, int MODE>
__global__ void __launch_bounds__(32 * PARTS)
    gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ y,
                    int M, int N, int K, long long ldx, long long ldy, int act, const float* __restrict__ col_scale, int tiles_m) {
  using T = F32Tile<TM, TN, KB, STAGES>;
  constexpr int BM = T::BM, BN = T::BN, LD = T::LD, CH = KB / 4, STEP = 32 / CH;      // CH 16-byte pieces of a row, STEP rows a pass
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x % tiles_m * BM, n0 = blockIdx.x / tiles_m * BN;
  const int ty = lane >> 3, tx = lane & 7;
  const int length = part_length(K), k0 = min(K, warp * length), k1 = min(K, k0 + length);
  const int blocks = (k1 - k0 + KB - 1) / KB;
  float* mine = smem + warp * T::WARP_FLOATS;
  const int r0 = lane / CH, c = lane % CH * 4;
  auto bring = [&](int block, const float* base, long long ld, int row0, int rows_have, float* dst, auto rows) {
    constexpr int ROWS = decltype(rows)::value;
    const int k = k0 + block * KB + c;
#pragma unroll
    for (int i = 0; i < (ROWS + STEP - 1) / STEP; ++i) {
      const int r = r0 + STEP * i;
      if (ROWS % STEP && r >= ROWS) break;
      float* d = dst + r * LD + c;
      const bool row_in = row0 + r < rows_have;
      const float* src = base + (size_t)(row_in ? row0 + r : 0) * ld;
      if (VEC) {
        const bool in = row_in && k < k1;
        copy16(d, in ? src + k : base, in ? 16 : 0);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = row_in && k + j < k1;
          copy4(d + j, in ? src + k + j : base, in ? 4 : 0);
        }
      }
    }
  };
  using RowsX = std::integral_constant<int, BM>;
  using RowsW = std::integral_constant<int, BN>;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < blocks) bring(s, w, K, n0, N, mine + s * T::STAGE_FLOATS + BM * LD, RowsW());
  pdl_wait_prior();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < blocks) bring(s, x, ldx, m0, M, mine + s * T::STAGE_FLOATS, RowsX());
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint64_t acc[TM][TN] = {};
  int at = 0, to = STAGES - 1;
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncwarp();                          // block b is there for all lanes, and block b - 1 has been read by all
    if (b + STAGES - 1 < blocks) {
      bring(b + STAGES - 1, x, ldx, m0, M, mine + to * T::STAGE_FLOATS, RowsX());
      bring(b + STAGES - 1, w, K, n0, N, mine + to * T::STAGE_FLOATS + BM * LD, RowsW());
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float *xs = mine + at * T::STAGE_FLOATS + ty * LD, *ws = mine + at * T::STAGE_FLOATS + (BM + tx) * LD;
    at = at + 1 == STAGES ? 0 : at + 1;
    to = to + 1 == STAGES ? 0 : to + 1;
#pragma unroll
    for (int kk = 0; kk < KB; kk += 4) {
      ulonglong2 v[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) v[j] = *(const ulonglong2*)(ws + j * 8 * LD + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *(const ulonglong2*)(xs + i * 4 * LD + kk);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.x, v[j].x);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.y, v[j].y);
      }
    }
  }
  pdl_release_next();
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) mine[(i * TN + j) * 32 + lane] = even_and_odd(acc[i][j]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < TM * TN / PARTS; ++q) {      // a warp finishes a quarter of the tile's results
    const int e = warp * (TM * TN / PARTS) + q, gm = m0 + 4 * (e / TN) + ty, gn = n0 + 8 * (e % TN) + tx;
    const float* p = smem + e * 32 + lane;
    float v = p[0];
#pragma unroll
    for (int part = 1; part < PARTS; ++part) v += p[part * T::WARP_FLOATS];
    if (gm >= M || gn >= N) continue;
    if (bias) v += bias[gn];
    if (act == ACT_GELU) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
    else if (act == ACT_RELU2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
    if (col_scale) v *= col_scale[gn];
    float* dst = y + (size_t)gm * ldy + gn;
    *dst = MODE == OUT_ACCUMULATE_F32 ? *dst + v : v;
  }
}

// The same sums for short inner dimensions and many results, where the four warps' parts are a block or two and their meeting
// most of the time: a CTA of 128 threads works 64 rows by 64 with whole sums, 4 x 8 results a thread, and adds up a part's even
// and odd sums when the part ends: the same bits.  What bounds it: the results' way to memory and, from 64 inner elements on, the
// 16-byte reads.  See short_pays.
struct F32Short {
  static constexpr int BM = 64, BN = 64, TM = 4, TN = 8, KB = 16, STAGES = 4, LD = KB + 4, MAX_K = 192;
  static constexpr int STAGE_FLOATS = (BM + BN) * LD;
};
static_assert(F32Short::STAGES * F32Short::STAGE_FLOATS * sizeof(float) <= 48 * 1024, "static shared memory");

template <bool VEC, int MODE>
__global__ void __launch_bounds__(128)
    gemm_f32_short_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ y,
                          int M, int N, int K, long long ldx, long long ldy, int act, const float* __restrict__ col_scale, int tiles_m) {
  using T = F32Short;
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, KB = T::KB, STAGES = T::STAGES, LD = T::LD, CH = KB / 4;
  __shared__ __align__(16) float smem[STAGES * T::STAGE_FLOATS];
  pdl_release_next();
  const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
  const int m0 = blockIdx.x % tiles_m * BM, n0 = blockIdx.x / tiles_m * BN;
  const int blocks = (K + KB - 1) / KB, length = part_length(K);
  auto bring = [&](int block, const float* base, long long ld, int row0, int rows_have, float* dst) {
    static_assert(BM == BN, "as many rows of both");
#pragma unroll
    for (int i = 0; i < BM * CH / 128; ++i) {
      const int r = (tid + 128 * i) / CH, c = tid % CH * 4, k = block * KB + c;
      float* d = dst + r * LD + c;
      const bool row_in = row0 + r < rows_have;
      const float* src = base + (size_t)(row_in ? row0 + r : 0) * ld;
      if (VEC) {
        const bool in = row_in && k < K;
        copy16(d, in ? src + k : base, in ? 16 : 0);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = row_in && k + j < K;
          copy4(d + j, in ? src + k + j : base, in ? 4 : 0);
        }
      }
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < blocks) bring(s, w, K, n0, N, smem + s * T::STAGE_FLOATS + BM * LD);
  pdl_wait_prior();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < blocks) bring(s, x, ldx, m0, M, smem + s * T::STAGE_FLOATS);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint64_t acc[TM][TN] = {};
  float sum[TM][TN];
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // block b is there for all, and block b - 1 has been read by all
    if (b + STAGES - 1 < blocks) {
      float* to = smem + (b + STAGES - 1) % STAGES * T::STAGE_FLOATS;
      bring(b + STAGES - 1, x, ldx, m0, M, to);
      bring(b + STAGES - 1, w, K, n0, N, to + BM * LD);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float *xs = smem + b % STAGES * T::STAGE_FLOATS + ty * LD, *ws = smem + b % STAGES * T::STAGE_FLOATS + (BM + tx) * LD;
#pragma unroll
    for (int kk = 0; kk < KB; kk += 4) {
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *(const ulonglong2*)(xs + i * 16 * LD + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 v = *(const ulonglong2*)(ws + j * 8 * LD + kk);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].x, v.x);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].y, v.y);
      }
    }
    const int end = (b + 1) * KB;
    if (end % length == 0 || b + 1 == blocks) {          // a part ends
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float part = even_and_odd(acc[i][j]);
          sum[i][j] = end <= length ? part : sum[i][j] + part;
          acc[i][j] = 0;
        }
    }
  }
  const bool fewer = (PARTS - 1) * length >= K;           // parts without an element, which are added as zeros
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + i * 16 + ty;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + j * 8 + tx;
      if (gn >= N) continue;
      float v = sum[i][j];
      if (fewer) v += 0.f;
      if (bias) v += bias[gn];
      if (act == ACT_GELU) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
      else if (act == ACT_RELU2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
      if (col_scale) v *= col_scale[gn];
      float* dst = y + (size_t)gm * ldy + gn;
      *dst = MODE == OUT_ACCUMULATE_F32 ? *dst + v : v;
    }
  }
}

struct F32Call {
  const float *x, *w, *bias;
  float* y;
  int M, N, K;
  long long ldx, ldy;
  int act;
  const float* col_scale;
};

static bool f32_vec(const F32Call& c) {
  return c.K % 4 == 0 && c.ldx % 4 == 0 && (((uintptr_t)c.x | (uintptr_t)c.w) & 15) == 0;
}

template <int TM, int TN, int KB, int STAGES>
static int launch_f32_tile(const F32Call& c, int mode, cudaStream_t stream) {
  using T = F32Tile<TM, TN, KB, STAGES>;
  const bool vec = f32_vec(c);
  const int tiles_m = (c.M + T::BM - 1) / T::BM;
  const long long tiles = (long long)tiles_m * ((c.N + T::BN - 1) / T::BN);
  if (tiles > 0x7fffffffLL) return GB_ERR_SIZE;
#define LAUNCH_F32(VEC, MODE)                                                                                          \
  do {                                                                                                                 \
    auto kernel = gemm_f32_kernel<TM, TN, KB, STAGES, VEC, MODE>;                                                      \
    if (T::SMEM > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);  \
    gb_launch(kernel, dim3((unsigned)tiles), 32 * PARTS, T::SMEM, stream, c.x, c.w, c.bias, c.y, c.M, c.N, c.K, c.ldx, \
              c.ldy, c.act, c.col_scale, tiles_m);                                                                     \
  } while (0)
  if (mode == OUT_ACCUMULATE_F32) {
    if (vec) LAUNCH_F32(true, OUT_ACCUMULATE_F32);
    else LAUNCH_F32(false, OUT_ACCUMULATE_F32);
  } else {
    if (vec) LAUNCH_F32(true, OUT_STORE);
    else LAUNCH_F32(false, OUT_STORE);
  }
#undef LAUNCH_F32
  return gb_launch_status();
}

static int launch_f32_short(const F32Call& c, int mode, cudaStream_t stream) {
  const int tiles_m = (c.M + F32Short::BM - 1) / F32Short::BM;
  const long long tiles = (long long)tiles_m * ((c.N + F32Short::BN - 1) / F32Short::BN);
  if (tiles > 0x7fffffffLL) return GB_ERR_SIZE;
#define LAUNCH_SHORT(VEC, MODE)                                                                                                \
  gb_launch(gemm_f32_short_kernel<VEC, MODE>, dim3((unsigned)tiles), 128, 0, stream, c.x, c.w, c.bias, c.y, c.M, c.N, c.K, c.ldx, \
            c.ldy, c.act, c.col_scale, tiles_m)
  if (mode == OUT_ACCUMULATE_F32) {
    if (f32_vec(c)) LAUNCH_SHORT(true, OUT_ACCUMULATE_F32);
    else LAUNCH_SHORT(false, OUT_ACCUMULATE_F32);
  } else {
    if (f32_vec(c)) LAUNCH_SHORT(true, OUT_STORE);
    else LAUNCH_SHORT(false, OUT_STORE);
  }
#undef LAUNCH_SHORT
  return gb_launch_status();
}

// The tiles, small to large, and what four k of a tile cost on an SM in cycles, as measured on a B200 over M of
// 1 to 2,048 rows and products of 1,024 x 2,048 to 151,936 x 1,024: `alone` when the SM has one CTA (a chain of
// shared-memory reads and multiply-adds: it bounds products with few tiles), `shared` for every CTA more than the
// chain hides (the shared-memory reads; W's stream for the smallest two).  The launcher takes the tile with the least of
// max(alone, shared x rounds), a round being a CTA on each of 148 SMs.  Tiles of 4 or 8 rows of x with one thread
// for every result's whole sum took, up to 64 x 64 for prompts (us, those kernels / these): 1 x 4,096 x 4,096: 47.1 / 19.5;
// 16 x 1,024 x 2,048: 24.0 / 10.6; 301 x 6,144 x 1,024: 160 / 101; 301 x 1,024 x 3,072: 149 / 61;
// 2,048 x 4,096 x 4,096: 1,810 / 1,496; 3 x 151,936 x 1,024 (W's stream): 110 / 111.  The same bits whatever the tile.
struct F32Cost {
  int bm, bn;
  float alone, shared;
};
static const F32Cost F32_TILES[] = {{4, 32, 36.6f, 24.5f}, {8, 32, 38.f, 26.5f},  {16, 32, 52.f, 28.3f},
                                    {32, 32, 65.f, 53.f},  {40, 32, 85.f, 66.6f}, {32, 64, 120.f, 100.f}};

static int pick_f32_tile(int M, int N) {
  int best = 0;
  float least = 0.f;
  for (int i = 0; i < (int)(sizeof(F32_TILES) / sizeof(F32_TILES[0])); ++i) {
    const F32Cost& t = F32_TILES[i];
    const long long tiles = (long long)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn);
    const float cost = fmaxf(t.alone, t.shared * (float)((tiles + 147) / 148));
    if (i == 0 || cost < least) least = cost, best = i;
  }
  return best;
}

static int launch_f32(int tile, const F32Call& c, int mode, cudaStream_t stream) {
  switch (tile) {
    case 0: return launch_f32_tile<1, 4, 32, 3>(c, mode, stream);
    case 1: return launch_f32_tile<2, 4, 32, 3>(c, mode, stream);
    case 2: return launch_f32_tile<4, 4, 32, 2>(c, mode, stream);
    case 3: return launch_f32_tile<8, 4, 32, 2>(c, mode, stream);
    case 4: return launch_f32_tile<10, 4, 32, 2>(c, mode, stream);
    default: return launch_f32_tile<8, 8, 32, 2>(c, mode, stream);
  }
}

// Whether gemm_f32_short_kernel is the faster of the two.  us, four parts / whole sums: 2,048 x 4,096 by K of 16 60.3 / 21.6, 64 71.7 /
// 41.2, 96 73.8 / 55.6, 128 78.5 / 69.3, 160 106 / 84, 192 110 / 98, 224 111 / 113; 2,048 x 1,024 by 16 18.0 / 9.4, 96 21.9 / 18.9, 128
// 22.5 / 23.4, 160 30.9 / 27.3, 192 32.0 / 31.8; 301 x 4,096 by 64 14.0 / 11.5, 96 14.4 / 14.8, 160 20.1 / 21.3; 1,024 x 1,024 by 64 9.8 / 9.0,
// 96 10.8 / 11.7; 301 x 2,048 by 16 6.4 / 5.5, 32 6.5 / 6.3, 64 7.4 / 9.0; 64 x 4,096 by 16 4.3 / 5.0.
static bool short_pays(int M, int N, int K) {
  const long long results = (long long)M * N;
  return K <= F32Short::MAX_K && results >= (K <= 32 ? 1 << 19 : K <= 64 ? 1 << 20 : K <= 96 || K > 128 ? 1 << 21 : 1 << 22);
}
GB_EXPORT int gb_gemm_ref_short(int M, int N, int K) { return short_pays(M, N, K) ? 1 : 0; }

// Which of F32_TILES a float32 product of these sizes takes where four warps share a tile.
GB_EXPORT int gb_gemm_ref_tile(int M, int N) { return pick_f32_tile(M, N); }

// x: [M, K] rows ldx apart; w: [N, K]; y: [M, N] rows ldy apart.
// mode OUT_STORE writes y in out_dtype; OUT_ACCUMULATE_F32 adds into a float32 y.  act: an activation of
// product + bias; col_scale (null: ones): [N], multiplied in after it, before the store or the add.
GB_EXPORT int gb_gemm_ref(const void* x, const void* w, int in_dtype, const float* bias, void* y, int out_dtype,
                          int mode, int M, int N, int K, long long ldx, long long ldy, int act, const float* col_scale,
                          cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return GB_ERR_SIZE;
  if (act < ACT_NONE || act > ACT_RELU2) return GB_ERR_ARG;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (mode == OUT_ACCUMULATE_F32 && out_dtype != GB_F32) return GB_ERR_DTYPE;
#define LAUNCH(TI, TO, MODE) \
  gb_launch(gemm_ref_kernel<TI, TO, MODE>, grid, 256, 0, stream, (const TI*)x, (const TI*)w, bias, (TO*)y, M, N, K, ldx, ldy, \
            act, col_scale)
  if (in_dtype == GB_F32) {
    if (out_dtype != GB_F32) return GB_ERR_DTYPE;
    const F32Call call{(const float*)x, (const float*)w, bias, (float*)y, M, N, K, ldx, ldy, act, col_scale};
    return short_pays(M, N, K) ? launch_f32_short(call, mode, stream) : launch_f32(pick_f32_tile(M, N), call, mode, stream);
  } else if (in_dtype == GB_BF16) {
    if (mode == OUT_ACCUMULATE_F32) LAUNCH(bf16, float, OUT_ACCUMULATE_F32);
    else if (out_dtype == GB_F32) LAUNCH(bf16, float, OUT_STORE);
    else if (out_dtype == GB_BF16) LAUNCH(bf16, bf16, OUT_STORE);
    else return GB_ERR_DTYPE;
  } else {
    return GB_ERR_DTYPE;
  }
#undef LAUNCH
  return gb_launch_status();
}
