// Plain CUDA-core matrix product  y[t, o] = sum_i W[o, i] * x[t, i] (+ bias[o])
// (src/kernels.rs:54-57), for float32 and for bfloat16 inputs, accumulating in float32 with
// FFMA only: no tensor-core or reduced-precision matrix mode is compiled into this unit.
//
// It is the whole matrix path of the float32 engine (gemm_f32_kernel) and the plain reference of the
// bfloat16 tensor-core kernels (gemm_ref_kernel).  Every output element is accumulated by one thread
// over i = 0..K-1 in ascending order, so a row's result does not depend on how many rows the call has
// (the property the reference tests as batch invariance, src/qwen_mtp.rs:748-776), nor on the tile
// that the launcher picks.
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
// The float32 product: a CTA works BM rows of x by BN rows of W, a thread TM x TN results in registers.
// Both operands lie in shared memory as they lie in memory (KB of K side by side, a row 4 floats longer so
// that the 16-byte reads of eight neighbouring rows touch all banks once), brought by asynchronous copies
// STAGES - 1 blocks ahead; a thread reads four k of each of its rows at a time: TM + TN 16-byte reads for
// 4 TM TN multiply-adds.  What bounds it: those reads and the FFMA pipe for prompts, the stream of W for a
// few rows.  The first blocks of W are asked for before the kernel before this one has ended.
__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}

template <int BM, int BN, int TM, int TN, int KB, int STAGES>
struct F32Tile {
  static constexpr int TY = BM / TM, TX = BN / TN, THREADS = TY * TX, LD = KB + 4;
  static constexpr int STAGE_FLOATS = (BM + BN) * LD;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_FLOATS * sizeof(float);
};

// VEC: rows of both operands start at 16-byte boundaries and K is a multiple of 4.
template <int BM, int BN, int TM, int TN, int KB, int STAGES, bool VEC, int MODE>
__global__ void __launch_bounds__(F32Tile<BM, BN, TM, TN, KB, STAGES>::THREADS)
    gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ y,
                    int M, int N, int K, long long ldx, long long ldy, int act, const float* __restrict__ col_scale) {
  using T = F32Tile<BM, BN, TM, TN, KB, STAGES>;
  constexpr int LD = T::LD, NT = T::THREADS, CH = KB / 4;      // 16-byte pieces of a row
  constexpr int WY = T::TY < 8 ? T::TY : 8, WX = 32 / WY;       // a warp's threads: WY rows by WX columns
  static_assert(T::TX % WX == 0 && T::TY % WY == 0, "whole warps");
  extern __shared__ __align__(16) float smem[];
  pdl_release_next();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int ty = warp / (T::TX / WX) * WY + lane % WY, tx = warp % (T::TX / WX) * WX + lane / WY;
  const int blocks = (K + KB - 1) / KB;
  auto bring = [&](int block, const float* base, long long ld, int row0, int rows_have, float* dst, int rows) {
    for (int e = tid; e < rows * CH; e += NT) {
      const int r = e / CH, c = (e % CH) * 4, k = block * KB + c;
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
  auto stage_x = [&](int block) { return smem + (block % STAGES) * T::STAGE_FLOATS; };
  auto stage_w = [&](int block) { return stage_x(block) + BM * LD; };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < blocks) bring(s, w, K, n0, N, stage_w(s), BN);
  pdl_wait_prior();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < blocks) bring(s, x, ldx, m0, M, stage_x(s), BM);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[TM][TN] = {};
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // block b is there for all, and block b - 1 has been read by all
    if (b + STAGES - 1 < blocks) {
      bring(b + STAGES - 1, x, ldx, m0, M, stage_x(b + STAGES - 1), BM);
      bring(b + STAGES - 1, w, K, n0, N, stage_w(b + STAGES - 1), BN);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float *xs = stage_x(b) + ty * LD, *ws = stage_w(b) + tx * LD;
#pragma unroll
    for (int kk = 0; kk < KB; kk += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *(const float4*)(xs + i * T::TY * LD + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 v = *(const float4*)(ws + j * T::TX * LD + kk);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, v.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, v.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, v.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, v.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int gn = n0 + j * T::TX + tx;
    if (gn >= N) continue;
    const float b0 = bias ? bias[gn] : 0.f, c0 = col_scale ? col_scale[gn] : 1.f;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + i * T::TY + ty;
      if (gm >= M) continue;
      float v = acc[i][j] + b0;
      if (act == ACT_GELU) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
      else if (act == ACT_RELU2) v = fmaxf(v, 0.f) * fmaxf(v, 0.f);
      if (col_scale) v *= c0;
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

template <int BM, int BN, int TM, int TN, int KB, int STAGES>
static int launch_f32_tile(const F32Call& c, int mode, cudaStream_t stream) {
  using T = F32Tile<BM, BN, TM, TN, KB, STAGES>;
  const bool vec = c.K % 4 == 0 && c.ldx % 4 == 0 && (((uintptr_t)c.x | (uintptr_t)c.w) & 15) == 0;
  const dim3 grid((c.N + BN - 1) / BN, (c.M + BM - 1) / BM);
#define LAUNCH_F32(VEC, MODE)                                                                                          \
  do {                                                                                                                 \
    auto kernel = gemm_f32_kernel<BM, BN, TM, TN, KB, STAGES, VEC, MODE>;                                              \
    if (T::SMEM > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);  \
    gb_launch(kernel, grid, T::THREADS, T::SMEM, stream, c.x, c.w, c.bias, c.y, c.M, c.N, c.K, c.ldx, c.ldy, c.act,    \
              c.col_scale);                                                                                            \
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

// The tiles, small to large, and what four k of a tile cost on an SM in cycles, as measured on a B200 over M of
// 1 to 2,048 rows and products of 1,024 x 2,048 to 151,936 x 1,024: `alone` when the SM has one CTA (a chain of
// shared-memory reads and multiply-adds: it bounds products with few tiles), `shared` for every CTA more than the
// chain hides (the shared-memory reads: a 16-byte read of a warp takes four cycles whether its lanes read one
// address or 32).  The launcher takes the tile with the least of max(alone, shared x CTAs an SM).
// One tile of 64 x 64 by 256 threads of 4 x 4, loaded without a pipeline, took (us, that kernel / these):
// 301 x 6,144 x 1,024: 188 / 131; 301 x 1,024 x 3,072: 403 / 129; 3 x 151,936 x 1,024: 743 / 117;
// 2,048 x 4,096 x 4,096: 2,435 / 1,757.  The same bits whatever the tile.
struct F32Cost {
  int bm, bn;
  float alone, shared;
};
static const F32Cost F32_TILES[] = {{4, 32, 100.f, 30.f},    {8, 32, 118.f, 33.f},   {16, 64, 174.f, 100.f},
                                    {32, 64, 225.f, 140.f},  {64, 64, 405.f, 244.f}, {128, 128, 874.f, 868.f}};

static int pick_f32_tile(int M, int N) {
  int best = -1;
  float least = 0.f;
  for (int i = 0; i < (int)(sizeof(F32_TILES) / sizeof(F32_TILES[0])); ++i) {
    const F32Cost& t = F32_TILES[i];
    const int rows = (M + t.bm - 1) / t.bm;
    if (rows > 65535) continue;             // what a grid has room for; the largest tile takes the most rows
    const float cost = fmaxf(t.alone, t.shared * (float)rows * (float)((N + t.bn - 1) / t.bn) / 148.f);
    if (best < 0 || cost < least) least = cost, best = i;
  }
  return best;
}

static int launch_f32(int tile, const F32Call& c, int mode, cudaStream_t stream) {
  switch (tile) {
    case 0: return launch_f32_tile<4, 32, 4, 1, 64, 4>(c, mode, stream);
    case 1: return launch_f32_tile<8, 32, 4, 1, 64, 4>(c, mode, stream);
    case 2: return launch_f32_tile<16, 64, 4, 2, 32, 4>(c, mode, stream);
    case 3: return launch_f32_tile<32, 64, 4, 4, 32, 3>(c, mode, stream);
    case 4: return launch_f32_tile<64, 64, 4, 8, 16, 4>(c, mode, stream);
    default: return launch_f32_tile<128, 128, 8, 8, 16, 3>(c, mode, stream);
  }
}

// Which of F32_TILES a float32 product of these sizes takes (-1: none).
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
    const int tile = pick_f32_tile(M, N);
    return tile < 0 ? GB_ERR_SIZE : launch_f32(tile, call, mode, stream);
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
