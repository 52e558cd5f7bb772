// bfloat16 latent attention on the tensor cores, for prompts and for single positions alike.
// Compiled for one latent size and one width of the rotated part (-DGB_LATENT_RANK, -DGB_LATENT_ROT).
//
// All heads read the same cached rows [c (RANK) | k_rot (ROT)], so the rows of a tile are
// (token, head) pairs: row r of a sequence's step is token r / H, head r % H, and a tile of keys
// that has been brought into shared memory once serves every head of several tokens (a prompt),
// or every head of the one token (decoding).  Per tile of KEYS keys:
//
//   S = Q K^T        mma.sync m16n8k16, Q [rows, RANK + ROT] and the key tile in shared memory
//   P = softmax      online, float32, log2 units, each row masked at its own position (and window)
//   O += P V         V = the first RANK columns of the same key tile (ldmatrix.trans)
//
// A group of 16 rows is worked by NSPLIT warps.  Each keeps its share of the queries' columns in
// registers for the whole kernel and scores every key of a tile over that share alone, so a key
// tile is read from shared memory once per group, not once per warp; the partial scores meet in
// shared memory and are added in warp order.  Each warp then owns RANK / NSPLIT of the output's
// columns, so that a wide latent does not have to fit one warp's registers.  Key tiles arrive by
// cp.async, one tile ahead; the queries pass through the same buffers before the first tile.
//
// The same kernel serves a prompt step whose keys and values were expanded per head (rows
// [v | k_nope | k_rot] with the value's width in RANK's place): head_stride > 0 gives every head rows
// of its own, contiguous from a sequence's first packed token, one head per grid layer, and
// out_scale (the layer's gate per head) or sigmoid(out_gate) (one per output number) is multiplied into
// the output.
//
// A step of single tokens has a kernel of its own (latent_decode_kernel), the same arithmetic over a stream of keys.
#include "latent_decode_ring.h"
#include "mma.cuh"
#include "tc_common.cuh"

#ifndef GB_LATENT_RANK
#define GB_LATENT_RANK 128
#endif
#ifndef GB_LATENT_ROT
#define GB_LATENT_ROT 16
#endif

namespace {

constexpr int RANK = GB_LATENT_RANK, ROT = GB_LATENT_ROT, KD = RANK + ROT;
static_assert(RANK % 16 == 0 && ROT % 16 == 0 && RANK >= 16, "latent and rotated widths must be multiples of 16");
constexpr int NSPLIT = RANK <= 128 ? 1 : (RANK <= 256 ? 2 : 4);
static_assert(RANK % (16 * NSPLIT) == 0, "the latent must divide into 16-column blocks per warp");
constexpr int LDS = KD + ((KD / 8) % 2 == 0 ? 8 : 0);   // row pitch in shared memory: an odd number of 16-byte units
constexpr int KSTEPS = KD / 16;                          // 16-column steps of a score
constexpr int KSW = (KSTEPS + NSPLIT - 1) / NSPLIT;      // steps a warp owns
constexpr int DW = RANK / NSPLIT;                        // output columns a warp owns
constexpr int MAX_GROUPS = NSPLIT == 4 ? 2 : 4;          // groups of 16 rows a CTA at most
constexpr int PART = RANK + 4;                           // floats of a split's part: o, then m and l (rows stay 16-byte aligned)
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void ldsm_x4(uint32_t* r, const void* p) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t* r, const void* p) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}

// grid (row tiles upper bound, 1, heads when they have rows of their own); block groups * NSPLIT * 32.  KEYS: keys a tile.
template <int KEYS>
__global__ void __launch_bounds__(MAX_GROUPS * NSPLIT * 32)
latent_attention_mma_kernel(const bf16* __restrict__ qa, long long ldq, bf16* __restrict__ out, long long ldo,
                            const bf16* __restrict__ cache, const int* __restrict__ page_table,
                            int table_width, int page_size, const int* __restrict__ cu_seqlens,
                            const int* __restrict__ seq_start, const int* __restrict__ seq_slot, int n_seqs, int H,
                            int window, long long head_stride, const float* __restrict__ out_scale,
                            const float* __restrict__ out_gate, long long ldg) {
  constexpr int NB = KEYS / 8;                         // blocks of 8 keys a tile
  constexpr int SXP = KEYS + 4;                        // pitch of the exchanged scores
  static_assert(NB % 2 == 0, "key blocks come in pairs");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_release_next();
  pdl_wait_prior();
  const int groups = blockDim.x / (32 * NSPLIT);
  const int tile_rows = groups * 16;
  bf16* Ks = (bf16*)smem_raw;                         // [2][KEYS][LDS]
  bf16* Qs = Ks;                                      // [tile_rows][LDS], before the first key tile
  float* Sx = (float*)(Ks + 2 * KEYS * LDS);          // [groups][NSPLIT][16][SXP], only with NSPLIT > 1
  // ---- which sequence and which tile of its rows
  const int heads_all = H;
  if (head_stride > 0) H = 1;                          // see per_head below
  int b = 0, tile = blockIdx.x, rows_b = 0;
  for (; b < n_seqs; ++b) {
    rows_b = (cu_seqlens[b + 1] - cu_seqlens[b]) * H;
    const int tiles = (rows_b + tile_rows - 1) / tile_rows;
    if (tile < tiles) break;
    tile -= tiles;
  }
  if (b >= n_seqs) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, c = lane & 3;
  const int rg = warp / NSPLIT, w = warp % NSPLIT;
  const int slot = seq_slot[b], start = seq_start[b], tok_base = cu_seqlens[b];
  const int row_base = tile * tile_rows;
  // head_stride > 0: every head has rows of its own (keys and values expanded per head), head
  // blockIdx.z's at cache + z * head_stride, a sequence's rows contiguous from its first packed token
  // (all sequences start at position 0); the rows of a tile are then tokens of that one head
  const bool per_head = head_stride > 0;
  const int hz = per_head ? (int)blockIdx.z : 0;
  if (per_head) {
    qa += (size_t)hz * KD;
    out += (size_t)hz * RANK;
    cache += (size_t)hz * head_stride;
  }
  // ---- the keys this CTA reads
  const int first_tok = row_base / H;
  const int last_tok = (min(rows_b, row_base + tile_rows) - 1) / H;
  const int hi = start + last_tok;
  const int lo_cta = window > 0 ? max(0, start + first_tok + 1 - window) : 0;
  const int my_begin = lo_cta / KEYS, my_end = hi / KEYS + 1;
  // ---- this thread's two rows
  const int r0 = row_base + rg * 16 + g, r1 = r0 + 8;
  const bool v0 = r0 < rows_b, v1 = r1 < rows_b;
  const int pos0 = v0 ? start + r0 / H : -1, pos1 = v1 ? start + r1 / H : -1;
  const int lo0 = window > 0 ? max(0, pos0 + 1 - window) : 0, lo1 = window > 0 ? max(0, pos1 + 1 - window) : 0;

  constexpr int CH = KD / 8;                           // 16-byte pieces of a row
  for (int e = tid; e < tile_rows * CH; e += blockDim.x) {
    const int r = e / CH, ch = e % CH, row = row_base + r;
    bf16* dst = Qs + (size_t)r * LDS + ch * 8;
    if (row < rows_b)
      cp_async16(dst, qa + (size_t)(tok_base + row / H) * ldq + (size_t)(row % H) * KD + ch * 8);
    else
      *(uint4*)dst = make_uint4(0, 0, 0, 0);
  }
  auto load_keys = [&](int t, int stage) {
    const int key0 = t * KEYS;
    const bf16* src;
    if (per_head) {
      src = cache + (size_t)(tok_base + key0) * KD;
    } else {
      const int page = page_table[(size_t)slot * table_width + (key0 / page_size) % table_width];
      src = cache + ((size_t)page * page_size + key0 % page_size) * KD;
    }
    bf16* dst = Ks + (size_t)stage * KEYS * LDS;
    for (int e = tid; e < KEYS * CH; e += blockDim.x) {
      const int r = e / CH, ch = e % CH;
      cp_async16(dst + (size_t)r * LDS + ch * 8, src + (size_t)r * KD + ch * 8);
    }
  };
  // ---- this warp's share of the queries' columns, into registers
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  uint32_t qf[KSW][4];
  {
    const bf16* q_lane = Qs + (size_t)(rg * 16 + (lane & 7) + 8 * ((lane >> 3) & 1)) * LDS + 8 * (lane >> 4);
#pragma unroll
    for (int i = 0; i < KSW; ++i) {
      const int ks = w * KSW + i;
      if (ks < KSTEPS) ldsm_x4(qf[i], q_lane + ks * 16);
      else qf[i][0] = qf[i][1] = qf[i][2] = qf[i][3] = 0;
    }
  }
  __syncthreads();                                     // the buffers are free for keys
  if (my_begin < my_end) load_keys(my_begin, 0);
  cp_async_commit();

  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  float o[DW / 8][4];
#pragma unroll
  for (int d = 0; d < DW / 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;

  for (int t = my_begin; t < my_end; ++t) {
    const int stage = (t - my_begin) & 1;
    cp_async_wait_all();
    __syncthreads();                                   // tile t (and Q) landed; everyone is done with tile t - 1
    if (t + 1 < my_end) load_keys(t + 1, stage ^ 1);
    cp_async_commit();
    const bf16* kt = Ks + (size_t)stage * KEYS * LDS;
    // ---- scores of all the tile's keys over this warp's share of the columns
    float s[NB][4];
#pragma unroll
    for (int j = 0; j < NB; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    {
      const bf16* k_lane = kt + (size_t)((lane & 7) + 8 * (lane >> 4)) * LDS + 8 * ((lane >> 3) & 1);
#pragma unroll
      for (int i = 0; i < KSW; ++i) {
        const int ks = w * KSW + i;
        if (ks < KSTEPS) {
#pragma unroll
          for (int j = 0; j < NB; j += 2) {
            uint32_t kb[4];                              // keys 8j..8j+7: regs 0, 1; keys 8j+8..8j+15: regs 2, 3
            ldsm_x4(kb, k_lane + (size_t)j * 8 * LDS + ks * 16);
            mma16816(s[j], qf[i][0], qf[i][1], qf[i][2], qf[i][3], kb[0], kb[1]);
            mma16816(s[j + 1], qf[i][0], qf[i][1], qf[i][2], qf[i][3], kb[2], kb[3]);
          }
        }
      }
      if (NSPLIT > 1) {
        float* sx = Sx + (size_t)rg * NSPLIT * 16 * SXP;
        float* mine = sx + (size_t)w * 16 * SXP;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          *(float2*)(mine + g * SXP + j * 8 + 2 * c) = make_float2(s[j][0], s[j][1]);
          *(float2*)(mine + (g + 8) * SXP + j * 8 + 2 * c) = make_float2(s[j][2], s[j][3]);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          float2 x = make_float2(0.f, 0.f), y = make_float2(0.f, 0.f);
#pragma unroll
          for (int ww = 0; ww < NSPLIT; ++ww) {
            const float2 a = *(const float2*)(sx + (size_t)ww * 16 * SXP + g * SXP + j * 8 + 2 * c);
            const float2 bb = *(const float2*)(sx + (size_t)ww * 16 * SXP + (g + 8) * SXP + j * 8 + 2 * c);
            x.x += a.x; x.y += a.y; y.x += bb.x; y.y += bb.y;
          }
          s[j][0] = x.x; s[j][1] = x.y; s[j][2] = y.x; s[j][3] = y.y;
        }
      }
    }
    // ---- softmax of the tile, each row masked at its own position
    const int key0 = t * KEYS;
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int key = key0 + 8 * j + 2 * c + e;
        s[j][e] = (key >= lo0 && key <= pos0) ? s[j][e] * LOG2E : -INFINITY;
        s[j][2 + e] = (key >= lo1 && key <= pos1) ? s[j][2 + e] * LOG2E : -INFINITY;
        mx0 = fmaxf(mx0, s[j][e]);
        mx1 = fmaxf(mx1, s[j][2 + e]);
      }
    const float n0 = fmaxf(m0, quad_max(mx0)), n1 = fmaxf(m1, quad_max(mx1));
    const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
    const float alpha0 = exp2f(m0 - u0), alpha1 = exp2f(m1 - u1);
    m0 = n0;
    m1 = n1;
    uint32_t p[NB][2];
    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const float a = exp2f(s[j][0] - u0), bb = exp2f(s[j][1] - u0);
      const float cc = exp2f(s[j][2] - u1), d = exp2f(s[j][3] - u1);
      sum0 += a + bb;
      sum1 += cc + d;
      p[j][0] = pack_bf16(a, bb);
      p[j][1] = pack_bf16(cc, d);
    }
    l0 = l0 * alpha0 + sum0;
    l1 = l1 * alpha1 + sum1;
#pragma unroll
    for (int d = 0; d < DW / 8; ++d) { o[d][0] *= alpha0; o[d][1] *= alpha0; o[d][2] *= alpha1; o[d][3] *= alpha1; }
    // ---- O += P V over this warp's columns of the latent
    const bf16* v_lane = kt + (size_t)((lane & 7) + 8 * ((lane >> 3) & 1)) * LDS + w * DW + 8 * (lane >> 4);
#pragma unroll
    for (int kk = 0; kk < KEYS / 16; ++kk) {
#pragma unroll
      for (int db = 0; db < DW / 16; ++db) {
        uint32_t vb[4];
        ldsm_x4_t(vb, v_lane + (size_t)kk * 16 * LDS + db * 16);
        mma16816(o[2 * db], p[2 * kk][0], p[2 * kk][1], p[2 * kk + 1][0], p[2 * kk + 1][1], vb[0], vb[1]);
        mma16816(o[2 * db + 1], p[2 * kk][0], p[2 * kk][1], p[2 * kk + 1][0], p[2 * kk + 1][1], vb[2], vb[3]);
      }
    }
  }
  cp_async_wait_all();
  l0 = quad_sum(l0);
  l1 = quad_sum(l1);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int row = half ? r1 : r0;
    if (!(half ? v1 : v0)) continue;
    float inv = 1.0f / (half ? l1 : l0);
    if (out_scale) inv *= out_scale[(size_t)(tok_base + row / H) * heads_all + (per_head ? hz : row % H)];
    bf16* dst = out + (size_t)(tok_base + row / H) * ldo + (size_t)(row % H) * RANK + w * DW + 2 * c;
    if (out_gate) {
      const float* z = out_gate + (size_t)(tok_base + row / H) * ldg + (size_t)(per_head ? hz : row % H) * RANK + w * DW + 2 * c;
#pragma unroll
      for (int d = 0; d < DW / 8; ++d)
        *(uint32_t*)(dst + d * 8) = pack_bf16(o[d][2 * half] * inv / (1.0f + __expf(-z[d * 8])),
                                              o[d][2 * half + 1] * inv / (1.0f + __expf(-z[d * 8 + 1])));
      continue;
    }
#pragma unroll
    for (int d = 0; d < DW / 8; ++d) *(uint32_t*)(dst + d * 8) = pack_bf16(o[d][2 * half] * inv, o[d][2 * half + 1] * inv);
  }
}

// ------------------------------------------------------------------ single tokens
// Decoding reads every cached row once for all heads, so it is a stream of key tiles, and its time is how steadily
// every SM pulls its share.  The tiles to read (KT keys of one sequence, for 16 GROUPS of its heads) are one flat list,
// sequence by sequence; CTA i of G takes the tiles [i P / G, (i + 1) P / G) whatever the lengths.  A producer warp asks
// for a tile in TMA boxes of KT rows x 128 bytes (swizzled, against bank conflicts) up to STAGES tiles ahead of
// KG teams of warps that take the tiles in turn, each with a softmax of its own; the teams meet at the end of a
// segment (the part of one sequence's list in the CTA's range), in their order.  A whole list is written out, a part
// goes to one of the CTA's two scratch places and latent_decode_merge_kernel adds the parts in key order: the same
// bits every run.  Every wait is bounded; one that runs out sets the status word and the CTA's abort flag.
// 16 sequences of 5,330 to 8,000 keys, 16 heads, rows of 512 + 64 (121 MB): 49 + 6 us with the keys dealt to 18 CTAs a
// sequence by the kernel above, two tiles in flight and a barrier of the block a tile; 37.5 + 6.5 us with a bulk copy a row,
// 30 + 6.5 us so (boxes of 32 rows x 128 bytes: 9 requests a tile instead of 32).
constexpr int KT = latent_ring::KT, MAX_SEQS = latent_ring::MAX_SEQS;
constexpr int BOXES = (KD + 63) / 64, BOX_BYTES = KT * 128, STAGE_BYTES = BOXES * BOX_BYTES;
static_assert(NSPLIT == latent_ring::warps_of(RANK), "the ring counts with as many warps");
template <int GROUPS>
struct Decode {
  static constexpr latent_ring::Ring R = latent_ring::ring(RANK, ROT, GROUPS);
  static constexpr bool FITS = R.stages > 0;
  static constexpr int KG = FITS ? R.teams : 1, STAGES = FITS ? R.stages : 2;
  static constexpr int WARPS = KG * NSPLIT * GROUPS, ROWS = 16 * GROUPS;
  static constexpr int SXP = KT + 8, PP = KT + 8;                // pitches of the scores' parts and of the weights
  static constexpr int SX = R.share, FLOATS = R.floats;
  static constexpr size_t SMEM = R.smem;
};

__device__ int g_latent_status;   // 0, or the first wait that ran out (1 free stage, 2 tile)

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort, int code) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255) == 255 && *abort) return false;
  }
  *abort = 1;
  atomicCAS(&g_latent_status, 0, code);
  return false;
}
__device__ __forceinline__ void team_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// A sequence's list: its first tile and how many, for every ROWS of its heads.
struct Span {
  int pos, lo, first, tiles;
};
__device__ __forceinline__ Span span_of(int b, const int* seq_start, int window) {
  Span s;
  s.pos = seq_start[b];
  s.lo = window > 0 ? max(0, s.pos + 1 - window) : 0;
  s.first = s.lo / KT;
  s.tiles = s.pos / KT + 1 - s.first;
  return s;
}
__device__ __forceinline__ int seq_of(const int* prefix, int n, int p) {      // the sequence whose tiles tile p is among
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// part: [G * 2][ROWS][PART].
template <int GROUPS>
__global__ void __launch_bounds__(Decode<GROUPS>::WARPS * 32 + 32, 1)
latent_decode_kernel(const __grid_constant__ CUtensorMap rows, const bf16* __restrict__ qa, long long ldq, bf16* __restrict__ out,
                     long long ldo, float* __restrict__ part, const int* __restrict__ page_table, int table_width, int page_size,
                     const int* __restrict__ seq_start, const int* __restrict__ seq_slot, int n_seqs, int H, int window) {
  using D = Decode<GROUPS>;
  constexpr int KG = D::KG, SXP = D::SXP, NB = KT / 8, STAGES = D::STAGES;
  extern __shared__ __align__(16) unsigned char smem_any[];
  unsigned char* smem_raw = smem_any + ((1024 - (smem_u32(smem_any) & 1023)) & 1023);      // the boxes' swizzle counts from there
  float* shared = (float*)(smem_raw + (size_t)STAGES * STAGE_BYTES);
  uint64_t* full = (uint64_t*)(shared + D::FLOATS);
  uint64_t* empty = full + STAGES;
  volatile int* abort = (volatile int*)(empty + STAGES);
  int* prefix = (int*)(abort + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_tiles = (H + D::ROWS - 1) / D::ROWS;
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], NSPLIT * GROUPS);
    }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // lengths and the page table are the step's inputs, not the work of the kernel before this one
  if (warp == 0) {
    int carry = 0;
    for (int base = 0; base < n_seqs; base += 32) {
      const int i = base + lane;
      int v = i < n_seqs ? span_of(i, seq_start, window).tiles * row_tiles : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += up;
      }
      if (i < n_seqs) prefix[i + 1] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) prefix[0] = 0;
  }
  __syncthreads();
  const long long P = prefix[n_seqs], G = gridDim.x;
  const int p0 = (int)(blockIdx.x * P / G), p1 = (int)((blockIdx.x + 1) * P / G);
  if (warp == D::WARPS) {
    // ---------------- producer.  A tile's page takes a chain of loads, so the lanes look up 32 tiles at a time
    auto lookup = [&](int p) -> long long {           // the first cache row of tile p
      if (p >= p1) return 0;
      const int b = seq_of(prefix, n_seqs, p);
      const Span sp = span_of(b, seq_start, window);
      const int key = (sp.first + (p - prefix[b]) % sp.tiles) * KT;
      return (long long)page_table[(size_t)seq_slot[b] * table_width + (key / page_size) % table_width] * page_size + key % page_size;
    };
    long long next = lookup(p0 + lane);
    pdl_wait_prior();
    bool ok = true;
    int it = 0;
    for (int base = p0; base < p1 && ok; base += 32) {
      const long long mine = next;
      next = lookup(base + 32 + lane);
      const int n = min(32, p1 - base);
      for (int i = 0; i < n && ok; ++i, ++it) {
        const long long row = __shfl_sync(0xffffffffu, mine, i);
        const int st = it % STAGES;
        if (it >= STAGES) ok = __all_sync(0xffffffffu, wait_or_abort(&empty[st], (it / STAGES - 1) & 1, abort, 1));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&full[st], STAGE_BYTES);
        __syncwarp();
        for (int x = lane; x < BOXES; x += 32)
          tma_load_2d(smem_raw + (size_t)st * STAGE_BYTES + (size_t)x * BOX_BYTES, &rows, x * 64, (int)row, &full[st]);
      }
    }
    pdl_release_next();
    return;
  }
  const int team = warp / (NSPLIT * GROUPS), rg = warp / NSPLIT % GROUPS, w = warp % NSPLIT;
  const int g = lane >> 2, c = lane & 3;
  pdl_wait_prior();
  float* mine = shared + (size_t)(team * GROUPS + rg) * D::SX;       // what the warps of these rows share
  float* tops = mine + NSPLIT * 16 * SXP;
  bf16* weights = (bf16*)(tops + NSPLIT * 16);
  const int bar = 2 + team * GROUPS + rg;
  // Where in a tile (boxes of KT rows x 128 bytes, their 16-byte pieces swizzled by the row) this lane's share of a piece lies
  auto piece = [&](int row, int at) { return (at >> 3) * BOX_BYTES + row * 128 + (((at & 7) ^ (row & 7)) << 4); };
  const int k_row = (lane & 7) + 8 * (lane >> 4), v_row = (lane & 7) + 8 * ((lane >> 3) & 1);
  bool ok = true;
  int it0 = 0, seg = 0;
  for (int p = p0; p < p1;) {
    const int b = seq_of(prefix, n_seqs, p);
    const Span sp = span_of(b, seq_start, window);
    const int rt = (p - prefix[b]) / sp.tiles, first = (p - prefix[b]) % sp.tiles, n = min(sp.tiles - first, p1 - p);
    const bool whole = first == 0 && n == sp.tiles;
    const int h0 = rt * D::ROWS + rg * 16 + g, h1 = h0 + 8;        // this thread's two heads
    const bool v0 = h0 < H, v1 = h1 < H;
    uint32_t qf[KSW][4];
    {
      const bf16* q0 = qa + (size_t)b * ldq + (size_t)h0 * KD + 2 * c;
      const bf16* q1 = q0 + 8 * KD;
#pragma unroll
      for (int i = 0; i < KSW; ++i) {
        const int ks = w * KSW + i;
        const bool in = ks < KSTEPS;
        qf[i][0] = in && v0 ? *(const uint32_t*)(q0 + ks * 16) : 0u;
        qf[i][1] = in && v1 ? *(const uint32_t*)(q1 + ks * 16) : 0u;
        qf[i][2] = in && v0 ? *(const uint32_t*)(q0 + ks * 16 + 8) : 0u;
        qf[i][3] = in && v1 ? *(const uint32_t*)(q1 + ks * 16 + 8) : 0u;
      }
    }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    float o[DW / 8][4];
#pragma unroll
    for (int d = 0; d < DW / 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    for (int i = (team + KG - it0 % KG) % KG; i < n; i += KG) {          // tile it0 + i of the CTA: team (it0 + i) % KG
      const int st = (it0 + i) % STAGES;
      // a wait that gives up ends no loop: the warps of a team go on to meet at their barriers
      if (ok) ok = wait_or_abort(&full[st], ((it0 + i) / STAGES) & 1, abort, 2);
      ok = __all_sync(0xffffffffu, ok);
      const unsigned char* kt = smem_raw + (size_t)st * STAGE_BYTES;
      float s[NB][4];
#pragma unroll
      for (int j = 0; j < NB; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
      for (int x = 0; x < KSW; ++x) {
        const int ks = w * KSW + x;
        if (ks < KSTEPS) {
#pragma unroll
          for (int j = 0; j < NB; j += 2) {
            uint32_t kb[4];
            ldsm_x4(kb, (const bf16*)(kt + j * 8 * 128 + piece(k_row, 2 * ks + ((lane >> 3) & 1))));
            mma16816(s[j], qf[x][0], qf[x][1], qf[x][2], qf[x][3], kb[0], kb[1]);
            mma16816(s[j + 1], qf[x][0], qf[x][1], qf[x][2], qf[x][3], kb[2], kb[3]);
          }
        }
      }
      // The parts of the scores meet in shared memory; a warp adds up those of its own share of the keys (in warp order),
      // takes their weights, and all warps read the weights back as the left operand of the second product.
      constexpr int OWN = NB / NSPLIT;                // blocks of 8 keys whose weights this warp takes
      if (NSPLIT > 1) {
        float* to = mine + (size_t)w * 16 * SXP;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          *(float2*)(to + g * SXP + j * 8 + 2 * c) = make_float2(s[j][0], s[j][1]);
          *(float2*)(to + (g + 8) * SXP + j * 8 + 2 * c) = make_float2(s[j][2], s[j][3]);
        }
        team_sync(bar, 32 * NSPLIT);
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
          float2 x = make_float2(0.f, 0.f), y = make_float2(0.f, 0.f);
#pragma unroll
          for (int ww = 0; ww < NSPLIT; ++ww) {
            const float* from = mine + (size_t)ww * 16 * SXP + (w * OWN + j) * 8 + 2 * c;
            const float2 aa = *(const float2*)(from + g * SXP), bb = *(const float2*)(from + (g + 8) * SXP);
            x.x += aa.x; x.y += aa.y; y.x += bb.x; y.y += bb.y;
          }
          s[j][0] = x.x; s[j][1] = x.y; s[j][2] = y.x; s[j][3] = y.y;
        }
      }
      const int key0 = (sp.first + first + i) * KT + w * (NSPLIT > 1 ? OWN * 8 : 0);
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int j = 0; j < OWN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = key0 + 8 * j + 2 * c + e;
          const bool in = key >= sp.lo && key <= sp.pos;
          s[j][e] = in ? s[j][e] * LOG2E : -INFINITY;
          s[j][2 + e] = in ? s[j][2 + e] * LOG2E : -INFINITY;
          mx0 = fmaxf(mx0, s[j][e]);
          mx1 = fmaxf(mx1, s[j][2 + e]);
        }
      mx0 = quad_max(mx0);
      mx1 = quad_max(mx1);
      if (NSPLIT > 1) {
        if (c == 0) tops[w * 16 + g] = mx0, tops[w * 16 + g + 8] = mx1;
        team_sync(bar, 32 * NSPLIT);
#pragma unroll
        for (int ww = 0; ww < NSPLIT; ++ww) mx0 = fmaxf(mx0, tops[ww * 16 + g]), mx1 = fmaxf(mx1, tops[ww * 16 + g + 8]);
      }
      const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
      const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
      const float alpha0 = exp2f(m0 - u0), alpha1 = exp2f(m1 - u1);
      m0 = n0;
      m1 = n1;
      uint32_t pk[NB][2];
      float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
      for (int j = 0; j < OWN; ++j) {
        const float aa = exp2f(s[j][0] - u0), bb = exp2f(s[j][1] - u0);
        const float cc = exp2f(s[j][2] - u1), dd = exp2f(s[j][3] - u1);
        sum0 += aa + bb;
        sum1 += cc + dd;
        pk[j][0] = pack_bf16(aa, bb);
        pk[j][1] = pack_bf16(cc, dd);
      }
      l0 = l0 * alpha0 + sum0;                        // of this warp's keys; the warps' sums meet at the segment's end
      l1 = l1 * alpha1 + sum1;
      if (NSPLIT > 1) {
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
          *(uint32_t*)(weights + g * D::PP + (w * OWN + j) * 8 + 2 * c) = pk[j][0];
          *(uint32_t*)(weights + (g + 8) * D::PP + (w * OWN + j) * 8 + 2 * c) = pk[j][1];
        }
        team_sync(bar, 32 * NSPLIT);
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk) {
          uint32_t a[4];
          ldsm_x4(a, weights + ((lane & 7) + 8 * ((lane >> 3) & 1)) * D::PP + kk * 16 + 8 * (lane >> 4));
          pk[2 * kk][0] = a[0]; pk[2 * kk][1] = a[1]; pk[2 * kk + 1][0] = a[2]; pk[2 * kk + 1][1] = a[3];
        }
      }
      if (__any_sync(0xffffffffu, alpha0 != 1.f || alpha1 != 1.f)) {      // most tiles leave the maxima where they are
#pragma unroll
        for (int d = 0; d < DW / 8; ++d) { o[d][0] *= alpha0; o[d][1] *= alpha0; o[d][2] *= alpha1; o[d][3] *= alpha1; }
      }
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk) {
#pragma unroll
        for (int db = 0; db < DW / 16; ++db) {
          uint32_t vb[4];
          ldsm_x4_t(vb, (const bf16*)(kt + kk * 16 * 128 + piece(v_row, w * (DW / 8) + 2 * db + (lane >> 4))));
          mma16816(o[2 * db], pk[2 * kk][0], pk[2 * kk][1], pk[2 * kk + 1][0], pk[2 * kk + 1][1], vb[0], vb[1]);
          mma16816(o[2 * db + 1], pk[2 * kk][0], pk[2 * kk][1], pk[2 * kk + 1][0], pk[2 * kk + 1][1], vb[2], vb[3]);
        }
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[st])) : "memory");
    }
    l0 = quad_sum(l0);
    l1 = quad_sum(l1);
    if (NSPLIT > 1) {           // the warps' sums, in warp order
      team_sync(bar, 32 * NSPLIT);
      if (c == 0) tops[w * 16 + g] = l0, tops[w * 16 + g + 8] = l1;
      team_sync(bar, 32 * NSPLIT);
      l0 = l1 = 0.f;
#pragma unroll
      for (int ww = 0; ww < NSPLIT; ++ww) l0 += tops[ww * 16 + g], l1 += tops[ww * 16 + g + 8];
      if (KG == 1) team_sync(bar, 32 * NSPLIT);
    }
    if (KG > 1) {
      // the teams meet in their order (in the memory of the scores' parts: all teams are past those)
      team_sync(1, D::WARPS * 32);
      if (team > 0) {
        float* to = shared + (size_t)((team - 1) * NSPLIT * GROUPS + warp % (NSPLIT * GROUPS)) * (DW / 2 + 4) * 32 + lane;
#pragma unroll
        for (int d = 0; d < DW / 8; ++d)
#pragma unroll
          for (int e = 0; e < 4; ++e) to[(4 * d + e) * 32] = o[d][e];
        to[DW / 2 * 32] = m0; to[(DW / 2 + 1) * 32] = m1; to[(DW / 2 + 2) * 32] = l0; to[(DW / 2 + 3) * 32] = l1;
      }
      team_sync(1, D::WARPS * 32);
      if (team == 0) {
#pragma unroll 1
        for (int k = 1; k < KG; ++k) {
          const float* from = shared + (size_t)((k - 1) * NSPLIT * GROUPS + warp) * (DW / 2 + 4) * 32 + lane;
          const float a0 = from[DW / 2 * 32], a1 = from[(DW / 2 + 1) * 32];
          const float n0 = fmaxf(m0, a0), n1 = fmaxf(m1, a1);
          const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
          const float x0 = exp2f(m0 - u0), x1 = exp2f(m1 - u1), y0 = exp2f(a0 - u0), y1 = exp2f(a1 - u1);
          m0 = n0;
          m1 = n1;
          l0 = l0 * x0 + from[(DW / 2 + 2) * 32] * y0;
          l1 = l1 * x1 + from[(DW / 2 + 3) * 32] * y1;
#pragma unroll
          for (int d = 0; d < DW / 8; ++d) {
            o[d][0] = o[d][0] * x0 + from[4 * d * 32] * y0;
            o[d][1] = o[d][1] * x0 + from[(4 * d + 1) * 32] * y0;
            o[d][2] = o[d][2] * x1 + from[(4 * d + 2) * 32] * y1;
            o[d][3] = o[d][3] * x1 + from[(4 * d + 3) * 32] * y1;
          }
        }
      }
      team_sync(1, D::WARPS * 32);
    }
    if (team == 0) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int h = half ? h1 : h0;
        if (h >= H) continue;
        if (whole) {
          const float inv = 1.0f / (half ? l1 : l0);
          bf16* dst = out + (size_t)b * ldo + (size_t)h * RANK + w * DW + 2 * c;
#pragma unroll
          for (int d = 0; d < DW / 8; ++d) *(uint32_t*)(dst + d * 8) = pack_bf16(o[d][2 * half] * inv, o[d][2 * half + 1] * inv);
        } else {
          float* dst = part + ((size_t)(blockIdx.x * 2 + (seg ? 1 : 0)) * D::ROWS + rg * 16 + g + 8 * half) * PART;
          if (w == 0 && c == 0) { dst[RANK] = half ? m1 : m0; dst[RANK + 1] = half ? l1 : l0; }
#pragma unroll
          for (int d = 0; d < DW / 8; ++d) *(float2*)(dst + w * DW + d * 8 + 2 * c) = make_float2(o[d][2 * half], o[d][2 * half + 1]);
        }
      }
    }
    p += n;
    it0 += n;
    ++seg;
  }
}

// A block per (token, head): adds the parts that the stream left for it, in key order, four columns a thread.  Which parts
// those are it works out from the step's lengths while the stream is still running; a thread's values of the first MERGE_AHEAD
// parts are asked for together with the parts' maxima and sums.
constexpr int MERGE_PARTS = 64, MERGE_AHEAD = 12;
__global__ void __launch_bounds__(128) latent_decode_merge_kernel(const float* __restrict__ part, const int* __restrict__ seq_start,
                                                                  bf16* __restrict__ out, long long ldo, int n_seqs, int H, int rows,
                                                                  int window, unsigned G) {
  __shared__ float ms[MERGE_PARTS], ls[MERGE_PARTS];
  __shared__ int at[MERGE_PARTS];
  __shared__ unsigned before, mine, all;
  pdl_release_next();
  const int b = blockIdx.x / H, h = blockIdx.x % H, row_tiles = (H + rows - 1) / rows;
  if (threadIdx.x < 32) {
    unsigned sum = 0, ahead = 0;
    for (int i = threadIdx.x; i < n_seqs; i += 32) {
      const unsigned v = span_of(i, seq_start, window).tiles;
      sum += v;
      if (i < b) ahead += v;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d), ahead += __shfl_xor_sync(0xffffffffu, ahead, d);
    if (threadIdx.x == 0) before = ahead * row_tiles, all = sum * row_tiles, mine = span_of(b, seq_start, window).tiles;
  }
  __syncthreads();
  const unsigned long long P = all;
  const unsigned u0 = before + h / rows * mine, u1 = u0 + mine;
  const int first = (int)(((unsigned long long)(u0 + 1) * G - 1) / P), last = (int)(((unsigned long long)u1 * G - 1) / P), n = last - first + 1;
  auto place = [&](int j) -> int {               // the scratch place of part j, -1: a CTA without tiles
    const unsigned long long cta = first + j, start = cta * P / G;
    return start == (cta + 1) * P / G ? -1 : (int)cta * 2 + (start >= u0 ? 0 : 1);
  };
  if ((int)threadIdx.x < min(n, MERGE_PARTS)) at[threadIdx.x] = place(threadIdx.x);
  pdl_wait_prior();                              // every block waits, also one with nothing to add
  if (n == 1) return;                            // one CTA had all of it
  __syncthreads();
  float M = -INFINITY, L = 0.f;
  constexpr int PER = (RANK + 511) / 512;        // four columns a thread, 512 a round of the block
  float4 acc[PER];
#pragma unroll
  for (int r = 0; r < PER; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int base = 0; base < n; base += MERGE_PARTS) {
    const int cn = min(MERGE_PARTS, n - base);
    if (base > 0) {
      __syncthreads();
      if ((int)threadIdx.x < cn) at[threadIdx.x] = place(base + threadIdx.x);
      __syncthreads();
    }
    const int d0 = 4 * threadIdx.x;
    float4 v[MERGE_AHEAD];
#pragma unroll
    for (int j = 0; j < MERGE_AHEAD; ++j)
      v[j] = j < cn && at[j] >= 0 && d0 < RANK ? *(const float4*)(part + ((size_t)at[j] * rows + h % rows) * PART + d0)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
    if ((int)threadIdx.x < cn) {
      const int slot = at[threadIdx.x];
      const float* src = part + ((size_t)max(slot, 0) * rows + h % rows) * PART;
      ms[threadIdx.x] = slot >= 0 ? src[RANK] : -INFINITY;
      ls[threadIdx.x] = slot >= 0 ? src[RANK + 1] : 0.f;
    }
    __syncthreads();
    float top = M;
    for (int s = 0; s < cn; ++s) top = fmaxf(top, ms[s]);
    const float was = M == -INFINITY ? 0.f : exp2f(M - top);
    M = top;
    L *= was;
    for (int s = 0; s < cn; ++s) L += ms[s] > -INFINITY ? ls[s] * exp2f(ms[s] - M) : 0.f;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
      const int d = d0 + 512 * r;
      if (d >= RANK) break;
      acc[r] = make_float4(acc[r].x * was, acc[r].y * was, acc[r].z * was, acc[r].w * was);
      int s0 = 0;
      if (r == 0) {
#pragma unroll
        for (int j = 0; j < MERGE_AHEAD; ++j) {
          if (j >= cn) break;
          const float f = ms[j] > -INFINITY ? exp2f(ms[j] - M) : 0.f;
          acc[0].x += v[j].x * f; acc[0].y += v[j].y * f; acc[0].z += v[j].z * f; acc[0].w += v[j].w * f;
        }
        s0 = MERGE_AHEAD;
      }
#pragma unroll 4
      for (int s = s0; s < cn; ++s) {
        if (at[s] < 0) continue;
        const float4 x = *(const float4*)(part + ((size_t)at[s] * rows + h % rows) * PART + d);
        const float f = ms[s] > -INFINITY ? exp2f(ms[s] - M) : 0.f;
        acc[r].x += x.x * f; acc[r].y += x.y * f; acc[r].z += x.z * f; acc[r].w += x.w * f;
      }
    }
  }
  const float inv = 1.0f / L;
#pragma unroll
  for (int r = 0; r < PER; ++r) {
    const int d = 4 * threadIdx.x + 512 * r;
    if (d >= RANK) break;
    bf16* dst = out + (size_t)b * ldo + (size_t)h * RANK + d;
    *(uint32_t*)dst = pack_bf16(acc[r].x * inv, acc[r].y * inv);
    *(uint32_t*)(dst + 2) = pack_bf16(acc[r].z * inv, acc[r].w * inv);
  }
}

template <int GROUPS>
int launch_decode(const CUtensorMap& rows, const bf16* qa, long long ldq, bf16* out, long long ldo, float* scratch, const int* page_table,
                  int table_width, int page_size, const int* seq_start, const int* seq_slot, int n_seqs, int H, int window, int ctas,
                  cudaStream_t stream) {
  using D = Decode<GROUPS>;
  static_assert(D::SMEM <= latent_ring::ROOM, "shared memory");
  static bool allowed = false;
  if (!allowed) {
    if (cudaFuncSetAttribute(latent_decode_kernel<GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)D::SMEM) != cudaSuccess)
      return GB_ERR_SIZE;
    allowed = true;
  }
  gb_launch(latent_decode_kernel<GROUPS>, dim3(ctas), dim3(D::WARPS * 32 + 32), D::SMEM, stream, rows, qa, ldq, out, ldo, scratch,
            page_table, table_width, page_size, seq_start, seq_slot, n_seqs, H, window);
  gb_launch(latent_decode_merge_kernel, dim3(n_seqs * H), dim3(128), 0, stream, (const float*)scratch, seq_start, out, ldo, n_seqs,
            H, D::ROWS, window, (unsigned)ctas);
  return gb_launch_status();
}

template <int KEYS>
int launch_latent(const bf16* qa, long long ldq, bf16* out, long long ldo, const bf16* cache, const int* page_table,
                  int table_width, int page_size, const int* cu_seqlens, const int* seq_start, const int* seq_slot, int n_seqs,
                  int ntok, int H, int groups, int window, long long head_stride, const float* out_scale,
                  const float* out_gate, long long ldg, cudaStream_t stream) {
  const int tile_rows = groups * 16;
  if (tile_rows > 2 * KEYS) return GB_ERR_SIZE;       // the queries are staged in the key buffers
  const size_t smem = 2 * (size_t)KEYS * LDS * sizeof(bf16) +
                      (NSPLIT > 1 ? (size_t)groups * NSPLIT * 16 * (KEYS + 4) * sizeof(float) : 0);
  static size_t allowed = 0;
  if (smem > allowed) {
    if (cudaFuncSetAttribute(latent_attention_mma_kernel<KEYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return GB_ERR_SIZE;
    allowed = smem;
  }
  const int row_heads = head_stride > 0 ? 1 : H;
  dim3 grid(((long long)ntok * row_heads + tile_rows - 1) / tile_rows + n_seqs, 1, head_stride > 0 ? H : 1);
  gb_launch(latent_attention_mma_kernel<KEYS>, grid, dim3(groups * NSPLIT * 32), smem, stream, qa, ldq, out, ldo, cache,
            page_table, table_width, page_size, cu_seqlens, seq_start, seq_slot, n_seqs, H, window, head_stride,
            out_scale, out_gate, ldg);
  return gb_launch_status();
}

}  // namespace

// qa: [ntok, H * (RANK + ROT)] bfloat16 rows ldq apart, packed by sequence (cu_seqlens [n_seqs + 1]);
// out: [ntok, H * RANK]; cache: [pages, page_size, RANK + ROT]; seq_start: each sequence's length
// before the step (the cache already holds the step's own rows).  max_rows: the most rows (tokens * H)
// one sequence brings, for the size of a CTA.  head_stride > 0: the rows are per head and contiguous
// (cache: [H][all packed tokens + a tile's worth][RANK + ROT], elements head_stride apart; every
// sequence starts at position 0; no page table).  out_scale: float32 [ntok, H] or null,
// multiplied into the output; out_gate: float32 [ntok, H * RANK] rows ldg apart or null, its
// sigmoid multiplied into the output.
GB_EXPORT int gb_latent_attention_mma(const void* qa, long long ldq, void* out, long long ldo, const void* cache,
                                      const int* page_table, int table_width, int page_size,
                                      const int* cu_seqlens, const int* seq_start, const int* seq_slot, int n_seqs,
                                      int ntok, int H, int rank, int rot, int max_rows, int window,
                                      long long head_stride, const float* out_scale, const float* out_gate, long long ldg,
                                      cudaStream_t stream) {
  if (ntok <= 0 || n_seqs <= 0) return 0;
  if (rank != RANK || rot != ROT || H <= 0 || page_size % 64) return GB_ERR_SIZE;
  if (((uintptr_t)qa & 15) || (ldq % 8) || ((uintptr_t)out & 3) || (ldo % 2) || ((uintptr_t)cache & 15)) return GB_ERR_SIZE;
  if (head_stride > 0 && (H > 65535 || head_stride % 8)) return GB_ERR_SIZE;
  int groups = (max_rows + 15) / 16;
  groups = groups < 1 ? 1 : (groups > MAX_GROUPS ? MAX_GROUPS : groups);
  return launch_latent<64>((const bf16*)qa, ldq, (bf16*)out, ldo, (const bf16*)cache, page_table, table_width, page_size,
                           cu_seqlens, seq_start, seq_slot, n_seqs, ntok, H, groups, window, head_stride, out_scale, out_gate, ldg, stream);
}

// Floats of scratch for a step of single tokens on `ctas` CTAs; 0: the rows are too wide for the stream (such steps run on
// the kernel of the prompts).
GB_EXPORT long long gb_latent_decode_scratch(int H, int ctas) {
  if (!(H > 16 ? Decode<2>::FITS : Decode<1>::FITS)) return 0;
  return (long long)ctas * 2 * (H > 16 ? 32 : 16) * PART;
}

// Every sequence brings one token: row b of qa and out is sequence b's.  cache: cache_rows rows.  scratch: gb_latent_decode_scratch() floats,
// 16-byte aligned.
GB_EXPORT int gb_latent_decode(const void* qa, long long ldq, void* out, long long ldo, float* scratch, const void* cache,
                               long long cache_rows, const int* page_table, int table_width, int page_size, const int* seq_start, const int* seq_slot,
                               int n_seqs, int H, int rank, int rot, int window, int ctas, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (rank != RANK || rot != ROT || H <= 0 || page_size % 64 || n_seqs > MAX_SEQS || ctas < 1) return GB_ERR_SIZE;
  if (((uintptr_t)qa & 15) || (ldq % 8) || ((uintptr_t)out & 3) || (ldo % 2) || ((uintptr_t)cache & 15) || ((uintptr_t)scratch & 15) || !scratch)
    return GB_ERR_SIZE;
  CUtensorMap rows;
  if (cache_rows < KT || cache_rows > INT_MAX || !tensor_map(&rows, cache, (uint64_t)cache_rows, KD, KD * 2, KT)) return GB_ERR_ARG;
  if (H > 16) {
    if constexpr (Decode<2>::FITS)
      return launch_decode<2>(rows, (const bf16*)qa, ldq, (bf16*)out, ldo, scratch, page_table, table_width, page_size, seq_start, seq_slot,
                              n_seqs, H, window, ctas, stream);
  } else {
    if constexpr (Decode<1>::FITS)
      return launch_decode<1>(rows, (const bf16*)qa, ldq, (bf16*)out, ldo, scratch, page_table, table_width, page_size, seq_start, seq_slot,
                              n_seqs, H, window, ctas, stream);
  }
  return GB_ERR_SIZE;
}

// 0, or the code of the first bounded wait that ran out (synchronizes the device).
GB_EXPORT int gb_latent_decode_status(int reset) {
  int v = -1;
  if (cudaMemcpyFromSymbol(&v, g_latent_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset) {
    int zero = 0;
    cudaMemcpyToSymbol(g_latent_status, &zero, sizeof(int));
  }
  return v;
}
