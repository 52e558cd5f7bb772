// Routed feed-forward (mixture of experts): the router and the token-major expert kernels.
//
//   z[t, e]  = router[e] . h[t] + bias[e]                       (float32)
//   chosen   = the `top` largest z (the lower index wins a tie); weight = softmax over the chosen z
//   expert:    g = min(gate h, limit), u = clamp(up h, -limit, limit)
//              y = g * sigmoid(alpha g) * (u + shift);  out = down y
//   residual[t] += sum over chosen of weight * expert_e(h[t])  +  sigmoid(sg . h[t]) * shared(h[t])
//
// Three more forms for designs that ask for them: ROUTE_SOFTMAX_ALL (the weights are the chosen experts'
// shares of the softmax over ALL experts, not renormalized); ROUTE_SIGMOID (scores s = sigmoid(router . h);
// chosen by s + bias, weighted by s / (sum of the chosen s + 1e-20) * scale, the bias left out; in
// ROUTE_SIGMOID_RAW by s * scale as it is); and
// experts without a gate (gb_moe_up: y = act(up h), act the exact, erf GELU or the square of relu; out =
// down y; the first matrices are [E, ff, width]).  `col_scale` [width] multiplies what is added into the residual.
// A design may weigh an expert's input instead of its output, expert(weight * h): `in_wts` multiplies the
// gate's and up's sums before the activation, and gb_moe_down is given no weights.
//
// The router's logits are a product like any other (the part computes them in float32); this unit
// picks the experts from them and runs the experts token-major: a block owns one (token, chosen
// expert) pair and a run of the expert's features, so the kernels need nothing from the host about
// who chose what and run inside captured steps.  Every pair's down product leaves a weighted
// float32 row, and a token's rows are added into the residual in the order of its chosen list,
// then the shared expert: the same bits whatever else is in the batch.  All sums are float32.
// (In bfloat16 a block owns an expert instead, with the entries that chose it: moe_few_kernel.)
#include "mma.cuh"

template <typename T> struct Vec;
template <> struct Vec<float> { static constexpr int N = 4; typedef float4 type; };
template <> struct Vec<bf16> { static constexpr int N = 8; typedef uint4 type; };

__device__ __forceinline__ void unpack(const float4& v, float* f) { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
__device__ __forceinline__ void unpack(const uint4& v, float* f) {
  const __nv_bfloat162* p = (const __nv_bfloat162*)&v;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(p[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}

// Lanes' shares of two rows . xs (xs float32 in shared memory) at once, so that twice the loads are
// in flight; the caller adds the lanes with warp_sum.  `vec`: the rows start on 16-byte boundaries
// and n is a multiple of the vector width.
template <typename T>
__device__ __forceinline__ void lane_dot2(const T* __restrict__ r0, const T* __restrict__ r1, const float* __restrict__ xs,
                                          int n, int lane, bool vec, float& a0, float& a1) {
  a0 = a1 = 0.f;
  if (vec) {
    constexpr int V = Vec<T>::N;
    const typename Vec<T>::type* p0 = (const typename Vec<T>::type*)r0;
    const typename Vec<T>::type* p1 = (const typename Vec<T>::type*)r1;
#pragma unroll 2
    for (int i = lane; i < n / V; i += 32) {
      float f0[V], f1[V];
      const typename Vec<T>::type v0 = p0[i], v1 = p1[i];
      unpack(v0, f0);
      unpack(v1, f1);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const float x = xs[i * V + k];
        a0 = fmaf(f0[k], x, a0);
        a1 = fmaf(f1[k], x, a1);
      }
    }
  } else {
    for (int i = lane; i < n; i += 32) {
      a0 = fmaf(to_f32(r0[i]), xs[i], a0);
      a1 = fmaf(to_f32(r1[i]), xs[i], a1);
    }
  }
}

template <typename T> __device__ __forceinline__ bool rows_vectorize(const T* base, int n) {
  return n % Vec<T>::N == 0 && ((uintptr_t)base & 15) == 0;
}

// ---- router: the logits come from a product (float32 [ntok, ldz]); a warp per token adds the
// bias, picks the `top` largest (the lower index wins a tie) and weighs them as `mode` says (the
// softmax over those alone by default).  Column E of z, when there is one, is the shared expert's gate logit.
enum { ROUTE_SOFTMAX_TOP = 0, ROUTE_SOFTMAX_ALL = 1, ROUTE_SIGMOID = 2, ROUTE_SIGMOID_RAW = 3 };
__global__ void __launch_bounds__(128) moe_topk_kernel(const float* __restrict__ zin, long long ldz,
                                                       const float* __restrict__ bias, int* __restrict__ idx,
                                                       float* __restrict__ wts, float* __restrict__ sg, int ntok, int E,
                                                       int top, int has_gate, int mode, float scale) {
  extern __shared__ float smem[];
  pdl_release_next();
  pdl_wait_prior();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * 4 + warp;
  if (t >= ntok) return;
  float* z = smem + (size_t)warp * E;
  for (int e = lane; e < E; e += 32) {
    const float v = zin[(size_t)t * ldz + e];
    z[e] = (mode >= ROUTE_SIGMOID ? 1.0f / (1.0f + expf(-v)) : v) + (bias ? bias[e] : 0.f);
  }
  if (has_gate && lane == 0) sg[t] = 1.0f / (1.0f + expf(-zin[(size_t)t * ldz + E]));
  __syncwarp();
  float mine = 0.f, first = 0.f;   // lane k keeps the k-th chosen logit
  int mine_at = 0;                 // and whose it is
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = z[e];
      if (v > best || (v == best && e < at)) { best = v; at = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (k == 0) first = best;
    if (lane == k) { mine = best; mine_at = at < E ? at : 0; }
    if (lane == 0) {
      idx[(size_t)t * top + k] = at < E ? at : 0;
      if (at < E) z[at] = -INFINITY;
    }
    __syncwarp();
  }
  if (mode >= ROUTE_SIGMOID) {
    const float s = lane < top ? 1.0f / (1.0f + expf(-zin[(size_t)t * ldz + mine_at])) : 0.f;
    const float total = mode == ROUTE_SIGMOID ? warp_sum(s) + 1e-20f : 1.f;
    if (lane < top) wts[(size_t)t * top + lane] = s / total * scale;
    return;
  }
  const float e = lane < top ? expf(mine - first) : 0.f;
  float sum = warp_sum(e);
  if (mode == ROUTE_SOFTMAX_ALL) {               // the experts not chosen join the denominator (the chosen ones' places hold -inf: nothing)
    float rest = 0.f;
    for (int i = lane; i < E; i += 32) rest += expf(z[i] - first);
    sum += warp_sum(rest);
  }
  if (lane < top) wts[(size_t)t * top + lane] = e / sum * scale;
}

// ---- gate and up of one (token, slot): FEATS features a block, a warp per feature in turn
constexpr int FEATS = 32;

template <typename T>
__global__ void __launch_bounds__(256) moe_gate_up_kernel(const T* __restrict__ h, long long ldh,
                                                          const int* __restrict__ idx, const T* __restrict__ w_gu,
                                                          const T* __restrict__ ws_gu, T* __restrict__ y, int width,
                                                          int ff, int ffs, int ffmax, int top, int slots, float limit,
                                                          float limit_s, float alpha, float shift,
                                                          const float* __restrict__ in_wts) {
  extern __shared__ float xs[];   // [width]
  pdl_release_next();
  pdl_wait_prior();
  const int t = blockIdx.x / slots, s = blockIdx.x % slots;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool routed = s < top;
  const int nf = routed ? ff : ffs;
  const int f0 = blockIdx.y * FEATS;
  if (f0 >= nf) return;
  const T* W = routed ? w_gu + (size_t)idx[(size_t)t * top + s] * 2 * ff * width : ws_gu;
  const float lim = routed ? limit : limit_s;
  for (int i = tid; i < width; i += 256) xs[i] = to_f32(h[(size_t)t * ldh + i]);
  __syncthreads();
  const bool vec = rows_vectorize(W, width);
  for (int f = f0 + warp; f < min(nf, f0 + FEATS); f += 8) {
    float g, u;
    lane_dot2(W + (size_t)f * width, W + (size_t)(nf + f) * width, xs, width, lane, vec, g, u);
    g = warp_sum(g);
    u = warp_sum(u);
    if (lane == 0) {
      if (in_wts && routed) {
        const float wt = in_wts[(size_t)t * top + s];
        g *= wt;
        u *= wt;
      }
      g = fminf(g, lim);
      u = fminf(fmaxf(u, -lim), lim);
      const float a = g / (1.0f + expf(-alpha * g)) * (u + shift);
      y[((size_t)t * slots + s) * ffmax + f] = from_f32<T>(a);
    }
  }
}

// ---- the same for experts without a gate: y = act(up h), two features a warp at a time
enum { ACT_GELU = 1, ACT_RELU2 = 2 };     // the exact (erf) GELU; the square of relu
__device__ __forceinline__ float plain_act(float x, int act) {
  if (act == ACT_RELU2) return fmaxf(x, 0.f) * fmaxf(x, 0.f);
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}

template <typename T>
__global__ void __launch_bounds__(256) moe_up_kernel(const T* __restrict__ h, long long ldh, const int* __restrict__ idx,
                                                     const T* __restrict__ w_up, T* __restrict__ y, int width, int ff, int top, int act) {
  extern __shared__ float xs[];   // [width]
  pdl_release_next();
  pdl_wait_prior();
  const int t = blockIdx.x / top, s = blockIdx.x % top;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f0 = blockIdx.y * FEATS;
  if (f0 >= ff) return;
  const T* W = w_up + (size_t)idx[(size_t)t * top + s] * ff * width;
  for (int i = tid; i < width; i += 256) xs[i] = to_f32(h[(size_t)t * ldh + i]);
  __syncthreads();
  const bool vec = rows_vectorize(W, width);
  for (int f = f0 + warp * 2; f < min(ff, f0 + FEATS); f += 16) {
    float a, b;
    const bool two = f + 1 < ff;
    lane_dot2(W + (size_t)f * width, W + (size_t)(two ? f + 1 : f) * width, xs, width, lane, vec, a, b);
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
      y[((size_t)t * top + s) * ff + f] = from_f32<T>(plain_act(a, act));
      if (two) y[((size_t)t * top + s) * ff + f + 1] = from_f32<T>(plain_act(b, act));
    }
  }
}

// ---- down of one (token, slot), weighted, into a float32 row of its own; the rows of a token are
// added into the residual in slot order by moe_sum_kernel
template <typename T>
__global__ void __launch_bounds__(256) moe_down_kernel(const T* __restrict__ y, const int* __restrict__ idx,
                                                       const float* __restrict__ wts, const float* __restrict__ sg,
                                                       const T* __restrict__ w_d, const T* __restrict__ ws_d,
                                                       float* __restrict__ rows, int width, int ff, int ffs, int ffmax,
                                                       int top, int slots) {
  extern __shared__ float ys[];   // [ffmax]
  pdl_release_next();
  pdl_wait_prior();
  const int t = blockIdx.x / slots, s = blockIdx.x % slots;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool routed = s < top;
  const int nf = routed ? ff : ffs;
  for (int i = tid; i < nf; i += 256) ys[i] = to_f32(y[((size_t)t * slots + s) * ffmax + i]);
  __syncthreads();
  const T* W = routed ? w_d + (size_t)idx[(size_t)t * top + s] * width * ff : ws_d;
  const float wt = routed ? (wts ? wts[(size_t)t * top + s] : 1.f) : sg[t];
  const bool vec = rows_vectorize(W, nf);
  const int n0 = blockIdx.y * FEATS;
  for (int n = n0 + warp * 2; n < min(width, n0 + FEATS); n += 16) {
    float a, b;
    const bool two = n + 1 < width;
    lane_dot2(W + (size_t)n * nf, W + (size_t)(two ? n + 1 : n) * nf, ys, nf, lane, vec, a, b);
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
      rows[((size_t)t * slots + s) * width + n] = a * wt;
      if (two) rows[((size_t)t * slots + s) * width + n + 1] = b * wt;
    }
  }
}

// ---- all three in bfloat16 for a few tokens, by expert on the tensor cores: a block owns an expert (or the shared one) and
// two runs of its rows, and works them for all the entries that chose it, so that weights come once however many tokens
// want them, and costs no arithmetic to speak of.  The weights are the left operand of mma.sync, straight from memory (a
// lane's 16 bytes are its share of 32 inner dims in both operands), the entries' vectors the right one, eight entries a
// column block; the inner dimension is dealt in pieces of 64 to KS warps whose sums meet in shared memory in warp order.
// An entry's column does not depend on the other columns: the same bits whatever else is in the batch.  Bound by the
// stream of the chosen experts' weights: 8 tokens, 6 of 64 experts of 1,408 and a shared one of 2,816, width 2,048
// (639 MB): gate and up, and down 89 + 55 us token by token on FFMA, 69 + 40 us so.
enum { FEW_GATED, FEW_PLAIN, FEW_DOWN };
constexpr int FEW_LIST = 2048;                    // entries a step may have
constexpr int FEW_KS = 4, FEW_RUNS = 8 / FEW_KS;  // warps along the inner dimension; runs of 32 rows (gate and up: 16 of each) a block
constexpr int FEW_COLS = 16;                      // entries a pass

template <int MODE, int NT>
__device__ __forceinline__ void few_sums(const bf16* const (&r)[4], const bf16* const (&x)[NT], int blocks, int kw, float (&acc)[2][NT][4]) {
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[t][n][0] = acc[t][n][1] = acc[t][n][2] = acc[t][n][3] = 0.f;
#pragma unroll 1
  for (int kb = 2 * kw; kb < blocks; kb += 2 * FEW_KS) {
    const bool both = kb + 1 < blocks;
    uint4 a[2][4], b[2][NT];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int at = (half && !both ? kb : kb + half) * 32;
#pragma unroll
      for (int i = 0; i < 4; ++i) a[half][i] = *(const uint4*)(r[i] + at);
#pragma unroll
      for (int n = 0; n < NT; ++n) b[half][n] = *(const uint4*)(x[n] + at);
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (half && !both) break;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 p = a[half][2 * t], q = a[half][2 * t + 1], v = b[half][n];
          mma16816(acc[t][n], p.x, q.x, p.y, q.y, v.x, v.y);
          mma16816(acc[t][n], p.z, q.z, p.w, q.w, v.z, v.w);
        }
    }
  }
}

// grid (the shared expert, if there is one, then every expert or, `by_entry`, every entry; runs of 32 FEW_RUNS rows).  Where there are
// fewer entries than experts a block stands for an entry and leaves where an earlier one has its expert: blocks of experts that
// nobody chose cost more than they find (one token, 10 of 512 experts of 256, width 768: 40 us a layer, 27 token by token).
template <int MODE>
__global__ void __launch_bounds__(256, 2) moe_few_kernel(const bf16* __restrict__ x, long long ldx, const int* __restrict__ idx,
                                                         const bf16* __restrict__ w, const bf16* __restrict__ ws, bf16* __restrict__ y,
                                                         float* __restrict__ rows, int ntok, int width, int ff, int ffs, int ffmax,
                                                         int top, int slots, float limit, float limit_s, float alpha, float shift,
                                                         int act, const float* __restrict__ in_wts, const float* __restrict__ wts,
                                                         const float* __restrict__ sg, int by_entry) {
  __shared__ int list[FEW_LIST], found;
  __shared__ float sums[8][2][16][FEW_COLS + 1];
  pdl_release_next();
  pdl_wait_prior();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  const bool routed = slots == top || blockIdx.x > 0;
  const int which = (int)blockIdx.x - (slots - top), e = routed && by_entry ? idx[which] : which, nf = routed ? ff : ffs;
  const int n_in = MODE == FEW_DOWN ? nf : width, n_out = MODE == FEW_DOWN ? width : nf;
  constexpr int OUT = (MODE == FEW_GATED ? 16 : 32) * FEW_RUNS;
  const int f0 = blockIdx.y * OUT;
  if (f0 >= n_out) return;
  int n = ntok;
  if (routed) {            // the entries that chose this expert, in order
    if (warp == 0) {
      int at = 0;
      for (int base = 0; base < ntok * top; base += 32) {
        const int i = base + lane;
        const bool mine = i < ntok * top && idx[i] == e;
        const unsigned votes = __ballot_sync(0xffffffffu, mine);
        if (mine) list[at + __popc(votes & ((1u << lane) - 1))] = i / top * slots + i % top;
        at += __popc(votes);
      }
      if (lane == 0) found = at;
    }
    __syncthreads();
    n = found;
    if (n == 0 || (by_entry && list[0] != which / top * slots + which % top)) return;
  } else {
    for (int t = tid; t < ntok; t += 256) list[t] = t * slots + top;
    __syncthreads();
  }
  const bf16* W = routed ? w + (size_t)e * (MODE == FEW_GATED ? 2 : 1) * ff * width : ws;
  const int run = warp / FEW_KS, kw = warp % FEW_KS;
  const bf16* r[4];         // this lane's rows: g and g + 8 of two blocks of 16 (beyond the last: the last, not stored)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int f = min(n_out - 1, MODE == FEW_GATED ? f0 + run * 16 + g + 8 * (i & 1) : f0 + run * 32 + g + 8 * i);
    r[i] = W + (size_t)(MODE == FEW_GATED && i >= 2 ? n_out + f : f) * n_in + 8 * c;
  }
  const float lim = routed ? limit : limit_s;
  for (int done = 0; done < n; done += FEW_COLS) {
    const int now = min(FEW_COLS, n - done);
    const bf16* src[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int entry = list[done + min(now - 1, 8 * j + g)];
      src[j] = (MODE == FEW_DOWN ? x + (size_t)entry * ffmax : x + (size_t)(entry / slots) * ldx) + 8 * c;
    }
    float acc[2][2][4];
    if (now > 8) {
      few_sums<MODE, 2>(r, src, n_in / 32, kw, acc);
    } else {
      const bf16* one[1] = {src[0]};
      float part[2][1][4];
      few_sums<MODE, 1>(r, one, n_in / 32, kw, part);
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[t][0][k] = part[t][0][k], acc[t][1][k] = 0.f;
    }
    if (done) __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) sums[warp][t][g + 8 * (k >> 1)][8 * j + 2 * c + (k & 1)] = acc[t][j][k];
    __syncthreads();
    auto total = [&](int rn, int t, int row, int col) {
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < FEW_KS; ++k) v += sums[rn * FEW_KS + k][t][row][col];
      return v;
    };
    for (int i = tid; i < OUT * now; i += 256) {
      const int o = i % OUT, col = i / OUT, f = f0 + o;
      if (f >= n_out) continue;
      const int entry = list[done + col];
      if (MODE == FEW_GATED) {
        float gate = total(o / 16, 0, o % 16, col), up = total(o / 16, 1, o % 16, col);
        if (in_wts && routed) {
          const float wt = in_wts[(size_t)(entry / slots) * top + entry % slots];
          gate *= wt;
          up *= wt;
        }
        gate = fminf(gate, lim);
        up = fminf(fmaxf(up, -lim), lim);
        y[(size_t)entry * ffmax + f] = from_f32<bf16>(gate / (1.0f + expf(-alpha * gate)) * (up + shift));
      } else {
        const float v = total(o / 32, o / 16 % 2, o % 16, col);
        if (MODE == FEW_PLAIN) {
          y[(size_t)entry * ffmax + f] = from_f32<bf16>(plain_act(v, act));
        } else {
          const int t = entry / slots;
          rows[(size_t)entry * width + f] = v * (routed ? (wts ? wts[(size_t)t * top + entry % slots] : 1.f) : sg[t]);
        }
      }
    }
  }
}

// Steps that moe_few_kernel takes: bfloat16 rows in whole blocks of 32 dims from 16-byte boundaries (other steps go token by
// token).
static int few_blocks(int E, int ntok, int top) { return E < ntok * top ? E : ntok * top; }
static bool few_usable(int dtype, int E, int ntok, int top, int n_in, int n_shared, long long ldx, const void* x, const void* w, const void* ws) {
  return dtype == GB_BF16 && E > 0 && E < 65535 && ntok <= FEW_LIST / top && n_in % 32 == 0 && (!ws || n_shared % 32 == 0) && ldx % 8 == 0 &&
         !(((uintptr_t)x | (uintptr_t)w | (uintptr_t)ws) & 15);
}

__global__ void __launch_bounds__(256) moe_sum_kernel(const float* __restrict__ rows, float* __restrict__ residual,
                                                      long long ldr, int width, int slots,
                                                      const float* __restrict__ col_scale, int store) {
  pdl_release_next();
  pdl_wait_prior();
  const int t = blockIdx.x;
  for (int n = blockIdx.y * 256 + threadIdx.x; n < width; n += gridDim.y * 256) {
    float total = 0.f;
#pragma unroll 8
    for (int s = 0; s < slots; ++s) total += rows[((size_t)t * slots + s) * width + n];
    if (col_scale) total *= col_scale[n];
    residual[(size_t)t * ldr + n] = store ? total : residual[(size_t)t * ldr + n] + total;
  }
}

GB_EXPORT int gb_moe_topk_mode(const float* z, long long ldz, const float* bias, int* idx, float* wts, float* sg, int ntok,
                               int E, int top, int has_gate, int mode, float scale, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  if (mode < ROUTE_SOFTMAX_TOP || mode > ROUTE_SIGMOID_RAW) return GB_ERR_ARG;
  if (E <= 0 || top <= 0 || top > 32 || top > E || E > 2048) return GB_ERR_SIZE;
  gb_launch(moe_topk_kernel, dim3((ntok + 3) / 4), dim3(128), (size_t)4 * E * sizeof(float), stream, z, ldz, bias, idx, wts, sg,
            ntok, E, top, has_gate, mode, scale);
  return gb_launch_status();
}

GB_EXPORT int gb_moe_topk(const float* z, long long ldz, const float* bias, int* idx, float* wts, float* sg, int ntok,
                          int E, int top, int has_gate, cudaStream_t stream) {
  return gb_moe_topk_mode(z, ldz, bias, idx, wts, sg, ntok, E, top, has_gate, ROUTE_SOFTMAX_TOP, 1.0f, stream);
}

// w_gu: [E, 2 ff, width] (an expert's gate rows, then its up rows); ws_gu: [2 ffs, width] or null;
// y: [ntok, slots, ffmax], slots = top (+ 1 with a shared expert), ffmax = max(ff, ffs).  in_wts: float32
// [ntok, top], factors on the routed experts' inputs, or null.  E: how many experts there are.
GB_EXPORT int gb_moe_gate_up(const void* h, long long ldh, int dtype, const int* idx, const void* w_gu, const void* ws_gu,
                             void* y, int ntok, int E, int width, int ff, int ffs, int top, float limit, float limit_s,
                             float alpha, float shift, const float* in_wts, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  const int slots = top + (ws_gu ? 1 : 0), ffmax = ff > ffs ? ff : ffs;
  if (width <= 0 || ffmax <= 0 || slots <= 0) return GB_ERR_SIZE;
  const size_t smem = (size_t)width * sizeof(float);
  if (smem > 48 * 1024) return GB_ERR_SIZE;
  if (few_usable(dtype, E, ntok, top, width, width, ldh, h, w_gu, ws_gu)) {
    gb_launch(moe_few_kernel<FEW_GATED>, dim3(few_blocks(E, ntok, top) + slots - top, (ffmax + 16 * FEW_RUNS - 1) / (16 * FEW_RUNS)), dim3(256), 0, stream,
              (const bf16*)h, ldh, idx, (const bf16*)w_gu, (const bf16*)ws_gu, (bf16*)y, (float*)nullptr, ntok, width, ff, ffs, ffmax,
              top, slots, limit, limit_s, alpha, shift, 0, in_wts, (const float*)nullptr, (const float*)nullptr, (int)(ntok * top < E));
    return gb_launch_status();
  }
  dim3 grid(ntok * slots, (ffmax + FEATS - 1) / FEATS);
  if (dtype == GB_F32)
    gb_launch(moe_gate_up_kernel<float>, grid, dim3(256), smem, stream, (const float*)h, ldh, idx, (const float*)w_gu,
              (const float*)ws_gu, (float*)y, width, ff, ffs, ffmax, top, slots, limit, limit_s, alpha, shift, in_wts);
  else if (dtype == GB_BF16)
    gb_launch(moe_gate_up_kernel<bf16>, grid, dim3(256), smem, stream, (const bf16*)h, ldh, idx, (const bf16*)w_gu,
              (const bf16*)ws_gu, (bf16*)y, width, ff, ffs, ffmax, top, slots, limit, limit_s, alpha, shift, in_wts);
  else
    return GB_ERR_DTYPE;
  return gb_launch_status();
}

// Experts without a gate: w_up [E, ff, width]; y: [ntok, top, ff] = act(up h) of every chosen expert.
GB_EXPORT int gb_moe_up(const void* h, long long ldh, int dtype, const int* idx, const void* w_up, void* y, int ntok, int E, int width,
                        int ff, int top, int act, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  if (act != ACT_GELU && act != ACT_RELU2) return GB_ERR_ARG;
  if (width <= 0 || ff <= 0 || top <= 0) return GB_ERR_SIZE;
  const size_t smem = (size_t)width * sizeof(float);
  if (smem > 48 * 1024) return GB_ERR_SIZE;
  if (few_usable(dtype, E, ntok, top, width, width, ldh, h, w_up, nullptr)) {
    gb_launch(moe_few_kernel<FEW_PLAIN>, dim3(few_blocks(E, ntok, top), (ff + 32 * FEW_RUNS - 1) / (32 * FEW_RUNS)), dim3(256), 0, stream, (const bf16*)h, ldh, idx,
              (const bf16*)w_up, (const bf16*)nullptr, (bf16*)y, (float*)nullptr, ntok, width, ff, 0, ff, top, top, 0.f, 0.f, 0.f, 0.f,
              act, (const float*)nullptr, (const float*)nullptr, (const float*)nullptr, (int)(ntok * top < E));
    return gb_launch_status();
  }
  dim3 grid(ntok * top, (ff + FEATS - 1) / FEATS);
  if (dtype == GB_F32)
    gb_launch(moe_up_kernel<float>, grid, dim3(256), smem, stream, (const float*)h, ldh, idx, (const float*)w_up, (float*)y,
              width, ff, top, act);
  else if (dtype == GB_BF16)
    gb_launch(moe_up_kernel<bf16>, grid, dim3(256), smem, stream, (const bf16*)h, ldh, idx, (const bf16*)w_up, (bf16*)y, width,
              ff, top, act);
  else
    return GB_ERR_DTYPE;
  return gb_launch_status();
}

// w_d: [E, width, ff]; ws_d: [width, ffs] or null; rows: float32 scratch [ntok, slots, width];
// residual: float32 [ntok, width] rows ldr apart, added to, or with `store` written.  wts: null: ones.
GB_EXPORT int gb_moe_down(const void* y, int dtype, const int* idx, const float* wts, const float* sg, const void* w_d,
                          const void* ws_d, float* rows, float* residual, long long ldr, int ntok, int E, int width, int ff, int ffs,
                          int top, const float* col_scale, int store, cudaStream_t stream) {
  if (ntok <= 0) return 0;
  const int slots = top + (ws_d ? 1 : 0), ffmax = ff > ffs ? ff : ffs;
  if (width <= 0 || ffmax <= 0 || slots <= 0) return GB_ERR_SIZE;
  const size_t smem = (size_t)ffmax * sizeof(float);
  if (smem > 48 * 1024) return GB_ERR_SIZE;
  dim3 grid(ntok * slots, (width + FEATS - 1) / FEATS);
  if (few_usable(dtype, E, ntok, top, ff, ffs, ffmax, y, w_d, ws_d))
    gb_launch(moe_few_kernel<FEW_DOWN>, dim3(few_blocks(E, ntok, top) + slots - top, (width + 32 * FEW_RUNS - 1) / (32 * FEW_RUNS)), dim3(256), 0, stream,
              (const bf16*)y, (long long)ffmax, idx, (const bf16*)w_d, (const bf16*)ws_d, (bf16*)nullptr, rows, ntok, width, ff, ffs,
              ffmax, top, slots, 0.f, 0.f, 0.f, 0.f, 0, (const float*)nullptr, wts, sg, (int)(ntok * top < E));
  else if (dtype == GB_F32)
    gb_launch(moe_down_kernel<float>, grid, dim3(256), smem, stream, (const float*)y, idx, wts, sg, (const float*)w_d,
              (const float*)ws_d, rows, width, ff, ffs, ffmax, top, slots);
  else if (dtype == GB_BF16)
    gb_launch(moe_down_kernel<bf16>, grid, dim3(256), smem, stream, (const bf16*)y, idx, wts, sg, (const bf16*)w_d,
              (const bf16*)ws_d, rows, width, ff, ffs, ffmax, top, slots);
  else
    return GB_ERR_DTYPE;
  gb_launch(moe_sum_kernel, dim3(ntok, (width + 255) / 256), dim3(256), 0, stream, (const float*)rows, residual, ldr, width,
            slots, col_scale, store);
  return gb_launch_status();
}
