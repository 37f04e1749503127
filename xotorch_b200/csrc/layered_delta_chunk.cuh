// layered_delta_chunk.cuh — the delta-rule recurrences over prompts, DCH = 32 tokens at a time.
//
// delta_rule_kernel (layered_kernels.cuh) walks the tokens one by one, so a prompt of one request is a chain of dot product, sum over lanes and update per
// token, on heads x column groups of the chip: 0.14 us a token (64 x 64 heads), 0.35 us (128 x 128), whatever else the chip could do.  Within a chunk the chain is
// a triangular system of numbers that do not depend on the state, so it is solved for all chunks at once by one kernel, and what is left to walk are the chunks.
// With S the state in front of the chunk and everything fp32:
//   gated form     G(t,s) = prod_{s < i <= t} g_i,  A(t,s) = beta_t G(t,s) k_t.k_s (s < t),  T = (I + A)^-1,  P(t,s) = G(t,s) r_t.k_s (s <= t)
//                  c = T (beta_t (v_t - G(t,0) S^T k_t)),   o_t = G(t,0) S^T r_t + P c,   S <- G(C,0) S + sum_s G(C,s) k_s c_s^T
//   general form   D_t = prod_{i <= t} diag(w_i),  u~_t = D_{t-1} u_t, r~_t = D_t r_t, k~_s = D_s^-1 k_s, a~_s = D_s^-1 (a u)_s,  B = u~ k~ (s < t), A = u~ a~ (s < t),
//                  T = (I + A)^-1, P1 = r~ k~, P2 = - r~ a~ (s <= t)
//                  c = T (S^T u~ + B v),   o = S^T r~ + P1 v + P2 c,   S <- D_C S + sum_s (D_C k~_s) v_s^T - (D_C a~_s) c_s^T
// The gated form's decays may be as small as they like: products of them are formed factor by factor and nothing is divided by one.  The general form's
// decays are exp(-exp(-1/2) sigmoid(.)) >= 0.545, so D over 32 tokens stays above 3.7e-9 and its reciprocal is harmless.  T's entries are the
// influence of one token's value on a later correction, which the recurrence itself contracts: at most about 1.
// Rows behind the end of a request's step count as tokens that neither decay nor write.
// Measured (B200, a launch): 3500 tokens, 32 heads of 64 x 64 (16 key heads), gated: 495 us token by token -> 31 (matrices) + 295 (walk); 1024 tokens, 32 heads of 128 x 128, general:
// 365 + 24 for its vectors -> 74 + 248.  The walk is bound by shared memory (wavefronts at 61 to 62 % of their rate on the SMs that have a block) and by the latency of its three steps a chunk (2.7 us, 7.8 us).
#pragma once
#include "layered_stream.cuh"

namespace xl {

constexpr int DCH = 32, DCH_THREADS = 256, DCH_LD = DCH + 4;   // tokens of a chunk; row stride of a 32-wide matrix in shared memory

__device__ __forceinline__ void cp_async16_or_zero(float* dst_smem, const float* src, bool on) {   // 16 bytes, or zeros (src is not read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4_or_zero(float* dst_smem, const float* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src), "r"(on ? 4 : 0) : "memory");
}
// chunks of request i of a step: from row0 / 32 + i on (no two requests share one)
__device__ __host__ __forceinline__ int dch_first(int row0, int i) { return row0 / DCH + i; }
__device__ __forceinline__ float dot2(f32x2 v) { const float2 p = unpack2(v); return p.x + p.y; }

struct DeltaChunkArgs {
  int H, rep, dk, dv;                                  // rep: value heads per key head (general form: 1)
  // sources [M, ld]: gated form: unit keys, scaled queries (ld = H / rep * dk); general form: projection columns
  const float *k, *r, *v;
  int k_ld, k_col, r_ld, r_col, v_ld, v_col;
  const float *g, *beta;                               // gated form: [M, H]
  // general form: removal logits in the projection, decay logits [M, H * dk], their biases
  const float *a, *wlog;
  int a_ld, a_col;
  const void *a_bias, *w_bias;
  // between the two kernels.  mats: per (chunk, head) T, P (general: T, P2, B, P1) of 32 x 32; vecs: gated: beta, G(t,0), G(C,t) of 32; general: D_C of dk
  float *mats, *vecs;
  float *x1, *x2, *y1, *y2;                            // general form: u~, r~, D_C k~, -D_C a~, [M, H * dk]
  float* state;                                        // this layer's part of slot 0
  size_t slot_stride;
  float* o;                                            // [M, H * dv]
};
__host__ __device__ constexpr int dch_mats(bool gated) { return (gated ? 2 : 4) * DCH * DCH; }
__host__ __device__ constexpr int dch_vecs(bool gated, int dk) { return gated ? 3 * DCH : dk; }

// column `lane` of (I + A)^-1 for a strictly lower triangular A (rows of stride DCH_LD, 16-byte aligned), by one warp
__device__ __forceinline__ void dch_inverse(const float* A, float (&c)[DCH], int lane) {
#pragma unroll
  for (int t = 0; t < DCH; ++t) {
    float s0 = lane == t ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
    for (int s = 0; s < t; s += 4) {
      const float4 x = *reinterpret_cast<const float4*>(A + t * DCH_LD + s);
      s0 = fmaf(-x.x, c[s], s0);
      if (s + 1 < t) s1 = fmaf(-x.y, c[s + 1], s1);
      if (s + 2 < t) s0 = fmaf(-x.z, c[s + 2], s0);
      if (s + 3 < t) s1 = fmaf(-x.w, c[s + 3], s1);
    }
    c[t] = s0 + s1;
  }
}

// acc(r, c) += sum_i X[r][i] Y[c][i] over i = i0, i0 + STEP, ... (four at a time) for rows r = rg + RG j and columns c = cg + CG n; X, Y of row strides LX, LY
template <int R, int C, int RG, int CG, int K, int STEP, int LX, int LY>
__device__ __forceinline__ void dch_tile(const float* X, const float* Y, int rg, int cg, int i0, f32x2 (&acc)[R][C]) {
#pragma unroll 2
  for (int i = i0; i < K; i += STEP) {
    ulonglong2 x[R], y[C];
#pragma unroll
    for (int j = 0; j < R; ++j) x[j] = *reinterpret_cast<const ulonglong2*>(X + (rg + RG * j) * LX + i);
#pragma unroll
    for (int n = 0; n < C; ++n) y[n] = *reinterpret_cast<const ulonglong2*>(Y + (cg + CG * n) * LY + i);
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int n = 0; n < C; ++n) {
        acc[j][n] = fma2(x[j].x, y[n].x, acc[j][n]);
        acc[j][n] = fma2(x[j].y, y[n].y, acc[j][n]);
      }
  }
}

// ---- the chunks' matrices, gated form.  grid (chunks of the longest request, requests, key heads), 128 threads; a warp per value head at the end
template <int DK> __host__ __device__ constexpr int dch_gated_smem() { return (2 * DCH * (DK + 4) + 6 * DCH * DCH_LD) * 4; }
template <int DK>
__global__ void __launch_bounds__(128) delta_chunk_gated_kernel(const DeltaChunkArgs a, const Item* __restrict__ seqs) {
  pdl_enter();
  constexpr int LD = DK + 4;
  extern __shared__ __align__(16) float dch_sm[];
  float* x = dch_sm;                                   // keys, queries [2 * DCH][LD]
  float *G1 = x + 2 * DCH * LD, *G2 = G1 + DCH * DCH_LD;   // keys . keys, queries . keys [DCH][DCH_LD]
  float* A = G2 + DCH * DCH_LD + (threadIdx.x >> 5) * DCH * DCH_LD;   // [DCH][DCH_LD] per warp
  const Item sq = seqs[blockIdx.y];
  const int c = blockIdx.x, t0 = c * DCH, kh = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (t0 >= sq.n_rows) return;
  const int n = min(DCH, sq.n_rows - t0);
  for (int e = tid; e < 2 * DCH * (DK / 4); e += 128) {
    const int row = e / (DK / 4), i = e % (DK / 4) * 4, t = row % DCH;
    const bool on = t < n && i < a.dk;
    const float* src = row < DCH ? a.k + (size_t)(sq.row0 + t0 + t) * a.k_ld + a.k_col : a.r + (size_t)(sq.row0 + t0 + t) * a.r_ld + a.r_col;
    cp_async16_or_zero(x + row * LD + i, on ? src + kh * a.dk + i : a.k, on);
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    f32x2 acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int m = 0; m < 4; ++m) acc[j][m] = 0;
    const int cg = tid % 8, rg = tid / 8;              // rows rg + 16 j of [keys; queries], columns cg + 8 m
    dch_tile<4, 4, 16, 8, DK, 4, LD, LD>(x, x, rg, cg, 0, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int m = 0; m < 4; ++m) (j < 2 ? G1 : G2)[(rg + 16 * j) % DCH * DCH_LD + cg + 8 * m] = dot2(acc[j][m]);
  }
  __syncthreads();
  for (int q = warp; q < a.rep; q += 4) {
    const int h = kh * a.rep + q;
    const size_t at = (size_t)(dch_first(sq.row0, blockIdx.y) + c) * a.H + h;
    float* T = a.mats + at * dch_mats(true);
    float* P = T + DCH * DCH;
    float* vec = a.vecs + at * dch_vecs(true, 0);
    const size_t row = (size_t)sq.row0 + t0 + lane;
    const float gl = lane < n ? a.g[row * a.H + h] : 1.f, bl = lane < n ? a.beta[row * a.H + h] : 0.f;
    float p = 0.f, p0 = 1.f;                           // G(t, lane), G(t, 0)
    for (int t = 0; t < DCH; ++t) {
      const float gt = __shfl_sync(0xffffffffu, gl, t), bt = __shfl_sync(0xffffffffu, bl, t);
      p0 *= gt;
      p = t == lane ? 1.f : p * gt;
      A[t * DCH_LD + lane] = t > lane ? bt * p * G1[t * DCH_LD + lane] : 0.f;
      P[t * DCH + lane] = t >= lane ? p * G2[t * DCH_LD + lane] : 0.f;
      if (lane == t) vec[DCH + t] = p0;
    }
    vec[lane] = bl;
    vec[2 * DCH + lane] = p;
    __syncwarp();
    float col[DCH];
    dch_inverse(A, col, lane);
#pragma unroll
    for (int t = 0; t < DCH; ++t) T[t * DCH + lane] = col[t];
    __syncwarp();
  }
}

// ---- the chunks' matrices and scaled vectors, general form.  grid (chunks of the longest request, requests, heads), 256 threads
template <int DK> __host__ __device__ constexpr int dch_general_smem() { return (5 * DCH * (DK + 4) + DCH * DCH_LD) * 4; }
template <typename T, int DK>
__global__ void __launch_bounds__(DCH_THREADS) delta_chunk_general_kernel(const DeltaChunkArgs a, const Item* __restrict__ seqs) {
  pdl_enter();
  constexpr int LD = DK + 4;
  extern __shared__ __align__(16) float dch_sm[];
  float* X = dch_sm;                                   // u~, r~ [2 * DCH][LD]
  float* Y = X + 2 * DCH * LD;                         // k~, a~ [2 * DCH][LD]
  float* W = Y + 2 * DCH * LD;                         // decays, then D_t [DCH][LD]
  float* A = W + DCH * LD;                             // [DCH][DCH_LD]
  const Item sq = seqs[blockIdx.y];
  const int c = blockIdx.x, t0 = c * DCH, h = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (t0 >= sq.n_rows) return;
  const int n = min(DCH, sq.n_rows - t0), HD = a.H * a.dk;
  const T *ab = static_cast<const T*>(a.a_bias) + h * a.dk, *wb = static_cast<const T*>(a.w_bias) + h * a.dk;
  // a warp per row, four entries a lane: unit key, its removal strength, decay; the loads of two rows under way together
  const int i4 = lane * 4;
  const bool has = i4 < a.dk, pad = i4 < DK;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 abv = has ? make_float4(ldf(ab + i4), ldf(ab + i4 + 1), ldf(ab + i4 + 2), ldf(ab + i4 + 3)) : zero;
  const float4 wbv = has ? make_float4(ldf(wb + i4), ldf(wb + i4 + 1), ldf(wb + i4 + 2), ldf(wb + i4 + 3)) : zero;
#pragma unroll 2
  for (int t = warp; t < DCH; t += DCH_THREADS / 32) {
    const bool in = t < n && has;
    const size_t m = (size_t)sq.row0 + t0 + (t < n ? t : 0);
    const float4 k = in ? ld4f(a.k + m * a.k_ld + a.k_col + h * a.dk + i4) : zero, r = in ? ld4f(a.r + m * a.r_ld + a.r_col + h * a.dk + i4) : zero;
    const float4 al = in ? ld4f(a.a + m * a.a_ld + a.a_col + h * a.dk + i4) : zero, wl = in ? ld4f(a.wlog + m * HD + h * a.dk + i4) : zero;
    const float inv = 1.0f / sqrtf(warp_sum(sq4(k)) + 1e-6f);
    const float4 u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
    auto decay = [](float x) { return expf(-0.60653065971263342f * sigmoidf_(x)); };
    if (pad) {
      st4f(X + t * LD + i4, u);
      st4f(X + (DCH + t) * LD + i4, r);
      st4f(Y + t * LD + i4, k);
      st4f(Y + (DCH + t) * LD + i4, in ? make_float4(sigmoidf_(al.x + abv.x) * u.x, sigmoidf_(al.y + abv.y) * u.y, sigmoidf_(al.z + abv.z) * u.z, sigmoidf_(al.w + abv.w) * u.w) : zero);
      st4f(W + t * LD + i4, in ? make_float4(decay(wl.x + wbv.x), decay(wl.y + wbv.y), decay(wl.z + wbv.z), decay(wl.w + wbv.w)) : make_float4(1.f, 1.f, 1.f, 1.f));
    }
  }
  __syncthreads();
  // the products of the decays down the chunk, one thread per channel
  if (tid < DK) {
    float d = 1.f;
#pragma unroll 8
    for (int t = 0; t < DCH; ++t) { d *= W[t * LD + tid]; W[t * LD + tid] = d; }
    if (tid < a.dk) a.vecs[((size_t)(dch_first(sq.row0, blockIdx.y) + c) * a.H + h) * dch_vecs(false, a.dk) + tid] = d;
  }
  __syncthreads();
#pragma unroll 2
  for (int t = warp; t < DCH; t += DCH_THREADS / 32) {
    if (!pad) continue;
    const float4 d = ld4f(W + t * LD + i4), before = t ? ld4f(W + (t - 1) * LD + i4) : make_float4(1.f, 1.f, 1.f, 1.f), whole = ld4f(W + (DCH - 1) * LD + i4);
    const float4 inv = make_float4(1.0f / d.x, 1.0f / d.y, 1.0f / d.z, 1.0f / d.w);
    auto mul = [](float4 x, float4 y) { return make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w); };
    const float4 u = mul(ld4f(X + t * LD + i4), before), r = mul(ld4f(X + (DCH + t) * LD + i4), d), k = mul(ld4f(Y + t * LD + i4), inv), au = mul(ld4f(Y + (DCH + t) * LD + i4), inv);
    st4f(X + t * LD + i4, u);
    st4f(X + (DCH + t) * LD + i4, r);
    st4f(Y + t * LD + i4, k);
    st4f(Y + (DCH + t) * LD + i4, au);
    if (t < n && has) {
      const size_t o = ((size_t)sq.row0 + t0 + t) * HD + h * a.dk + i4;
      st4f(a.x1 + o, u);
      st4f(a.x2 + o, r);
      st4f(a.y1 + o, mul(k, whole));
      const float4 w = mul(au, whole);
      st4f(a.y2 + o, make_float4(-w.x, -w.y, -w.z, -w.w));
    }
  }
  __syncthreads();
  float* mats = a.mats + ((size_t)(dch_first(sq.row0, blockIdx.y) + c) * a.H + h) * dch_mats(false);   // T, P2, B, P1
  {
    f32x2 acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int m = 0; m < 4; ++m) acc[j][m] = 0;
    const int cg = tid % 16, rg = tid / 16;            // rows rg + 16 j of [u~; r~], columns cg + 16 m of [k~; a~]
    dch_tile<4, 4, 16, 16, DK, 4, LD, LD>(X, Y, rg, cg, 0, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int t = (rg + 16 * j) % DCH, s = (cg + 16 * m) % DCH;
        const float v = dot2(acc[j][m]);
        if (j < 2 && m < 2) mats[2 * DCH * DCH + t * DCH + s] = s < t ? v : 0.f;
        else if (j < 2) A[t * DCH_LD + s] = s < t ? v : 0.f;
        else if (m < 2) mats[3 * DCH * DCH + t * DCH + s] = s <= t ? v : 0.f;
        else mats[DCH * DCH + t * DCH + s] = s <= t ? -v : 0.f;
      }
  }
  __syncthreads();
  if (warp == 0) {
    float col[DCH];
    dch_inverse(A, col, lane);
#pragma unroll
    for (int t = 0; t < DCH; ++t) mats[t * DCH + lane] = col[t];
  }
}

// ---- what a prompt of the gated form needs per token, in one pass over the projection: the channels' convolution (its window in registers), silu, unit key, scaled
// query, values (at v [M, C], the value channels' place), decay and write strength.  LPH lanes have the 4 LPH channels of one query, key or value head (dk = dv) and
// walk a stretch of rows; grid (requests, groups of heads, stretches).  Stretch 0 reads the window that the slot keeps and moves it on.  Up to four taps.
// 3500 rows of 4096 channels: 65 us (convolution) + 37 (unit vectors, decays) -> 36.
struct GatedConvArgs {
  const float* proj;
  int ld, col_c, C, taps, col_b, col_a, H, G;
  const void *conv_w, *a_log, *dt_bias;
  float* window;
  size_t slot_stride;
  float *g, *beta, *k, *r, *v;
};
template <typename T, int LPH>
__global__ void __launch_bounds__(256) gated_conv_prepare_kernel(const GatedConvArgs a, const Item* __restrict__ seqs) {
  pdl_enter();
  constexpr int DK = 4 * LPH, W = 4, NB = 4;           // taps at most, rows whose loads are in flight
  const Item sq = seqs[blockIdx.x];
  const int l = threadIdx.x % LPH, vec = blockIdx.y * (256 / LPH) + threadIdx.x / LPH, c = vec * DK + 4 * l;
  const int per = max((sq.n_rows + (int)gridDim.z - 1) / (int)gridDim.z, W - 1);
  const int t_begin = blockIdx.z * per, t_end = min(sq.n_rows, t_begin + per), skip = W - a.taps;
  if (t_begin >= t_end) return;
  const bool on = vec < 2 * a.G + a.H;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* src = a.proj + (size_t)sq.row0 * a.ld + a.col_c + (on ? c : 0);
  float* st = a.window + (size_t)sq.slot * a.slot_stride + (on ? c : 0);
  float w[W][4];
  float4 win[W - 1], first[W - 1];                     // inputs of the three rows in front; the same at the stretch's begin
#pragma unroll
  for (int i = 0; i < W; ++i)
#pragma unroll
    for (int x = 0; x < 4; ++x) w[i][x] = on && i >= skip ? ldf(static_cast<const T*>(a.conv_w) + (size_t)(c + x) * a.taps + i - skip) : 0.f;
#pragma unroll
  for (int i = 0; i < W - 1; ++i) {
    const int t = t_begin - (W - 1) + i;
    first[i] = win[i] = !on || i < skip ? zero : t >= 0 ? ld4f(src + (size_t)t * a.ld) : ld4f(st + (size_t)(t + a.taps - 1) * a.C);
  }
  const float qs = vec < a.G ? sqrtf((float)DK) : 1.0f;
  float* dst = vec < a.G ? a.r + (size_t)sq.row0 * (a.G * DK) + c : vec < 2 * a.G ? a.k + (size_t)sq.row0 * (a.G * DK) + c - a.G * DK : a.v + (size_t)sq.row0 * a.C + c;
  const int ld_dst = vec < 2 * a.G ? a.G * DK : a.C;
  for (int t0 = t_begin; t0 < t_end; t0 += NB) {
    float4 cur[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) cur[b] = on && t0 + b < t_end ? ld4f(src + (size_t)(t0 + b) * a.ld) : zero;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float4 acc = zero;
#pragma unroll
      for (int i = 0; i < W; ++i) {
        if (i < skip) continue;
        const float4 in = i == W - 1 ? cur[b] : win[i < W - 1 ? i : 0];
        acc = make_float4(fmaf(w[i][0], in.x, acc.x), fmaf(w[i][1], in.y, acc.y), fmaf(w[i][2], in.z, acc.z), fmaf(w[i][3], in.w, acc.w));
      }
#pragma unroll
      for (int i = 0; i + 1 < W - 1; ++i) win[i] = win[i + 1];
      win[W - 2] = cur[b];
      acc = make_float4(siluf_(acc.x), siluf_(acc.y), siluf_(acc.z), siluf_(acc.w));
      float s = sq4(acc);
#pragma unroll
      for (int x = LPH / 2; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      const float f = vec < 2 * a.G ? 1.0f / (sqrtf(s + 1e-6f) * qs) : 1.0f;
      if (on && t0 + b < t_end) st4f(dst + (size_t)(t0 + b) * ld_dst, make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f));
    }
  }
  if (!on) return;
  if (vec >= 2 * a.G) {
    const int h = vec - 2 * a.G;
    const float al = expf(ldf(static_cast<const T*>(a.a_log) + h)), db = ldf(static_cast<const T*>(a.dt_bias) + h);
    for (int t = t_begin + l; t < t_end; t += LPH) {
      const size_t m = (size_t)sq.row0 + t;
      a.beta[m * a.H + h] = sigmoidf_(a.proj[m * a.ld + a.col_b + h]);
      a.g[m * a.H + h] = expf(-al * softplusf_(a.proj[m * a.ld + a.col_a + h] + db));
    }
  }
  if (blockIdx.z == 0)
#pragma unroll
    for (int i = 0; i < W - 1; ++i) {
      if (i < skip) continue;
      const int t = sq.n_rows - (W - 1) + i;           // the row whose input entry i - skip of the window becomes
      float4 v = zero;
      if (t >= 0) v = ld4f(src + (size_t)t * a.ld);
#pragma unroll
      for (int x = 0; x < W - 1; ++x)
        if (t < 0 && x == t + W - 1) v = first[x];
      st4f(st + (size_t)(i - skip) * a.C, v);
    }
}

// ---- the walk over the chunks.  One CTA of THR threads per (request, head, NC value columns); S^T, and everything a chunk needs, in shared memory, the next chunk on its
// way.  A 16-byte load of a warp takes four turns of shared memory, shared addresses or not, so every product is cut into tiles of 4 x 4 to 8 x 8 results whose K
// is shared by four lanes: two loads feed 2 to 4 times as many sums as with a 2 x 2 tile per thread (349 -> 295 us for 3500 tokens), and shuffles add the lanes' parts.
// DCH_KS lanes that share a tile; rows that two tiles of a quarter warp read at once lie 16 banks apart (strides DCH_CL, LS).
constexpr int DCH_KS = 4, DCH_CL = DCH + 16;
// sums over the four lanes kq = 0 .. 3 (neighbours O apart) of R x C partial results, C = 4 m: lane kq gets columns kq m .. kq m + m - 1 in f[.][0 .. m - 1]
template <int R, int C, int O>
__device__ __forceinline__ void dch_share(float (&f)[R][C], int kq) {
#pragma unroll
  for (int half = C / 2, o = 2; o > 0; half >>= 1, o >>= 1) {
    const bool up = kq & o;
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int n = 0; n < C / 2; ++n)
        if (n < half) {
          const float keep = up ? f[j][n + half] : f[j][n], give = up ? f[j][n] : f[j][n + half];
          f[j][n] = keep + __shfl_xor_sync(0xffffffffu, give, o * O);
        }
  }
}
template <int DK, int NC, bool GATED>
struct DeltaWalk {
  static constexpr int LD = DK + 4, LS = DK + 16, NX = 2 * DCH * LD, NY = GATED ? 0 : 2 * DCH * LD, NM = (GATED ? 2 : 4) * DCH * DCH_LD, NV = NC * DCH_CL, NVEC = GATED ? 3 * DCH : DK,
                       STAGE = NX + NY + NM + NV + NVEC, SMEM = (2 * STAGE + NC * LS + (GATED ? 3 : 2) * NC * DCH_CL) * 4;
};
template <int DK, int NC, bool GATED, int THR>
__global__ void __launch_bounds__(THR, 256 / THR) delta_chunk_walk_kernel(const DeltaChunkArgs a, const Item* __restrict__ seqs) {
  pdl_enter();
  typedef DeltaWalk<DK, NC, GATED> L;
  constexpr int LD = L::LD, LS = L::LS;
  extern __shared__ __align__(16) float dch_sm[];
  float* St = dch_sm + 2 * L::STAGE;                   // [NC][LS]
  float *zt = St + NC * LS, *ct = zt + NC * DCH_CL, *cs = GATED ? ct + NC * DCH_CL : ct;   // [NC][DCH_CL]: right sides, corrections, corrections as they enter the state
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x % a.H, req = blockIdx.x / a.H, col0 = blockIdx.y * NC, HD = a.H * a.dk;
  const Item sq = seqs[req];
  const int nch = (sq.n_rows + DCH - 1) / DCH, kh = h / a.rep;
  for (int e = tid; e < 2 * L::STAGE + NC * LS; e += THR) dch_sm[e] = 0.f;   // padding (key rows beyond dk) stays zero
  __syncthreads();
  // chunk c into stage c & 1
  const int q4 = a.dk / 4;
  const float* xs = GATED ? a.k + a.k_col + kh * a.dk : a.x1 + h * a.dk;
  const float* xr = GATED ? a.r + a.r_col + kh * a.dk : a.x2 + h * a.dk;
  const int ldk = GATED ? a.k_ld : HD, ldr = GATED ? a.r_ld : HD;
  auto issue = [&](int c) {
    float* X = dch_sm + (c & 1) * L::STAGE;
    const int t0 = c * DCH, n = min(DCH, sq.n_rows - t0);
    const size_t m0 = (size_t)sq.row0 + t0;
    constexpr int TPP = THR / (DK / 4);                // rows that one pass of the threads covers
    const int i = tid % (DK / 4), tf = tid / (DK / 4);
    if (i < q4)
#pragma unroll
      for (int t = tf; t < DCH; t += TPP) {
        const bool on = t < n;
        const size_t m = m0 + (on ? t : 0);
        cp_async16_or_zero(X + t * LD + 4 * i, xs + m * ldk + 4 * i, on);
        cp_async16_or_zero(X + (DCH + t) * LD + 4 * i, xr + m * ldr + 4 * i, on);
        if constexpr (!GATED) {
          cp_async16_or_zero(X + L::NX + t * LD + 4 * i, a.y1 + m * HD + h * a.dk + 4 * i, on);
          cp_async16_or_zero(X + L::NX + (DCH + t) * LD + 4 * i, a.y2 + m * HD + h * a.dk + 4 * i, on);
        }
      }
    const size_t at = (size_t)(dch_first(sq.row0, req) + c) * a.H + h;
    const float* mats = a.mats + at * dch_mats(GATED);
    float* M = X + L::NX + L::NY;
#pragma unroll
    for (int e = tid; e < (GATED ? 2 : 4) * DCH * (DCH / 4); e += THR) cp_async16(M + e / (DCH / 4) * DCH_LD + e % (DCH / 4) * 4, mats + 4 * e);
    float* V = M + L::NM;
#pragma unroll
    for (int e = tid; e < DCH * NC; e += THR) {
      const int t = e / NC, cc = e % NC;
      const bool on = t < n && col0 + cc < a.dv;
      cp_async4_or_zero(V + cc * DCH_CL + t, on ? a.v + (m0 + t) * a.v_ld + a.v_col + h * a.dv + col0 + cc : a.v, on);
    }
    const float* vec = a.vecs + at * dch_vecs(GATED, a.dk);
    if (tid < dch_vecs(GATED, a.dk) / 4) cp_async16(V + L::NV + 4 * tid, vec + 4 * tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(0);
  // the state: a tile is four key rows from 4 ig on (DK = 128: and four from 64 + 4 ig on) of CS columns cgp + CGN n; of its columns lane kqs keeps n = kqs CK .. kqs CK + CK - 1
  constexpr int IP = DK / 64, CGN = THR / 64, CS = NC / CGN, CK = CS / 4;   // a pair of warps per column group: 16 tiles of rows x 4 lanes
  static_assert(CGN * 64 == THR && CK >= 1 && CK * 4 * CGN == NC && IP * 64 == DK, "the threads cover the state, each part once");
  const int ig = (warp & 1) * 8 + (lane & 7), cgp = warp >> 1, kqs = lane >> 3;
  float* S = a.state + (size_t)sq.slot * a.slot_stride + (size_t)h * a.dk * a.dv;
  float s[4 * IP][CK];
#pragma unroll
  for (int m = 0; m < CK; ++m) {
    const int cc = cgp + CGN * (kqs * CK + m), col = col0 + cc;
#pragma unroll
    for (int p = 0; p < IP; ++p) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = 64 * p + 4 * ig + r;
        s[4 * p + r][m] = i < a.dk && col < a.dv ? S[(size_t)i * a.dv + col] : 0.f;
      }
      *reinterpret_cast<float4*>(St + cc * LS + 64 * p + 4 * ig) = make_float4(s[4 * p][m], s[4 * p + 1][m], s[4 * p + 2][m], s[4 * p + 3][m]);
    }
  }
  // products with a token per row: tokens tr + TR j, columns tc + TC n, of which lane kq keeps n = kq
  constexpr int TC = NC / 4, TR = THR / (DCH_KS * TC), RT = DCH / TR;
  static_assert(RT >= 1 && RT * TR == DCH, "the threads cover a chunk's tokens");
  const int kq = tid % DCH_KS, tc = tid / DCH_KS % TC, tr = tid / (DCH_KS * TC), cc = tc + TC * kq;
  // a 32 x 32 lower triangular matrix of the chunk against 32 numbers per column.  `careful`: a number of the chunk is not finite, and 0 * Inf above the diagonal
  // would carry it to tokens in front of its own
  bool careful = false;
  auto lower = [&](const float* M, const float* cols, float (&out)[RT]) {
    if (!careful) {
      f32x2 acc[RT][4];
#pragma unroll
      for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc[j][n] = 0;
      dch_tile<RT, 4, TR, TC, DCH, 4 * DCH_KS, DCH_LD, DCH_CL>(M, cols, tr, tc, 4 * kq, acc);
      float f[RT][4];
#pragma unroll
      for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int n = 0; n < 4; ++n) f[j][n] = dot2(acc[j][n]);
      dch_share<RT, 4, 1>(f, kq);
#pragma unroll
      for (int j = 0; j < RT; ++j) out[j] += f[j][0];
      return;
    }
#pragma unroll
    for (int j = 0; j < RT; ++j)
      for (int t = 0; t <= tr + TR * j; ++t) out[j] = fmaf(M[(tr + TR * j) * DCH_LD + t], cols[cc * DCH_CL + t], out[j]);
  };
  for (int c = 0; c < nch; ++c) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                   // the chunk is there for all threads, the other stage is free, S^T has been written
    if (c + 1 < nch) issue(c + 1);
    const float* X = dch_sm + (c & 1) * L::STAGE;
    const float *Y = X + L::NX, *M = Y + L::NY, *V = M + L::NM, *vec = V + L::NV;
    // S^T against both vectors of every token
    float y[2 * RT][4];
    {
      f32x2 acc[2 * RT][4];
#pragma unroll
      for (int j = 0; j < 2 * RT; ++j)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc[j][n] = 0;
      dch_tile<2 * RT, 4, TR, TC, DK, 4 * DCH_KS, LD, LS>(X, St, tr, tc, 4 * kq, acc);
#pragma unroll
      for (int j = 0; j < 2 * RT; ++j)
#pragma unroll
        for (int n = 0; n < 4; ++n) y[j][n] = dot2(acc[j][n]);
      dch_share<2 * RT, 4, 1>(y, kq);
    }
    // right sides
    careful = false;
    for (;;) {
      bool bad = false;
      float z[RT];
#pragma unroll
      for (int j = 0; j < RT; ++j) z[j] = 0.f;
      if constexpr (!GATED) lower(M + 2 * DCH * DCH_LD, V, z);
#pragma unroll
      for (int j = 0; j < RT; ++j) {
        const int t = tr + TR * j;
        const float v = GATED ? vec[t] * fmaf(-vec[DCH + t], y[j][0], V[cc * DCH_CL + t]) : y[j][0] + z[j];
        zt[cc * DCH_CL + t] = v;
        bad |= !(fabsf(v) <= 3.402823466e38f);
      }
      const bool any = __syncthreads_or(bad);
      if (!any || careful) break;
      careful = true;
    }
    // corrections
    float f[RT];
#pragma unroll
    for (int j = 0; j < RT; ++j) f[j] = 0.f;
    lower(M, zt, f);
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      const int t = tr + TR * j;
      ct[cc * DCH_CL + t] = f[j];
      if constexpr (GATED) cs[cc * DCH_CL + t] = vec[2 * DCH + t] * f[j];
    }
    __syncthreads();
    // outputs
#pragma unroll
    for (int j = 0; j < RT; ++j) f[j] = 0.f;
    lower(M + DCH * DCH_LD, ct, f);
    if constexpr (!GATED) lower(M + 3 * DCH * DCH_LD, V, f);
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      const int t = tr + TR * j;
      const float d = y[RT + j][0];
      if (c * DCH + t < sq.n_rows && col0 + cc < a.dv)
        a.o[((size_t)sq.row0 + c * DCH + t) * (size_t)(a.H * a.dv) + h * a.dv + col0 + cc] = GATED ? fmaf(vec[DCH + t], d, f[j]) : d + f[j];
    }
    // the state moves on: lane kqs takes tokens 4 kqs .. and 16 + 4 kqs ..
    f32x2 acc[2 * IP][CS];
#pragma unroll
    for (int p = 0; p < 2 * IP; ++p)
#pragma unroll
      for (int n = 0; n < CS; ++n) acc[p][n] = 0;
    auto add = [&](const float* rows, const float* cols) {
#pragma unroll 1
      for (int t = 4 * kqs; t < DCH; t += 4 * DCH_KS) {
        ulonglong2 k[4][IP];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int p = 0; p < IP; ++p) k[b][p] = *reinterpret_cast<const ulonglong2*>(rows + (t + b) * LD + 64 * p + 4 * ig);
#pragma unroll
        for (int n = 0; n < CS; ++n) {
          const float4 v = *reinterpret_cast<const float4*>(cols + (cgp + CGN * n) * DCH_CL + t);
          const f32x2 v4[4] = {pack2(v.x, v.x), pack2(v.y, v.y), pack2(v.z, v.z), pack2(v.w, v.w)};
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int p = 0; p < IP; ++p) {
              acc[2 * p][n] = fma2(k[b][p].x, v4[b], acc[2 * p][n]);
              acc[2 * p + 1][n] = fma2(k[b][p].y, v4[b], acc[2 * p + 1][n]);
            }
        }
      }
    };
    if constexpr (GATED) add(X, cs);
    else { add(Y, V); add(Y + DCH * LD, ct); }
    float g[4 * IP][CS];
#pragma unroll
    for (int p = 0; p < 2 * IP; ++p)
#pragma unroll
      for (int n = 0; n < CS; ++n) {
        const float2 v = unpack2(acc[p][n]);
        g[2 * p][n] = v.x;
        g[2 * p + 1][n] = v.y;
      }
    dch_share<4 * IP, CS, 8>(g, kqs);
#pragma unroll
    for (int m = 0; m < CK; ++m)
#pragma unroll
      for (int p = 0; p < IP; ++p) {
        const float4 w = GATED ? make_float4(vec[2 * DCH - 1], vec[2 * DCH - 1], vec[2 * DCH - 1], vec[2 * DCH - 1]) : *reinterpret_cast<const float4*>(vec + 64 * p + 4 * ig);
        s[4 * p][m] = fmaf(w.x, s[4 * p][m], g[4 * p][m]);
        s[4 * p + 1][m] = fmaf(w.y, s[4 * p + 1][m], g[4 * p + 1][m]);
        s[4 * p + 2][m] = fmaf(w.z, s[4 * p + 2][m], g[4 * p + 2][m]);
        s[4 * p + 3][m] = fmaf(w.w, s[4 * p + 3][m], g[4 * p + 3][m]);
        *reinterpret_cast<float4*>(St + (cgp + CGN * (kqs * CK + m)) * LS + 64 * p + 4 * ig) = make_float4(s[4 * p][m], s[4 * p + 1][m], s[4 * p + 2][m], s[4 * p + 3][m]);
      }                                                // read again behind the next barrier
  }
#pragma unroll
  for (int m = 0; m < CK; ++m) {
    const int col = col0 + cgp + CGN * (kqs * CK + m);
#pragma unroll
    for (int p = 0; p < IP; ++p)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = 64 * p + 4 * ig + r;
        if (i < a.dk && col < a.dv) S[(size_t)i * a.dv + col] = s[4 * p + r][m];
      }
  }
}

}  // namespace xl
