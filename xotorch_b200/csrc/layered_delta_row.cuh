// layered_delta_row.cuh — one token of a delta-rule mixer, all of it between the input projection and the output product: the decode form of
// delta_rule_kernel and of the kernels around it (layered_kernels.cuh, layered_blocks.cuh), for steps in which every request brings one row.
//
//   general delta rule:  tanh of the low-rank branch, its second product, decay / removal / unit key, S <- diag(w) S - (a u)(u^T S) + k v^T, o = S^T r,
//                        head norm, sigmoid gate
//   gated delta rule:    the channels' short convolution (its window moves on), unit key and query, S <- g S + k (beta (v - g k^T S))^T, o = S^T r, head
//                        norm shared by the heads, silu gate
//
// A token reads and writes dk x dv floats of state a head and does next to nothing else: bound by that traffic when there are many heads and by latency when
// there are few.  One block of 256 threads has one (request, value head): a thread holds four neighbouring columns of RPT rows, so that a warp's accesses are whole
// rows, and the state is on its way before the block waits for the kernel in front (it was last written in the step before, which has ended; the slot that says where it
// lies comes from the staged index arrays, which were complete before the step's first kernel started: launch_early).  The sums over
// rows run over the thread's rows, then over the warps through shared memory, one barrier each.  The heads that share a query / key head are a cluster: all read the
// shared channels' window before the first of them moves it on.
// Measured (B200): 16 requests, 32 heads of 128 x 128 (67 MB of state a step): five launches of 54 us -> one step of it 31 us shorter; 8 requests, 32 heads of 64 x 64: four launches
// of 19 us, a step 11.4 us shorter; one request, 16 heads of 64 x 64: a step 7.4 us shorter (144.7 -> 137.4 with everything else in it).
#pragma once
#include "layered_stream.cuh"

namespace xl {

constexpr int DROW_THREADS = 256, DROW_TAPS = 8;   // taps of the convolution held in registers

struct DeltaRowArgs {
  const float* proj;                                   // [M, ld]
  int ld, H, rep, dk, dv;                              // rep: value heads that share a query / key head (general form: 1)
  float* state;                                        // this layer's part of slot 0
  size_t slot_stride;
  // general form: columns of k, r, v, removal logits and low-rank inputs; w2 [H * dk, low_rank], biases [H * dk]
  int col_k, col_r, col_v, col_a, col_w1, low_rank;
  const void *w2, *w0, *a_b;
  // gated form: channels [q (G * dk) | k (G * dk) | v (H * dv)] from column col_c on, filter [C, taps], window of slot 0 [taps - 1, C]; logits at col_b, col_a
  int col_c, C, taps, col_b;
  const void *conv_w, *a_log, *dt_bias;
  float* window;
  // out [M, H * dv]: head norm weight (norm_stride: dv, or 0 when shared), gate columns from col_g on
  const void* norm_w;
  int norm_stride, col_g;
  float eps;
  void* out;
};

// CGP: column groups of four a row is cut into (a power of two, dv <= 4 CGP); RPT: rows of a thread (dk <= RPT * 256 / CGP)
template <typename T, int CGP, int RPT, bool GATED>
__global__ void __launch_bounds__(DROW_THREADS, 2) delta_row_kernel(const DeltaRowArgs a, const Item* __restrict__ seqs) {
  constexpr int SUBS = 32 / CGP, RG = 8 * SUBS, DKP = RPT * RG, DVP = 4 * CGP, TPR = DROW_THREADS / DKP;
  static_assert(TPR >= 1, "a thread per row");
  __shared__ __align__(16) float vk[DKP], vr[DKP], vw[DKP], vu[DKP], vau[DKP], vv[DVP], red[2][8][DVP];
  __shared__ float th[256];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.x % a.H;
  const int row0 = __ldcg(&seqs[blockIdx.x / a.H].row0), slot = __ldcg(&seqs[blockIdx.x / a.H].slot);
  const int col = 4 * (lane % CGP), rg = warp * SUBS + lane / CGP;
  const bool in_col = col < a.dv;
  float* S = a.state + (size_t)slot * a.slot_stride + (size_t)h * a.dk * a.dv;
  float4 s[RPT];
#pragma unroll
  for (int j = 0; j < RPT; ++j) s[j] = in_col && rg + RG * j < a.dk ? __ldcg(reinterpret_cast<const float4*>(S + (size_t)(rg + RG * j) * a.dv + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t m = row0;
  const float* pr = a.proj + m * a.ld;
  float g = 0.f, beta = 0.f, ik = 1.f, iq = 1.f;      // gated form
  constexpr int NCH = (2 * DKP + DVP + DROW_THREADS - 1) / DROW_THREADS;   // its channels per thread
  float cur[NCH], win[NCH][DROW_TAPS - 1];
  auto channel = [&](int e, int& c) {                  // the e-th channel of this head: q, then k, then v
    c = e < a.dk ? h / a.rep * a.dk + e : e < 2 * a.dk ? (a.H / a.rep) * a.dk + h / a.rep * a.dk + e - a.dk : 2 * (a.H / a.rep) * a.dk + h * a.dv + e - 2 * a.dk;
    return e < 2 * a.dk + a.dv;
  };
  float* const wst = GATED ? a.window + (size_t)slot * a.slot_stride : nullptr;
  if constexpr (GATED) {
#pragma unroll
    for (int n = 0; n < NCH; ++n) {
      int c;
      const bool on = channel(tid + n * DROW_THREADS, c);
#pragma unroll
      for (int i = 0; i < DROW_TAPS - 1; ++i) win[n][i] = on && i < a.taps - 1 ? __ldcg(wst + (size_t)i * a.C + c) : 0.f;
    }
    pdl_wait();
    if (a.rep > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // the window has been read
    const T* cw = static_cast<const T*>(a.conv_w);
#pragma unroll
    for (int n = 0; n < NCH; ++n) {
      const int e = tid + n * DROW_THREADS;
      int c;
      if (!channel(e, c)) continue;
      cur[n] = pr[a.col_c + c];
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < DROW_TAPS - 1; ++i)
        if (i < a.taps - 1) acc = fmaf(ldf(cw + (size_t)c * a.taps + i), win[n][i], acc);
      acc = siluf_(fmaf(ldf(cw + (size_t)c * a.taps + a.taps - 1), cur[n], acc));
      if (e < a.dk) vr[e] = acc;
      else if (e < 2 * a.dk) vk[e - a.dk] = acc;
      else vv[e - 2 * a.dk] = acc;
    }
    beta = sigmoidf_(pr[a.col_b + h]);
    g = expf(-expf(ldf(static_cast<const T*>(a.a_log) + h)) * softplusf_(pr[a.col_a + h] + ldf(static_cast<const T*>(a.dt_bias) + h)));
    __syncthreads();
    float sq = 0.f, sk = 0.f;
    for (int i = lane; i < a.dk; i += 32) {
      sq = fmaf(vr[i], vr[i], sq);
      sk = fmaf(vk[i], vk[i], sk);
    }
    iq = 1.0f / (sqrtf(warp_sum(sq) + 1e-6f) * sqrtf((float)a.dk));
    ik = 1.0f / sqrtf(warp_sum(sk) + 1e-6f);
  } else {
    // the second product of the decay branch: TPR threads per row, its weights ahead of the wait
    const int i = tid / TPR, part = tid % TPR, at = h * a.dk + i;
    constexpr int VEC = 16 / sizeof(T), PRE = 4;
    const int per = a.low_rank / TPR;
    const T* w2 = static_cast<const T*>(a.w2) + (size_t)at * a.low_rank + (size_t)part * per;
    const bool vec = a.low_rank % (TPR * VEC) == 0 && per <= PRE * VEC && (reinterpret_cast<uintptr_t>(a.w2) & 15) == 0;
    uint4 raw[PRE];
    if (vec)
#pragma unroll
      for (int q = 0; q < PRE; ++q) raw[q] = i < a.dk && q * VEC < per ? *reinterpret_cast<const uint4*>(w2 + q * VEC) : make_uint4(0, 0, 0, 0);
    pdl_wait();
    for (int j = tid; j < a.low_rank; j += DROW_THREADS) {
      T t;
      stf(&t, tanhf(pr[a.col_w1 + j]));
      th[j] = ldf(&t);
    }
    float sk = 0.f;
    for (int j = lane; j < a.dk; j += 32) { const float v = pr[a.col_k + h * a.dk + j]; sk = fmaf(v, v, sk); }
    const float inv = 1.0f / sqrtf(warp_sum(sk) + 1e-6f);
    for (int j = tid; j < a.dv; j += DROW_THREADS) vv[j] = pr[a.col_v + h * a.dv + j];
    float kv = 0.f, rv = 0.f, av = 0.f;
    if (i < a.dk && part == 0) { kv = pr[a.col_k + at]; rv = pr[a.col_r + at]; av = pr[a.col_a + at]; }
    __syncthreads();
    float acc = 0.f;
    if (i < a.dk) {
      if (vec) {
#pragma unroll
        for (int q = 0; q < PRE; ++q)
          if (q * VEC < per) {
            const T* w = reinterpret_cast<const T*>(&raw[q]);
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc = fmaf(ldf(w + v), th[part * per + q * VEC + v], acc);
          }
      } else {
        const T* w = static_cast<const T*>(a.w2) + (size_t)at * a.low_rank;
        for (int j = part; j < a.low_rank; j += TPR) acc = fmaf(ldf(w + j), th[j], acc);
      }
    }
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (i < a.dk && part == 0) {
      const float u = kv * inv;
      vk[i] = kv;
      vr[i] = rv;
      vu[i] = u;
      vau[i] = sigmoidf_(av + ldf(static_cast<const T*>(a.a_b) + at)) * u;
      vw[i] = expf(-0.60653065971263342f * sigmoidf_(acc + ldf(static_cast<const T*>(a.w0) + at)));
    }
    __syncthreads();
  }
  // sums over all rows of four columns: this thread's, the warp's, the block's
  auto total = [&](float4 v, float (*buf)[DVP]) {
#pragma unroll
    for (int o = CGP; o < 32; o <<= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
      v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
    }
    if (lane < CGP) *reinterpret_cast<float4*>(&buf[warp][col]) = v;
    __syncthreads();
    float4 t = *reinterpret_cast<const float4*>(&buf[0][col]);
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      const float4 p = *reinterpret_cast<const float4*>(&buf[w][col]);
      t = make_float4(t.x + p.x, t.y + p.y, t.z + p.z, t.w + p.w);
    }
    return t;
  };
  float4 d = make_float4(0.f, 0.f, 0.f, 0.f), o = d;
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int r = rg + RG * j;
    const float u = r < a.dk ? (GATED ? vk[r] * ik : vu[r]) : 0.f;
    d = make_float4(fmaf(u, s[j].x, d.x), fmaf(u, s[j].y, d.y), fmaf(u, s[j].z, d.z), fmaf(u, s[j].w, d.w));
  }
  d = total(d, red[0]);
  const float4 v = in_col ? *reinterpret_cast<const float4*>(&vv[col]) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 c = make_float4(beta * fmaf(-g, d.x, v.x), beta * fmaf(-g, d.y, v.y), beta * fmaf(-g, d.z, v.z), beta * fmaf(-g, d.w, v.w));   // gated form
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int r = rg + RG * j;
    if (r >= a.dk) break;
    if constexpr (GATED) {
      const float k = vk[r] * ik;
      s[j] = make_float4(fmaf(k, c.x, g * s[j].x), fmaf(k, c.y, g * s[j].y), fmaf(k, c.z, g * s[j].z), fmaf(k, c.w, g * s[j].w));
    } else {
      const float k = vk[r], n = -vau[r], w = vw[r];
      s[j] = make_float4(fmaf(w, s[j].x, fmaf(n, d.x, k * v.x)), fmaf(w, s[j].y, fmaf(n, d.y, k * v.y)), fmaf(w, s[j].z, fmaf(n, d.z, k * v.z)),
                         fmaf(w, s[j].w, fmaf(n, d.w, k * v.w)));
    }
    const float q = GATED ? vr[r] * iq : vr[r];
    o = make_float4(fmaf(q, s[j].x, o.x), fmaf(q, s[j].y, o.y), fmaf(q, s[j].z, o.z), fmaf(q, s[j].w, o.w));
    if (in_col) *reinterpret_cast<float4*>(S + (size_t)r * a.dv + col) = s[j];
  }
  o = total(o, red[1]);
  if (warp == 0) {
    const bool mine = in_col && lane < CGP;
    const float rs = 1.0f / sqrtf(warp_sum(mine ? sq4(o) : 0.f) / (float)a.dv + a.eps);
    if (mine) {
      const float4 z = ld4f(pr + a.col_g + h * a.dv + col);
      const T* w = static_cast<const T*>(a.norm_w) + h * a.norm_stride + col;
      auto gate = [](float x) { return GATED ? x * sigmoidf_(x) : sigmoidf_(x); };
      st4f(static_cast<T*>(a.out) + m * a.H * a.dv + h * a.dv + col,
           make_float4(o.x * rs * ldf(w) * gate(z.x), o.y * rs * ldf(w + 1) * gate(z.y), o.z * rs * ldf(w + 2) * gate(z.z), o.w * rs * ldf(w + 3) * gate(z.w)));
    }
  }
  if constexpr (GATED) {
    if (a.rep > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
    for (int n = 0; n < NCH; ++n) {
      const int e = tid + n * DROW_THREADS;
      int ch;
      if (!channel(e, ch) || (e < 2 * a.dk && h % a.rep != 0)) continue;   // shared channels: the first head of the cluster moves them on
#pragma unroll
      for (int i = 0; i < DROW_TAPS - 1; ++i)
        if (i < a.taps - 1) wst[(size_t)i * a.C + ch] = i + 1 < a.taps - 1 ? win[n][i + 1 < DROW_TAPS - 1 ? i + 1 : i] : cur[n];
    }
  }
}

}  // namespace xl
