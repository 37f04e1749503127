// layered_gqa_row.cuh — attention of one row per request over cached keys and values: the decode form of gqa_attention_kernel (layered_gqa.cuh), whose tiles of 32 keys,
// staged in shared memory as fp32 for up to 32 warps, leave four warps at work and three dependent round trips in front of them when a request brings a single row.
//
// One block has one (request, key/value head, share of the keys: every gridDim.z-th 32 of them); REP of the query heads that share it.  Eight lanes hold a key: its entries and its value's come straight
// from the pool in 16-byte pieces, the next key's on their way meanwhile, the queries and the sums stay in registers in fp32.  Each lane of a key finishes the score of one head (soft
// cap, distance terms, mask), keeps that head's running maximum and sum, and hands the weight round.  The shares of a request are a cluster: their sums meet in
// shared memory and every block finishes a part of the outputs (sink, gate).  More shares than a cluster holds leave them in `part` for gqa_combine_kernel.
// Bound by latency while the cache is short, by the fp32 arithmetic on each key when it is long (16 requests behind 8000 tokens, 32 + 8 heads of 128, a layer: 525 MB in 460 us, general kernel 1590); heads
// that share a key head beyond four read its keys again: gqa_row_pays (layered.cu) has the line.  Measured (B200): 8 requests of
// some 40 cached tokens, 16 + 4 heads of 128, a launch and what follows it in a step: 9.3 + 3.1 us (general kernel, merge) -> 7.6; a step with two such layers 305 -> 299 us.
#pragma once
#include "layered_gqa.cuh"
#include "layered_stream.cuh"

namespace xl {

constexpr int GROW_THREADS = 256, GROW_KEYS = 32;   // keys a block has under way: four per warp

struct GqaRowArgs {
  const float* qf;                                   // [M, H, D]
  const void* pool;
  Paging pg;
  const Item* items;
  int H, G;
  GqaScore sc;
  const float* gate;
  int gate_mode, gate_ld, gate_col0;
  void* out;                                         // [M, H * D]
  float* part;                                       // NULL: the shares of the keys (gridDim.z) are a cluster
};

// D = entries of a key and of a value
template <typename T, int D, int REP>
__global__ void __launch_bounds__(GROW_THREADS) gqa_row_kernel(const GqaRowArgs a) {
  pdl_enter();
  constexpr int VEC = 16 / sizeof(T), NP = D / (8 * VEC), DPL = D / 8;   // entries and pieces of 16 bytes, and entries in all, of a lane
  __shared__ float so[9][REP][D], sm[9][REP], sd[9][REP];                // per warp, and [8]: the block's
  const Item it = a.items[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane & 7, rep = a.H / a.G, per_g = rep / REP;
  const int g = blockIdx.y / per_g, h0 = g * rep + blockIdx.y % per_g * REP, z = blockIdx.z, nz = gridDim.z;
  const int m = it.row0, pos = it.pos0;
  const GqaScore& sc = a.sc;
  const int first = gqa_first_key(pos, sc.window, sc.chunk), extra = gqa_extra_keys(first, pos, sc.window, sc.keep_first, sc.pool), keys = extra + pos - first + 1;
  const int v0 = z * GROW_KEYS, step = nz * GROW_KEYS, seen = sc.pool > 0 ? gqa_blocks_seen(pos, sc.window, sc.pool) : 0;
  const size_t rowlen = (size_t)a.G * 2 * D;
  const T* pool = static_cast<const T*>(a.pool) + (size_t)g * D + l * VEC;
  auto row_of = [&](int v) { return v >= extra ? a.pg.row(it.slot, first + v - extra) : sc.pool > 0 ? sc.pool_rows + a.pg.row(it.slot, v) : a.pg.row(it.slot, v); };
  auto load = [&](int v, uint4 (&k)[NP], uint4 (&x)[NP]) {
    const T* src = pool + row_of(v) * rowlen;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      k[p] = *reinterpret_cast<const uint4*>(src + p * 8 * VEC);
      x[p] = *reinterpret_cast<const uint4*>(src + (size_t)a.G * D + p * 8 * VEC);
    }
  };
  uint4 kn[NP], vn[NP];
  const int mine = v0 + warp * 4 + (lane >> 3);        // this group's first key
  if (mine < keys) load(mine, kn, vn);
  float q[REP][DPL], acc[REP][DPL];
#pragma unroll
  for (int r = 0; r < REP; ++r)
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int e = 0; e < VEC; e += 4) {
        const float4 f = ld4f(a.qf + ((size_t)m * a.H + h0 + r) * D + (p * 8 + l) * VEC + e);
        q[r][p * VEC + e] = f.x; q[r][p * VEC + e + 1] = f.y; q[r][p * VEC + e + 2] = f.z; q[r][p * VEC + e + 3] = f.w;
      }
#pragma unroll
  for (int r = 0; r < REP; ++r)
#pragma unroll
    for (int d = 0; d < DPL; ++d) acc[r][d] = 0.f;
  const int own = l % REP;                             // the head whose score, maximum and sum this lane keeps
  const float r1 = sc.r1 ? ldf(static_cast<const T*>(sc.r1) + h0 + own) : 0.f, r2 = sc.r1 ? ldf(static_cast<const T*>(sc.r2) + h0 + own) : 0.f;
  const float* rel_head = sc.rel ? sc.rel + (size_t)(h0 + own) * sc.rel_n : nullptr;
  float mx = -INFINITY, den = 0.f;
  for (int v = mine, left = (keys - v0 + step - 1) / step; left > 0; v += step, --left) {   // the same number of turns for all lanes: they exchange
    uint4 k[NP], x[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) { k[p] = kn[p]; x[p] = vn[p]; }
    const bool on = v < keys;
    if (v + step < keys) load(v + step, kn, vn);
    float dot[REP];
#pragma unroll
    for (int r = 0; r < REP; ++r) dot[r] = 0.f;
    if (on)
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float f = ldf(reinterpret_cast<const T*>(&k[p]) + e);
#pragma unroll
          for (int r = 0; r < REP; ++r) dot[r] = fmaf(q[r][p * VEC + e], f, dot[r]);
        }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < REP; ++r) dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], o);
    float s = dot[0];
#pragma unroll
    for (int r = 1; r < REP; ++r) s = own == r ? dot[r] : s;
    const int j = v >= extra ? first + v - extra : v;  // a token's position (kept first tokens keep theirs); a pooled block's index
    const bool vis = on && (v >= extra ? gqa_visible(pos, j, sc.window, sc.chunk, sc.keep_first) : (sc.pool > 0 ? v < seen : true));
    s = vis ? gqa_adjust<T>(s, sc, r1, r2, rel_head, pos - j) : -INFINITY;
    const float nm = fmaxf(mx, s), corr = mx == -INFINITY ? 0.f : expf(mx - nm), w = s == -INFINITY ? 0.f : expf(s - nm);
    den = fmaf(den, corr, w);
    mx = nm;
#pragma unroll
    for (int r = 0; r < REP; ++r) {
      const float c = __shfl_sync(0xffffffffu, corr, (lane & 24) + r), wr = __shfl_sync(0xffffffffu, w, (lane & 24) + r);
      if (c != 1.f)
#pragma unroll
        for (int d = 0; d < DPL; ++d) acc[r][d] *= c;
      if (wr != 0.f)                                   // a weight of 0 takes nothing from its value, not even 0 * Inf
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[r][p * VEC + e] = fmaf(wr, ldf(reinterpret_cast<const T*>(&x[p]) + e), acc[r][p * VEC + e]);
    }
  }
  // From here on sums are merged without a look at their weights: who saw no key has parked zeros, and who saw keys whose scores are all NaN (its maximum is still -inf, its
  // weight 0) must not drop out of the denominator.
  // the warp's four keys of every turn: one maximum, sums over the groups; lane group i ends with a quarter of the entries
  float wm = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
  wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, 16));
  const float f = mx == -INFINITY ? 0.f : expf(mx - wm);
  den *= f;
  den += __shfl_xor_sync(0xffffffffu, den, 8);
  den += __shfl_xor_sync(0xffffffffu, den, 16);
  if (lane < REP) { sm[warp][lane] = wm; sd[warp][lane] = den; }
  const bool up16 = lane & 16, up8 = lane & 8;
#pragma unroll
  for (int r = 0; r < REP; ++r) {
    const float fr = __shfl_sync(0xffffffffu, f, (lane & 24) + r);
    float t[DPL];
#pragma unroll
    for (int d = 0; d < DPL; ++d) t[d] = acc[r][d] * fr;
#pragma unroll
    for (int d = 0; d < DPL / 2; ++d) t[d] = (up16 ? t[d + DPL / 2] : t[d]) + __shfl_xor_sync(0xffffffffu, up16 ? t[d] : t[d + DPL / 2], 16);
#pragma unroll
    for (int d = 0; d < DPL / 4; ++d) t[d] = (up8 ? t[d + DPL / 4] : t[d]) + __shfl_xor_sync(0xffffffffu, up8 ? t[d] : t[d + DPL / 4], 8);
#pragma unroll
    for (int d = 0; d < DPL / 4; ++d) {
      const int i = (up16 ? DPL / 2 : 0) + (up8 ? DPL / 4 : 0) + d;      // entry i of the lane
      so[warp][r][(i / VEC * 8 + l) * VEC + i % VEC] = t[d];
    }
  }
  __syncthreads();
  // the block
  auto scale = [](float mi, float top) { return mi == -INFINITY ? 0.f : expf(mi - top); };
  for (int i = threadIdx.x; i < REP * D; i += GROW_THREADS) {
    const int r = i / D, d = i % D;
    float top = sm[0][r], o = 0.f, dn = 0.f;
#pragma unroll
    for (int w = 1; w < 8; ++w) top = fmaxf(top, sm[w][r]);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float c = scale(sm[w][r], top);
      o = fmaf(c, so[w][r][d], o);
      dn = fmaf(c, sd[w][r], dn);
    }
    so[8][r][d] = o;
    if (d == 0) { sm[8][r] = top; sd[8][r] = dn; }
    if (a.part) {
      float* dst = a.part + (((size_t)m * a.H + h0 + r) * nz + z) * (size_t)(2 + D);
      if (d == 0) { dst[0] = top; dst[1] = dn; }
      dst[2 + d] = o;
    }
  }
  if (a.part) return;
  __syncthreads();
  if (nz > 1) xb::cluster_sync_all();
  // the cluster: block z finishes every nz-th piece of 32 entries
  for (int i = (z + nz * warp) * 32 + lane; i < REP * D; i += 32 * nz * (GROW_THREADS / 32)) {
    const int r = i / D, d = i % D, h = h0 + r;
    float top = -INFINITY, o = 0.f, dn = 0.f;
    if (nz == 1) {
      top = sm[8][r];
      o = so[8][r][d];
      dn = sd[8][r];
    } else {
      float mi[8], oi[8], di[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) {
          mi[c] = ld_dsmem_f32(xb::smem_u32(&sm[8][r]), c);
          di[c] = ld_dsmem_f32(xb::smem_u32(&sd[8][r]), c);
          oi[c] = ld_dsmem_f32(xb::smem_u32(&so[8][r][d]), c);
        }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) top = fmaxf(top, mi[c]);
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) {
          const float w = scale(mi[c], top);
          o = fmaf(w, oi[c], o);
          dn = fmaf(w, di[c], dn);
        }
    }
    const float corr = sc.sink || sc.sink_one ? apply_sink(gqa_sink_score<T>(sc.sink, h), top, dn) : 1.0f;
    stf(static_cast<T*>(a.out) + ((size_t)m * a.H + h) * D + d, o * (corr / dn) * gqa_gate(a.gate, a.gate_mode, m, a.gate_ld, a.gate_col0, h, D, d));
  }
  if (nz > 1) xb::cluster_sync_all();                  // nobody's shared memory goes away while a peer reads it
}

}  // namespace xl
