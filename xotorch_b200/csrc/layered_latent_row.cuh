// layered_latent_row.cuh — latent attention of one row per request: the decode form of latent_attention_kernel (layered_kernels.cuh), which stages tiles of 32 cached rows in
// shared memory 4 bytes at a time and leaves its sums to a second launch.
//
// A block has eight heads of one request and a share of its keys (every gridDim.z-th four); a warp has one head.  Eight lanes hold a cached row [latent R | rotated part] in 16-byte
// pieces straight from the pool, the next one's on its way meanwhile: its latent entries are the key's and, with the weight, the value's, so a row is read once a head and the
// eight warps of a block meet in L1.  Queries and sums stay in registers in fp32.  The shares of a request are a cluster, whose blocks finish a part of the outputs
// each (sink, gate); more shares than a cluster holds leave them in `part` for latent_attention_combine_kernel.  Measured (B200): 16 requests of
// some 30 cached tokens, 32 heads, rows of 576 (bound by latency; behind more tokens every block reads the request's rows anew and the general kernel takes over: latent_row_pays, layered.cu), a step with two such layers: 16 + 8 us a layer (general kernel, merge) -> the step 18 us shorter (7115 -> 6877 us for 13 steps).
#pragma once
#include "layered_stream.cuh"

namespace xl {

constexpr int LROW_THREADS = 256, LROW_KEYS = 4;     // keys a warp has under way

struct LatentRowArgs {
  const float* q;                                    // [M, H, R + dr]: absorbed queries, rotated parts
  const void* pool;                                  // rows of R + dr
  Paging pg;
  const Item* items;
  int H, dr, window;
  float scale;
  const float* gate;
  int gate_ld, gate_col0;
  const void* sink;
  void* out;                                         // [M, H, R]
  float* part;                                       // NULL: the shares of the keys (gridDim.z) are a cluster
};

// R: whole pieces of 8 lanes x 16 bytes; the rotated part is one such piece or less
template <typename T, int R>
__global__ void __launch_bounds__(LROW_THREADS) latent_row_kernel(const LatentRowArgs a) {
  pdl_enter();
  constexpr int VEC = 16 / sizeof(T), NP = R / (8 * VEC), DPL = R / 8;   // pieces and entries of the latent that a lane holds
  extern __shared__ __align__(16) float lrow_sm[];   // [8][R] sums, [8] maxima, [8] denominators
  float *so = lrow_sm, *sm = so + 8 * R, *sd = sm + 8;
  const Item it = a.items[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane & 7, z = blockIdx.z, nz = gridDim.z, W = R + a.dr;
  const int h = blockIdx.y * 8 + warp, m = it.row0, pos = it.pos0;
  const bool active = h < a.H;                       // warp-uniform
  const int first = a.window > 0 ? max(0, pos - a.window + 1) : 0, keys = pos - first + 1, v0 = z * LROW_KEYS, step = nz * LROW_KEYS;
  const bool rot = l * VEC < a.dr;
  const T* pool = static_cast<const T*>(a.pool) + l * VEC;
  auto load = [&](int v, uint4 (&k)[NP + 1]) {
    const T* src = pool + a.pg.row(it.slot, first + v) * (size_t)W;
#pragma unroll
    for (int p = 0; p < NP; ++p) k[p] = *reinterpret_cast<const uint4*>(src + p * 8 * VEC);
    k[NP] = rot ? *reinterpret_cast<const uint4*>(src + R) : make_uint4(0, 0, 0, 0);
  };
  uint4 kn[NP + 1];
  const int mine = v0 + (lane >> 3);
  if (active && mine < keys) load(mine, kn);
  float q[DPL + VEC], acc[DPL];
  const float* qs = a.q + ((size_t)m * a.H + (active ? h : 0)) * W + l * VEC;
#pragma unroll
  for (int p = 0; p <= NP; ++p)
#pragma unroll
    for (int e = 0; e < VEC; e += 4) {
      const float4 f = p < NP || rot ? ld4f(qs + p * 8 * VEC + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      q[p * VEC + e] = f.x; q[p * VEC + e + 1] = f.y; q[p * VEC + e + 2] = f.z; q[p * VEC + e + 3] = f.w;
    }
#pragma unroll
  for (int d = 0; d < DPL; ++d) acc[d] = 0.f;
  float mx = -INFINITY, den = 0.f;
  if (active) {
    for (int v = mine, left = (keys - v0 + step - 1) / step; left > 0; v += step, --left) {   // the same number of turns for all lanes: they exchange
      uint4 k[NP + 1];
#pragma unroll
      for (int p = 0; p <= NP; ++p) k[p] = kn[p];
      const bool on = v < keys;
      if (v + step < keys) load(v + step, kn);
      float s0 = 0.f, s1 = 0.f;
      if (on)
#pragma unroll
        for (int p = 0; p <= NP; ++p)
#pragma unroll
          for (int e = 0; e < VEC; e += 2) {
            s0 = fmaf(q[p * VEC + e], ldf(reinterpret_cast<const T*>(&k[p]) + e), s0);
            s1 = fmaf(q[p * VEC + e + 1], ldf(reinterpret_cast<const T*>(&k[p]) + e + 1), s1);
          }
      float s = s0 + s1;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s = on ? s * a.scale : -INFINITY;
      const float nm = fmaxf(mx, s), corr = mx == -INFINITY ? 0.f : expf(mx - nm), w = s == -INFINITY ? 0.f : expf(s - nm);
      den = fmaf(den, corr, w);
      mx = nm;
      if (corr != 1.f)
#pragma unroll
        for (int d = 0; d < DPL; ++d) acc[d] *= corr;
      if (on)
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[p * VEC + e] = fmaf(w, ldf(reinterpret_cast<const T*>(&k[p]) + e), acc[p * VEC + e]);
    }
    // From here on sums are merged without a look at their weights: who saw no key has parked zeros, and who saw keys whose scores are all NaN (its maximum is still
    // -inf, its weight 0) must not drop out of the denominator.
    // the warp: one maximum, sums over the four keys of every turn; lane group i ends with a quarter of the entries
    float top = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
    const float f = mx == -INFINITY ? 0.f : expf(mx - top);
    den *= f;
    den += __shfl_xor_sync(0xffffffffu, den, 8);
    den += __shfl_xor_sync(0xffffffffu, den, 16);
    mx = top;
    if (lane == 0) { sm[warp] = top; sd[warp] = den; }
    const bool up16 = lane & 16, up8 = lane & 8;
#pragma unroll
    for (int d = 0; d < DPL; ++d) acc[d] *= f;
#pragma unroll
    for (int d = 0; d < DPL / 2; ++d) acc[d] = (up16 ? acc[d + DPL / 2] : acc[d]) + __shfl_xor_sync(0xffffffffu, up16 ? acc[d] : acc[d + DPL / 2], 16);
#pragma unroll
    for (int d = 0; d < DPL / 4; ++d) acc[d] = (up8 ? acc[d + DPL / 4] : acc[d]) + __shfl_xor_sync(0xffffffffu, up8 ? acc[d] : acc[d + DPL / 4], 8);
#pragma unroll
    for (int d = 0; d < DPL / 4; ++d) {
      const int i = (up16 ? DPL / 2 : 0) + (up8 ? DPL / 4 : 0) + d;      // entry i of the lane
      so[warp * R + (i / VEC * 8 + l) * VEC + i % VEC] = acc[d];
    }
  }
  if (a.part) {
    if (!active) return;
    __syncwarp();
    float* dst = a.part + (((size_t)m * a.H + h) * nz + z) * (size_t)(2 + R);
    if (lane == 0) { dst[0] = mx; dst[1] = den; }
    for (int d = lane; d < R; d += 32) dst[2 + d] = so[warp * R + d];
    return;
  }
  __syncthreads();
  if (nz > 1) xb::cluster_sync_all();
  // the cluster: a warp finishes every nz-th piece of 32 entries of its head
  if (active) {
    float ms[8], ds[8], top = -INFINITY, dn = 0.f;
    if (nz > 1) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) { ms[c] = ld_dsmem_f32(xb::smem_u32(sm + warp), c); ds[c] = ld_dsmem_f32(xb::smem_u32(sd + warp), c); }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) top = fmaxf(top, ms[c]);
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nz) { ms[c] = ms[c] == -INFINITY ? 0.f : expf(ms[c] - top); dn = fmaf(ms[c], ds[c], dn); }
    } else {
      __syncwarp();
      top = sm[warp];
      dn = sd[warp];
    }
    float g = a.sink ? apply_sink(ldf(static_cast<const T*>(a.sink) + h), top, dn) : 1.0f;
    g /= dn;
    if (a.gate) g *= sigmoidf_(a.gate[(size_t)m * a.gate_ld + a.gate_col0 + h]);
    T* out = static_cast<T*>(a.out) + ((size_t)m * a.H + h) * R;
    for (int d = z * 32 + lane; d < R; d += nz * 32) {
      float o = 0.f;
      if (nz > 1) {
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < nz) v[c] = ld_dsmem_f32(xb::smem_u32(so + warp * R + d), c);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < nz) o = fmaf(ms[c], v[c], o);
      } else {
        o = so[warp * R + d];
      }
      stf(out + d, o * g);
    }
  }
  if (nz > 1) xb::cluster_sync_all();                // nobody's shared memory goes away while a peer reads it
}

}  // namespace xl
