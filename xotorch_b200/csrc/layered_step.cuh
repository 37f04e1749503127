// layered_step.cuh — the two ends of a step of the layered-model engine.  Index arrays come in and results go out through page-locked host memory that the kernels themselves read and write: a copy
// engine's transfer costs little, but handing over to it and back does (about 35 us between the copy in and the first kernel of a step of one row, 10 us
// around the copies out).
#pragma once
#include "layered_stream.cuh"

namespace xl {

// Where a step's results go; the first ints of the staged block, so that a replayed step reads the pointers of this call.
struct StepOut {
  float* logits;                                       // [n_want, V] the finished logits: page-locked host memory, or in place; NULL: not asked for
  int* tail;                                           // page-locked: [n_want] argmax, then the step's error word
};
constexpr int STEP_OUT_INTS = sizeof(StepOut) / 4;

// n16 pieces of 16 bytes, page-locked host memory -> device; then the page table entries that this step adds: n_pages pairs (entry, page) from int
// `pages` of the block on, entry < 0 = none.  One round trip over PCIe: the loads depend on nothing.
__global__ void stage_in_kernel(const int4* __restrict__ src, int4* __restrict__ dst, int n16, int pages, int n_pages, int* __restrict__ table) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n16) dst[i] = __ldcv(src + i);
  if (i < n_pages) {
    const int2 pr = make_int2(__ldcv(reinterpret_cast<const int*>(src) + pages + 2 * i), __ldcv(reinterpret_cast<const int*>(src) + pages + 2 * i + 1));
    if (pr.x >= 0) table[pr.x] = pr.y;
  }
}

// finishes the logits of every row — l <- l * scale, then l <- cap * tanh(l / cap) when cap > 0 —, takes the lowest-index argmax of the row
// (greedy sampling on the device) and sends both where the caller wants them, the step's error word behind the rows' results.  A cluster of `parts` blocks shares a row
// (grid n_want * parts, along x: as many rows as a step may want): its reads and its writes over PCIe are in flight together (one row of 32000: 5.6 us by one block without the copy out).
// A launch has columns c0 .. c1 - 1, segment `seg` of `segs`: the segments follow one another on one stream, each leaves its best entry of a row in `seg_best` [segs][n_want] and the last
// one has the row's.
__global__ void __launch_bounds__(512) finish_rows_kernel(float* logits, int V, int n_want, int parts, float scale, float cap, const StepOut* __restrict__ to,
                                                          const int* __restrict__ err, int c0, int c1, int seg, int segs, float2* __restrict__ seg_best) {
  pdl_enter();
  __shared__ float bv[32];
  __shared__ int bi[32];
  const size_t m = blockIdx.x / parts;
  const int rank = blockIdx.x % parts;
  const float* r = logits + m * V;
  const StepOut so = *to;
  float* w = so.logits ? so.logits + m * V : nullptr;
  float best = -INFINITY;
  int idx = 0x7fffffff;
  auto finish = [&](float v) { v *= scale; return cap > 0.f ? cap * tanhf(v / cap) : v; };
  auto take = [&](float v, int i) { if (v > best || (v == best && i < idx)) { best = v; idx = i; } };
  const bool change = scale != 1.0f || cap > 0.f, write = w && (change || w != r);
  constexpr int NV = 4;                                        // 16-byte loads in flight per thread
  const int per = ((c1 - c0 + 3) / 4 + parts - 1) / parts * 4, v0 = min(c1, c0 + rank * per), v1 = min(c1, v0 + per);   // this block's stretch, from a piece of four on (c0 is one)
  int done = v0;
  if (((reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(w)) & 15) == 0) {
    done = v0 + ((v1 - v0) & ~3);
    for (int i0 = v0 + threadIdx.x * 4; i0 < done; i0 += blockDim.x * 4 * NV) {
      float4 q[NV];
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        const int i = i0 + u * (int)blockDim.x * 4;
        if (i < done) q[u] = *reinterpret_cast<const float4*>(r + i);
      }
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        const int i = i0 + u * (int)blockDim.x * 4;
        if (i >= done) continue;
        if (change) q[u] = make_float4(finish(q[u].x), finish(q[u].y), finish(q[u].z), finish(q[u].w));
        if (write) *reinterpret_cast<float4*>(w + i) = q[u];
        take(q[u].x, i); take(q[u].y, i + 1); take(q[u].z, i + 2); take(q[u].w, i + 3);
      }
    }
  }
  for (int i = done + threadIdx.x; i < v1; i += blockDim.x) {
    float v = r[i];
    if (change) v = finish(v);
    if (write) w[i] = v;
    take(v, i);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
  }
  if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int u = 1; u < (int)(blockDim.x >> 5); ++u)
      if (bv[u] > best || (bv[u] == best && bi[u] < idx)) { best = bv[u]; idx = bi[u]; }
    bv[0] = best;
    bi[0] = idx;
  }
  if (parts > 1) {
    xb::cluster_sync_all();
    if (rank == 0 && threadIdx.x == 0) {
      for (int u = 1; u < parts; ++u) {
        const float ov = ld_dsmem_f32(xb::smem_u32(bv), u);
        const int oi = __float_as_int(ld_dsmem_f32(xb::smem_u32(bi), u));
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
      }
    }
    xb::cluster_sync_all();                                    // nobody's shared memory goes away while it is read
  }
  if (rank == 0 && threadIdx.x == 0) {
    if (segs > 1) {
      if (seg + 1 < segs) { seg_best[(size_t)seg * n_want + m] = make_float2(best, __int_as_float(idx)); return; }
      for (int u = 0; u < seg; ++u) {
        const float2 o = __ldcg(seg_best + (size_t)u * n_want + m);
        const int oi = __float_as_int(o.y);
        if (o.x > best || (o.x == best && oi < idx)) { best = o.x; idx = oi; }
      }
    }
    so.tail[m] = idx;
    if (m == 0) so.tail[n_want] = *err;
  }
}

}  // namespace xl
