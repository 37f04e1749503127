// layered_fma.cuh — products of the all-32-bit mode: C[z][m, n] = sum_k A[z][m, k] * B[z][n, k], fp32 operands, true fp32 FMA.
//
// One CTA = 8 * RM rows x 64 columns, 128 threads, a thread RM x 4 outputs.  Both operands come as they lie (K-major) by 16-byte cp.async into
// a ring of 32-wide K blocks; a thread reads four k of a row per 16-byte shared-memory load (RM + 4 loads for 16 RM FMAs), so the FMA pipes and
// not shared memory set the pace.  RM (2 .. 12) is chosen so that few rows of the last row tile are empty.  K is cut over the CTAs of a
// cluster (gridDim.x, up to 8) while two CTAs per SM are not exceeded: a product of some ten rows is bound by reading B, and a narrow one has
// only N / 64 column tiles.  The partial tiles meet through distributed shared memory, added in the order of K (deterministic).
// Operands whose rows are not whole 16-byte pieces stay with gemm_tiled_kernel.
// Measured (B200, some 70 rows, width 1024): gemm_tiled_kernel 247 / 201 us a launch, this kernel 73 / 80; its error against 64 bits 2e-6 -> 8.5e-7
// (shorter partial sums).
#pragma once
#include "layered_stream.cuh"

namespace xl {

constexpr int FMA_THREADS = 128, FMA_BN = 64, FMA_BK = 32, FMA_LD = FMA_BK + 4, FMA_STAGES = 3, FMA_PLD = FMA_BN + 4;
__host__ __device__ constexpr int fma_smem_bytes(int rm) { return FMA_STAGES * (8 * rm + FMA_BN) * FMA_LD * 4; }
static_assert(8 * 12 * FMA_PLD <= FMA_STAGES * (8 * 12 + FMA_BN) * FMA_LD && 8 * 2 * FMA_PLD <= FMA_STAGES * (8 * 2 + FMA_BN) * FMA_LD, "the partial tile reuses the ring");

// 16 bytes global -> shared memory; zeros when `on` is false (the address is then not read)
__device__ __forceinline__ void cp_async16_zfill(float* dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}

template <int RM, int EPI>
__global__ void __launch_bounds__(FMA_THREADS)
gemm_fma_kernel(const float* __restrict__ A, long lda, long a_batch, const float* __restrict__ B, long ldb, long b_batch, float* __restrict__ C, long ldc,
                long c_batch, int M, int N, int K, int n_tiles, const EpiArgs epi) {
  extern __shared__ __align__(16) float fma_sm[];
  constexpr int BM = 8 * RM, STAGE = (BM + FMA_BN) * FMA_LD;
  pdl_enter();
  const int S = gridDim.x, split = blockIdx.x, n0 = blockIdx.y % n_tiles * FMA_BN, m0 = blockIdx.y / n_tiles * BM;
  A += (size_t)blockIdx.z * a_batch;
  B += (size_t)blockIdx.z * b_batch;
  C += (size_t)blockIdx.z * c_batch;
  const int nkb = (K + FMA_BK - 1) / FMA_BK, per = (nkb + S - 1) / S, kb0 = min(nkb, split * per), nk = min(nkb, kb0 + per) - kb0;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;   // columns tx + 16 j, rows ty + 8 i
  // a thread copies the same 16-byte column of rows r0, r0 + 16, ... of both tiles
  const int c4 = (tid & 7) * 4, r0 = tid >> 3;
  constexpr int NL = (BM + FMA_BN) / 16;
  const float* src[NL];
  bool on[NL];
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    const int r = r0 + 16 * i;
    if (r < BM) {
      on[i] = m0 + r < M;
      src[i] = A + (size_t)(on[i] ? m0 + r : 0) * lda;
    } else {
      const int n = n0 + r - BM;
      on[i] = n < N;
      size_t row = on[i] ? n : 0;
      if constexpr (epi_is_glu(EPI)) row = row & 1 ? glu_up_row((int)row >> 1, N >> 1, epi.il8) : glu_gate_row((int)row >> 1, N >> 1, epi.il8);
      src[i] = B + row * ldb;
    }
  }
  auto issue = [&](int i) {
    float* dst = fma_sm + (size_t)(i % FMA_STAGES) * STAGE + r0 * FMA_LD + c4;
    const int k = (kb0 + i) * FMA_BK + c4;
#pragma unroll
    for (int l = 0; l < NL; ++l) cp_async16_zfill(dst + l * 16 * FMA_LD, src[l] + (k < K ? k : 0), on[l] && k < K);
  };
  float acc[RM][4];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int i = 0; i < FMA_STAGES - 1; ++i) {
    if (i < nk) issue(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FMA_STAGES - 2) : "memory");
    __syncthreads();                                           // block `it` is there; everybody is done with the buffer refilled next
    if (it + FMA_STAGES - 1 < nk) issue(it + FMA_STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = fma_sm + (size_t)(it % FMA_STAGES) * STAGE + ty * FMA_LD;
    const float* bs = fma_sm + (size_t)(it % FMA_STAGES) * STAGE + (BM + tx) * FMA_LD;
#pragma unroll
    for (int k = 0; k < FMA_BK; k += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(bs + j * 16 * FMA_LD + k);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(as + i * 8 * FMA_LD + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, acc[i][j]))));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* part = fma_sm;                                           // [BM][FMA_PLD]
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) part[(ty + 8 * i) * FMA_PLD + tx + 16 * j] = acc[i][j];
  __syncthreads();
  if (S > 1) xb::cluster_sync_all();
  float ap = 0.f, aq = 0.f;
  if (EPI == EPI_XIELU) { ap = softplusf_(static_cast<const float*>(epi.p)[0]); aq = 0.5f + softplusf_(static_cast<const float*>(epi.p)[1]); }
  const uint32_t part_addr = xb::smem_u32(part);
  auto total = [&](int m, int c) {                             // sum of the cluster's partial tiles, in the order of K: all loads under way before the first sum
    if (S == 1) return part[m * FMA_PLD + c];
    float p[8], v = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < S) p[r] = ld_dsmem_f32(part_addr + (uint32_t)(m * FMA_PLD + c) * 4, r);
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < S) v += p[r];
    return v;
  };
  const int rows = min(BM, M - m0);
  constexpr int W = epi_is_glu(EPI) ? FMA_BN / 2 : FMA_BN;
  for (int i = tid; i < (rows - split + S - 1) / S * W; i += FMA_THREADS) {
    const int r = split + i / W * S, c = i % W;
    const size_t m = m0 + r;
    if constexpr (epi_is_glu(EPI)) {                           // gate and up columns in turn
      if (n0 + 2 * c + 1 < N) C[m * ldc + (n0 >> 1) + c] = glu_f<EPI>(total(r, 2 * c), total(r, 2 * c + 1), epi);
    } else if (n0 + c < N) {
      float v = total(r, c);
      if constexpr (EPI == EPI_CLOSE) {
        stream_close<float>(epi, m, n0 + c, v);
      } else {
        if (EPI == EPI_RELU2) { v = fmaxf(v, 0.f); v *= v; }
        if (EPI == EPI_XIELU) v = xielu_f(v, ap, aq);
        if (EPI == EPI_GELU) v = gelu_erf_f(v);
        C[m * ldc + n0 + c] = v;
      }
    }
  }
  if (S > 1) {
    __syncthreads();
    xb::cluster_sync_all();                                    // nobody's shared memory goes away while a peer reads it
  }
}

}  // namespace xl
