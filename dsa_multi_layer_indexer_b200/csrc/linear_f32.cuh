// y_i = x W_i^T in fp32 for up to three weights that read the same x, one launch; or, as `swiglu`,
// y = silu(x W_0^T) * (x W_1^T). The projections of a small fp32 layer (src/lagged_indexer_dsa/
// dsa_layer.py:87-143, :194-196), where the library's GEMMs are launch- and latency-bound: a few dozen
// CTAs of 7-8 us each, nine launches a layer.
//
// 64 x 32 output tiles of 4 x 4 outputs per thread (rows ty + 16 i, columns tx + 8 j: the 16-byte reads
// of a warp fall into distinct banks). Small tiles because the matrices are small: 1024 x 192 x 256 is 96
// tiles, less than one per SM, so the inner dimension is split inside the CTA: four groups of 128 threads
// (two for `swiglu`) take a part of every 64-deep slice each, 16 warps per SM instead of 4 to hide the
// shared-memory reads' latency, and their sums are folded in order at the end. Slices of x and W are brought in by
// 16-byte asynchronous copies, three in flight. Bound: shared-memory reads (eight 16-byte reads per 64
// multiply-adds) and, at one tile per SM, the slices' latency; larger products stay with the library.
// In a 1024-row forward of the small preset, per launch: k = 512, 256 columns 20.5 us with one group and 32-deep
// slices -> 12.2; three weights of 224 columns 18.7 -> 11; 16 warps at 64 registers instead of 122: 21.8.
// `swiglu` (2 x 512 columns) 20 us either way: two groups are as fast as four (one CTA per SM, two waves).
#pragma once

#include "common.cuh"

namespace dsa {
namespace lin {

constexpr int kBM = 64, kBN = 32, kBK = 64, kStages = 3;
constexpr int kGroup = 128;  // threads that cover a tile
template <bool kSwiglu>  // groups, which share a slice's depth (two matrices' sums leave registers for two at two CTAs per SM)
__host__ __device__ constexpr int groups() { return kSwiglu ? 2 : 4; }
constexpr int kPitch = kBK + 4;
template <bool kSwiglu>
__host__ __device__ constexpr int stage_floats() { return (kBM + (kSwiglu ? 2 : 1) * kBN) * kPitch; }
template <bool kSwiglu>
constexpr size_t smem_bytes() { return size_t(kStages) * stage_floats<kSwiglu>() * 4; }

// 16 bytes global -> shared, zeros when !ok (the source address must be valid all the same).
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

struct Params {
  const float* x;
  const float* w[3];
  float* y[3];
  int n[3];
  int tiles[3];  // column tiles of each output
  int64_t m;
  int k, count;
};

template <bool kSwiglu>
__global__ void __launch_bounds__(kGroup * groups<kSwiglu>(), kSwiglu ? 2 : 1)
linear_f32_kernel(const Params p) {
  constexpr int NB = kSwiglu ? 2 : 1, kGroups = groups<kSwiglu>(), kThreads = kGroup * kGroups;
  extern __shared__ __align__(16) float s_lin[];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, group = tid / kGroup, gt = tid % kGroup, tx = gt & 7, ty = gt >> 3;
  int t = blockIdx.y, n = p.n[0];
  const float* w0 = p.w[0];
  float* y = p.y[0];
  if (!kSwiglu && t >= p.tiles[0]) {  // (the parameters are only indexed by constants)
    t -= p.tiles[0], n = p.n[1], w0 = p.w[1], y = p.y[1];
    if (p.count > 2 && t >= p.tiles[1]) t -= p.tiles[1], n = p.n[2], w0 = p.w[2], y = p.y[2];
  }
  const int n0 = t * kBN;
  const int64_t m0 = int64_t(blockIdx.x) * kBM;
  const float* wm[2] = {w0, p.w[1]};
  const int slices = (p.k + kBK - 1) / kBK;
  auto fetch = [&](int sl) {
    if (sl < slices) {
      float* st = s_lin + (sl % kStages) * stage_floats<kSwiglu>();
      constexpr int kChunks = (kBM + NB * kBN) * (kBK / 4);
#pragma unroll
      for (int c0 = 0; c0 < kChunks; c0 += kThreads) {
        const int c = c0 + tid;
        if (kChunks % kThreads != 0 && c >= kChunks) break;
        const int row = c / (kBK / 4), kc = sl * kBK + (c % (kBK / 4)) * 4;
        const bool is_x = row < kBM;
        const int64_t gr = is_x ? m0 + row : int64_t(n0 + (row - kBM) % kBN);
        const float* base = is_x ? p.x : wm[NB > 1 && row >= kBM + kBN ? 1 : 0];
        const bool ok = kc < p.k && (is_x ? gr < p.m : gr < n);
        cp_async16_zfill(smem_u32(st + row * kPitch + (c % (kBK / 4)) * 4), ok ? base + gr * p.k + kc : base, ok);
      }
    }
    cp_async_commit();  // (an empty group past the end keeps the count)
  };
  float acc[NB][4][4] = {};
#pragma unroll
  for (int sl = 0; sl < kStages - 1; ++sl) fetch(sl);
  for (int sl = 0; sl < slices; ++sl) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // slice sl is there; the buffer of slice sl - 1 has been read
    fetch(sl + kStages - 1);
    const float* sa = s_lin + (sl % kStages) * stage_floats<kSwiglu>() + group * (kBK / kGroups);
    const float* sb = sa + kBM * kPitch;
#pragma unroll
    for (int kk = 0; kk < kBK / kGroups; kk += 4) {
      float4 av[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4*>(sa + (ty + 16 * i) * kPitch + kk);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 w = *reinterpret_cast<const float4*>(sb + (b * kBN + tx + 8 * j) * kPitch + kk);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            acc[b][i][j] = fmaf(av[i].x, w.x, acc[b][i][j]);
            acc[b][i][j] = fmaf(av[i].y, w.y, acc[b][i][j]);
            acc[b][i][j] = fmaf(av[i].z, w.z, acc[b][i][j]);
            acc[b][i][j] = fmaf(av[i].w, w.w, acc[b][i][j]);
          }
        }
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();  // the slices have been read: their memory takes the other groups' sums, [group - 1][value][thread]
  constexpr int kVals = NB * 16;
  static_assert((kGroups - 1) * kVals * kGroup <= kStages * stage_floats<kSwiglu>(), "linear: sums do not fit");
  if (group > 0) {
    float* dst = s_lin + (group - 1) * kVals * kGroup + gt;
#pragma unroll
    for (int v = 0; v < kVals; ++v) dst[v * kGroup] = acc[v / 16][v / 4 % 4][v % 4];
  }
  __syncthreads();
  if (group > 0) return;
#pragma unroll
  for (int g = 0; g < kGroups - 1; ++g)
#pragma unroll
    for (int v = 0; v < kVals; ++v) acc[v / 16][v / 4 % 4][v % 4] += s_lin[(g * kVals + v) * kGroup + gt];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t m = m0 + ty + 16 * i;
    if (m >= p.m) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx + 8 * j;
      if (c >= n) break;
      float v = acc[0][i][j];
      if constexpr (kSwiglu) v = __fmul_rn(v / (1.f + expf(-v)), acc[NB - 1][i][j]);
      y[m * n + c] = v;
    }
  }
}

}  // namespace lin
}  // namespace dsa
