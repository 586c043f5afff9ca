// Exact top-k of MANY short rows (a prompt's indexer: one row per token, up to 16384 logits, no
// histogram from the scan): one small CTA per row instead of the cluster kernel's 512 threads and
// 192 KB of shared memory, so that several rows share an SM and hide one another's latencies.
//
// Same contract as topk_cluster_kernel (topk_select.cuh): the k largest of the row's first seq_lens[r]
// logits, ties to the lower position, ascending positions, padding behind them. The row sits in
// registers, warp w holding the contiguous positions [w * 32 * ITEMS, ...) as (i, lane); three radix
// levels over the order-preserving key (11 + 11 + 10 bits, shared-memory histograms: only elements that
// share the prefix found so far add) give the k-th key k* and how many of the elements equal to it are
// kept; one pass of warp votes in position order then gives each kept element its slot. Rows that are
// no longer than k go out as they are.
//
// What bounds it: instruction issue and the shared-memory atomics of the first level (one per logit).
// 1024 rows of up to 512 logits, k = 16: 8 us against 45; 4099 rows of up to 4099 logits, k = 2048: 149 us
// against 226 (both against the cluster kernel).
#pragma once

#include "topk_select.cuh"

namespace dsa {
namespace topk {

constexpr int kRowsBins = 2048;
constexpr int64_t kRowsMaxN = 16384;  // 512 threads x 32 logits

// Bin (from the top) that holds the k-th largest of an NB-bin histogram; thread t owns the NB / T bins
// below NB - t * NB / T. s_res: bin, rank inside it. Every thread calls it; ends with a barrier.
template <int T, int NB>
__device__ __forceinline__ void rows_find_bin(const uint32_t* h, uint32_t k, uint32_t* s_warp, uint32_t* s_res) {
  constexpr int PER = NB / T;
  static_assert(PER * T == NB, "whole bins per thread");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t cnt[PER];  // highest bin first
  const uint32_t* mine = h + NB - PER * (tid + 1);
#pragma unroll
  for (int i = 0; i < PER; ++i) cnt[i] = mine[PER - 1 - i];
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) s += cnt[i];
  const uint32_t inc = warp_inclusive_scan(s);
  if (lane == 31) s_warp[warp] = inc;
  if (tid == 0) s_res[0] = 0u, s_res[1] = 1u;  // stays if the row holds fewer than k numbers (NaNs)
  __syncthreads();
  const uint32_t wt = lane < T / 32 ? s_warp[lane] : 0u;
  const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
  uint32_t running = before + inc - s;
  if (running < k && k <= running + s) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (running < k && k <= running + cnt[i]) {
        s_res[0] = uint32_t(NB - 1 - PER * tid - i);
        s_res[1] = k - running;
      }
      running += cnt[i];
    }
  }
  __syncthreads();
}

template <int T, int ITEMS>
__global__ void __launch_bounds__(T, T > 256 ? 1 : T < 256 ? 8 : ITEMS > 16 ? 3 : ITEMS > 8 ? 4 : 6)
topk_rows_kernel(const Params p) {
  constexpr int kWarps = T / 32;
  __shared__ __align__(16) uint32_t s_hist[kRowsBins];
  __shared__ uint32_t s_warp[kWarps];
  __shared__ uint32_t s_res[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r = blockIdx.x;
  auto clear = [&]() {
    for (int i = tid; i < kRowsBins / 4; i += T) reinterpret_cast<uint4*>(s_hist)[i] = make_uint4(0, 0, 0, 0);
  };
  clear();
  pdl_wait();
  pdl_launch_dependents();
  int64_t len64 = p.seq_lens ? int64_t(p.seq_lens[r]) : p.n;
  const int len = int(len64 < 0 ? 0 : (len64 > p.n ? p.n : len64));
  const float* row = p.logits + r * p.slab_stride;
  int32_t* out_idx = p.out_idx + r * p.topk;
  float* out_val = p.out_val ? p.out_val + r * p.topk : nullptr;
  const int32_t* imap = p.index_map ? p.index_map + r * p.n : nullptr;
  const float neg_inf = __int_as_float(0xff800000);
  auto emit = [&](uint32_t slot, int pos, bool is_neg_inf) {
    out_idx[slot] = is_neg_inf ? p.pad : imap ? imap[pos] : pos + p.index_offset;
    if (out_val) out_val[slot] = row[pos];
  };
  auto pad_from = [&](uint32_t first) {
    for (uint32_t i = first + tid; i < uint32_t(p.topk); i += T) {
      out_idx[i] = p.pad;
      if (out_val) out_val[i] = neg_inf;
    }
  };
  if (len <= p.topk) {  // every visible key is kept, in place
    for (int i = tid; i < len; i += T) emit(uint32_t(i), i, row[i] == neg_inf);
    pad_from(uint32_t(len));
    return;
  }
  const int base = warp * (32 * ITEMS) + lane;
  // keys, not values, stay in registers; 0 (below every number) past the row's length
  uint32_t key[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) key[i] = base + 32 * i < len ? ordered_key(row[base + 32 * i]) : 0u;
  __syncthreads();  // the histogram is clear
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    hist_add_warp(s_hist, key[i] != 0u, key[i] >> 21);
  __syncthreads();
  rows_find_bin<T, kRowsBins>(s_hist, uint32_t(p.topk), s_warp, s_res);
  const uint32_t b1 = s_res[0];
  uint32_t need = s_res[1];
  clear();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) hist_add_warp(s_hist, key[i] != 0u && (key[i] >> 21) == b1, (key[i] >> 10) & 2047u);
  __syncthreads();
  rows_find_bin<T, kRowsBins>(s_hist, need, s_warp, s_res);
  const uint32_t p22 = (b1 << 11) | s_res[0];
  need = s_res[1];
  clear();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) hist_add_warp(s_hist, key[i] != 0u && (key[i] >> 10) == p22, key[i] & 1023u);
  __syncthreads();
  rows_find_bin<T, 1024>(s_hist, need, s_warp, s_res);
  const uint32_t kstar = (p22 << 10) | s_res[0];
  const uint32_t ties_kept = kstar ? s_res[1] : 0u;  // (0: fewer than k numbers in the row, all of them kept)

  // (kept, tie) counts of the warps' shares in position order, then the slots
  uint32_t cnt = 0;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    cnt += (key[i] > kstar ? 1u : 0u) + (key[i] == kstar ? 0x10000u : 0u);
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  __syncthreads();  // (s_warp's readers in rows_find_bin are done)
  if (lane == 0) s_warp[warp] = cnt;
  __syncthreads();
  const uint32_t wt = lane < kWarps ? s_warp[lane] : 0u;
  const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
  if (kstar == 0u) pad_from(__reduce_add_sync(0xffffffffu, wt) & 0xFFFFu);
  uint32_t g = before & 0xFFFFu, q = before >> 16;
  const uint32_t below = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t gm = __ballot_sync(0xffffffffu, key[i] > kstar), qm = __ballot_sync(0xffffffffu, key[i] == kstar);
    if (gm | qm) {
      const uint32_t gb = g + __popc(gm & below), qb = q + __popc(qm & below);
      if ((gm >> lane) & 1u) emit(gb + min(qb, ties_kept), base + 32 * i, key[i] == 0x007FFFFFu);
      else if (((qm >> lane) & 1u) && qb < ties_kept) emit(gb + qb, base + 32 * i, key[i] == 0x007FFFFFu);
      g += __popc(gm);
      q += __popc(qm);
    }
  }
}

}  // namespace topk
}  // namespace dsa
