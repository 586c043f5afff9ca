// Exact top-k of MANY short rows (a prompt's indexer: one row per token, up to 8192 logits, no
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
constexpr int64_t kRowsMaxN = 8192;  // 256 threads x 32 logits

// A NaN takes a rank above every number, as in topk_cluster_kernel, but is never selected: the places that this
// leaves are padding. (The bits of a NaN behind an addition are the compiler's choice: it is asked for by value.)
constexpr uint32_t kNanKey = 0xFFFFFFFFu;

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
__global__ void __launch_bounds__(T, T < 256 ? 8 : ITEMS > 16 ? 3 : ITEMS > 8 ? 4 : 6)
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
  const bool take_all = len <= p.topk;
  bool nan = false;
  if (take_all) {  // every visible number is kept, in place unless there is a NaN among them
    for (int i = tid; i < len; i += T) {
      const float v = row[i];
      nan |= v != v;
      emit(uint32_t(i), i, v == neg_inf);
    }
    pad_from(uint32_t(len));
    if (!__syncthreads_or(nan)) return;
  }
  const int base = warp * (32 * ITEMS) + lane;
  // keys, not values, stay in registers; 0 (below every number) past the row's length
  uint32_t key[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const float v = base + 32 * i < len ? row[base + 32 * i] : 0.f;
    nan |= v != v;
    key[i] = base + 32 * i < len ? ordered_key(v) : 0u;
  }
  // (a row with NaNs takes a detour at either end; telling them by value there only leaves one compare per logit
  // to the others: 297 rows of 6144 18.1 us, 21.7 with a NaN's key in the loops)
  const bool nans = __syncthreads_or(nan);  // and the histogram is clear
  if (nans) {
#pragma unroll 1
    for (int i = 0; i < ITEMS; ++i) {
      const bool is_nan = base + 32 * i < len && row[base + 32 * i] != row[base + 32 * i];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (j == i && is_nan) key[j] = kNanKey;
    }
  }
  uint32_t kstar = 0u, ties_kept = 0u;  // (take_all: whatever is above 0)
  if (!take_all) {
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
    kstar = (p22 << 10) | s_res[0];
    ties_kept = s_res[1];
  }
  if (nans) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (key[i] == kNanKey) key[i] = 0u;
  }

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
  const uint32_t all = __reduce_add_sync(0xffffffffu, wt), total = (all & 0xFFFFu) + min(all >> 16, ties_kept);
  if (total < uint32_t(p.topk)) pad_from(total);
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

// ------------------------------------------------------------------------------
// One row of up to kSoloMaxN logits that comes with the scan's histogram (a decode step at a short
// context): one CTA of 512 threads with the row in registers. The cluster kernel's way for such a row is a
// chain of phases laid out for 32 logits per thread and eight CTAs; here
//   threshold bin from the histogram -> candidates of that bin counted by their next 7 key bits -> the
//   second bin -> the few candidates in it ("survivors") ranked by comparison (key descending, position
//   ascending) -> one pass of warp votes in position order gives each kept element its slot,
// and candidates never leave their owner. More than kSoloSurv survivors (many equal logits): two more
// counting rounds down to the k-th key, ties resolved in position order in the last pass.
// Latency-bound: about a dozen dependent steps, and the unrolled code itself. scan + top-k of 4096 logits,
// k = 2048: 9.3 -> 7.3 us; with 16 elements per thread (8192 logits) it is no faster than the cluster
// kernel for one row and slower for eight (15.3 against 13.0 us), with 32 slower for one; the same kernel
// with its elements in shared memory and rolled loops: 8.0 us at 4096, 14.8 at 16384. Hence the limit.
constexpr int kSoloSurv = 256;
constexpr int64_t kSoloMaxN = 4096;
template <int ITEMS, bool kPages>
__global__ void __launch_bounds__(kClThreads)
topk_solo_kernel(const Params p) {
  __shared__ uint32_t s_warp[kClWarps];
  __shared__ uint32_t s_res[4];
  __shared__ __align__(16) uint32_t s_h2[kL2Bins];
  __shared__ uint32_t s_mask[kClWarps * ITEMS];  // survivors that are kept, word (warp, i), bit lane
  __shared__ uint64_t s_surv[kSoloSurv];
  __shared__ uint32_t s_nsurv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r = blockIdx.x;
  for (int i = tid; i < kClWarps * ITEMS; i += kClThreads) s_mask[i] = 0u;
  if (tid < kL2Bins) s_h2[tid] = 0u;
  if (tid == 0) s_nsurv = 0u, s_res[3] = 0u;
  DSA_KTIME_BEGIN(1);
  pdl_launch_dependents();  // (before the wait, as the cluster kernel does: see there)
  pdl_wait();
  const float* row = p.logits + r * p.slab_stride;
  const int base = warp * (32 * ITEMS) + lane;   // element i of this thread is position base + 32 i
  const int n = int(p.n);
  uint32_t key[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) key[i] = base + 32 * i < n ? __float_as_uint(__ldcg(row + base + 32 * i)) : 0xFFFFFFFFu;
  uint4* gh = reinterpret_cast<uint4*>(p.hist + size_t(r) * kBins + (kBins - 8 * (tid + 1)));
  const uint4 h1a = __ldcg(gh), h1b = __ldcg(gh + 1);
  int64_t len64 = p.seq_lens ? int64_t(p.seq_lens[r]) : p.n;
  const int len = int(len64 < 0 ? 0 : (len64 > p.n ? p.n : len64));
  int32_t page[ITEMS / 2];                       // kPages: one table entry per two groups of 32 positions
  if constexpr (kPages) {
#pragma unroll
    for (int i = 0; i < ITEMS / 2; ++i) {
      const int first = warp * (32 * ITEMS) + 64 * i;
      page[i] = first < n ? p.page_table[r * p.pt_stride + (first >> 6)] : 0;
    }
  }
  // ordered keys; 0 (below every number) for NaNs and past the row's length
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const float v = __uint_as_float(key[i]);
    key[i] = base + 32 * i < len && v == v ? ordered_key(v) : 0u;
  }
  gh[0] = make_uint4(0, 0, 0, 0);                // re-armed: every thread clears the bins that it has read
  gh[1] = make_uint4(0, 0, 0, 0);

  uint32_t kept = 0;                             // bit i: key[i] is certainly kept
  uint32_t kstar = 0xFFFFFFFFu, ties_kept = 0;
  bool pad_inf = true;                           // a kept -inf can only appear when the row has fewer than k finite logits
  if (len <= p.topk) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (key[i] != 0u) kept |= 1u << i;
    __syncthreads();
  } else {
    const uint32_t cnt8[8] = {h1b.w, h1b.z, h1b.y, h1b.x, h1a.w, h1a.z, h1a.y, h1a.x};  // highest bin first
    find_kth_in_registers<kBins, 8>(cnt8, uint32_t(p.topk), s_warp, s_res);
    const uint32_t T = s_res[0], need = s_res[1];
    uint32_t cand = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint32_t bin = key[i] >> kLowBits;
      if (key[i] != 0u && bin > T) kept |= 1u << i;
      if (key[i] != 0u && bin == T) {
        cand |= 1u << i;
        smem_red_add(&s_h2[(key[i] >> kL3Bits) & (kL2Bins - 1)], 1u);
      }
    }
    __syncthreads();
    find_kth_bin_warp<kL2Bins>(s_h2, need, s_res);
    const uint32_t p19 = (T << kL2Bits) | s_res[0], need2 = s_res[1];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if ((cand >> i) & 1u) {
        const uint32_t k19 = key[i] >> kL3Bits;
        if (k19 > p19) kept |= 1u << i;
        if (k19 == p19) {
          const uint32_t at = atomicAdd(&s_nsurv, 1u);
          if (at < uint32_t(kSoloSurv)) s_surv[at] = (uint64_t(key[i]) << 32) | uint32_t(~uint32_t(base + 32 * i));
        }
      }
    }
    __syncthreads();
    const uint32_t n_surv = s_nsurv;
    if (n_surv <= uint32_t(kSoloSurv)) {
      if (uint32_t(tid) < n_surv) {
        const uint64_t mine = s_surv[tid];       // larger = earlier
        uint32_t before = 0;
        for (uint32_t j = 0; j < n_surv; ++j) before += uint32_t(s_surv[j] > mine);
        const uint32_t pos = ~uint32_t(mine);
        if (before < need2) atomicOr(&s_mask[pos >> 5], 1u << (pos & 31u));
        if (before + 1u == need2) s_res[3] = uint32_t(mine >> 32);
      }
      __syncthreads();
      pad_inf = s_res[3] <= 0x007FFFFFu;
    } else {                                     // many equal logits: down to the k-th key itself
      uint32_t prefix = p19, left = need2;
#pragma unroll 1
      for (int shift = 6; shift >= 0; shift -= 6) {  // 7 bits, then 6
        const int bits = shift == 6 ? 7 : 6;
        if (tid < kL2Bins) s_h2[tid] = 0u;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
          hist_add_warp(s_h2, ((cand >> i) & 1u) && (key[i] >> (shift + bits)) == prefix, (key[i] >> shift) & ((1u << bits) - 1u));
        __syncthreads();
        find_kth_bin_warp<kL2Bins>(s_h2, left, s_res);
        prefix = (prefix << bits) | s_res[0];
        left = s_res[1];
      }
      kstar = prefix;
      ties_kept = left;
      pad_inf = kstar <= 0x007FFFFFu;
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (((cand >> i) & 1u) && key[i] > kstar) kept |= 1u << i;
    }
  }
  // ---- totals of the warps' shares, then the slots in position order
  uint32_t cnt = uint32_t(__popc(kept));
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) cnt += (key[i] == kstar ? 0x10000u : 0u);
  if (lane < ITEMS) cnt += uint32_t(__popc(s_mask[warp * ITEMS + lane]));
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) s_warp[warp] = cnt;
  __syncthreads();
  const uint32_t wt = lane < kClWarps ? s_warp[lane] : 0u;
  const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u), all = __reduce_add_sync(0xffffffffu, wt);
  uint32_t g = before & 0xFFFFu, q = before >> 16;
  const uint32_t below = (1u << lane) - 1u;
  int32_t* out_idx = p.out_idx + r * p.topk;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t gm = __ballot_sync(0xffffffffu, (kept >> i) & 1u) | s_mask[warp * ITEMS + i];
    const uint32_t qm = ties_kept ? __ballot_sync(0xffffffffu, key[i] == kstar) : 0u;
    const uint32_t gb = g + __popc(gm & below), qb = q + __popc(qm & below);
    const bool is_g = (gm >> lane) & 1u, is_q = ((qm >> lane) & 1u) && qb < ties_kept;
    if (is_g || is_q) {
      const int pos = base + 32 * i;
      int32_t id = pos + p.index_offset;
      if constexpr (kPages) id = page[i >> 1] * DSA_PAGE_TOKENS + (pos & (DSA_PAGE_TOKENS - 1));
      if (pad_inf && key[i] == 0x007FFFFFu) id = p.pad;
      out_idx[is_g ? gb + min(qb, ties_kept) : gb + qb] = id;
    }
    g += __popc(gm);
    q += __popc(qm);
  }
  for (uint32_t i = (all & 0xFFFFu) + min(all >> 16, ties_kept) + tid; i < uint32_t(p.topk); i += kClThreads) out_idx[i] = p.pad;
  DSA_KTIME_END(1);
}

}  // namespace topk
}  // namespace dsa
