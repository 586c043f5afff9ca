// Sparse MLA of 128 heads, or of two rows' 64, on a pair of CTAs (tcgen05 with cta_group::2), bf16 rows.
//
// Same contract and the same partials as sparse_mla_tc.cuh. A persistent pair takes (row, 128 heads, split) triples in
// turn; 128-key tiles, 64 heads in each CTA:
//
//   S [128 heads x 128 keys]  = Q K^T   M = 128: each CTA its 64 heads; N = 128: each CTA brings 64 of the keys, all dims
//   O [128 heads x 512 dims] += P V     M = 128: each CTA its 64 heads; N = 256, twice: each CTA brings half of the value
//                                       dims of all 128 keys
//
// so an operand row is read from shared memory once for 128 heads, no score row is padding, and a CTA's accumulators (its
// 64 heads over 128 lanes: lane l has head l % 64, and keys or dims of half l / 64) take 64 + 256 columns of tensor memory.
// The other 192 hold the first six chunks of Q, in both lane halves. One S buffer is enough: the score product of tile t + 1
// is issued behind the value product of tile t - 1, by when the softmax has read S(t).
//
// What bounds it. The products of a tile take 2280 cycles (36 of 32.6 at M 128 N 128 K 16 and 16 of 68.9 at N 256, each measured
// alone). A tile takes 3300 - 3450 with up to 37 pairs at work and 3600 - 4000 with all 74 (times of 2048 and 4096 keys, at the
// clock sampled meanwhile): the products wait for rows and probabilities, and with all pairs at work the board's power limit
// also lowers the clock (1.6 GHz at 1000 W). 1024 rows of 128 heads x 2048 keys 803 -> 500 us, 700 x 700 250 -> 155 us (one CTA
// per 64 heads / this kernel). What it took:
//   * rows come by TMA row gathers (tile::gather4), four rows of one 64-dim chunk each. A gather costs a warp 35 - 60 cycles
//     behind other gathers and 85 - 140 where it waits, looks something up or shuffles indices in between, so a warp issues
//     eight in a row, from indices laid out in shared memory: 340 -> 270 cycles per 16 KB. (16-byte asynchronous copies with
//     the wait, fence and hand-over that they need: 705 us where gathers took 567);
//   * K and V of a tile are separate loads, although CTA 0 has half of its V among its K: both CTAs must have an operand at
//     the same offset, and at the offset of a K chunk the other CTA has another chunk;
//   * one ring of 16 KB units in the order of use, keys of tile t + 1 before values of tile t. A place is loaded again about
//     2400 cycles before it is needed, which the loads just meet: nine units and two S buffers 532, ten and one 514 us;
//   * the softmax takes S into registers and gives its buffer back at once, since the next score product waits for it: given
//     back behind the exponentials 523 us. The heads' maxima are compared only where one ran away;
//   * the MMA warp tests all its barriers in one look (a wait per unit, ready or not, took 200 cycles: 589 -> 548 us);
//   * arrivals at the other CTA's barriers without cluster scope (they order nothing but shared memory of the arriving CTA,
//     whose proxy fence precedes them): 1400 cycles each, twice a tile, before: 794 -> 580 us;
//   * result and partials leave through shared memory and TMA stores: 4 rows in 16 splits 18.0 -> 16.1 us.
// Tried: two softmax groups on alternate tiles (564 us: longer in total, and not what a tile waits for), eight gather warps
// (539), fp8 rows converted by the gather warps (32 rows 48.9 us against 45.8 with one CTA per 64 heads: of a tile's 17 chunks
// eight are converted a second time).
//
// kTwoRows: 64 heads. Neighbouring rows of a prompt that is no longer than the list attend the same keys, the second one
// its own as well: two rows' heads fill the pair's 128, with one list and each row's own view of what is masked. The plan
// compares the two lists entry by entry; rows that do not nest, or whose one key more is not finite, go through their
// own list alone, with the other CTA's result dropped. Prompt of 700 tokens 82 -> 61 us, 2048 465 -> 320 (four passes over
// each list with a few loads under way instead of one with sixteen: 127 us, the plan was what everything waited for).
//
// Warps (864 threads): 0-7 softmax, queries to tensor memory, result; 8 products (in CTA 0); 9 plans the triples and loads
// the rest of the queries; 10-25 gather; 26 lays out a tile's rows and gathers its last chunk.
#pragma once

#include "sparse_mla_tc.cuh"

namespace dsa {
namespace mla_pair {

constexpr int kHeads = 128;                    // heads of a pair
constexpr int kBN = 128;                       // keys per tile
constexpr int kChunkBytes = 64 * 128;          // [64 rows][64 dims] of bf16
constexpr int kUnitBytes = 2 * kChunkBytes;    // [2 chunks][64 rows][64 dims]
constexpr int kUnits = 10;                     // ring
constexpr int kQTmem = 6;                      // chunks of Q in tensor memory
constexpr int kGatherWarps = 16;               // and one for the rows of the tiles and their last chunk
constexpr int kSoftWarps = 8;                  // two per lane quadrant of tensor memory
constexpr int kMmaWarp = kSoftWarps, kPlanWarp = kSoftWarps + 1, kGatherWarp0 = kSoftWarps + 2;
constexpr int kThreads = 32 * (kGatherWarp0 + kGatherWarps + 1);
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0;                  // S: 64 columns
constexpr uint32_t kColO = 64;                 // O: 2 x 128 columns
constexpr uint32_t kColQ = 320;                // Q: kQTmem x 32 columns
constexpr int kLists = 4;                      // tiles whose rows are laid out
constexpr int kPlan = 4;                       // entries of the plan ring
constexpr float kRescaleLog2 = mla_tc::kRescaleLog2;
enum { kBoth = 0, kFirst = 1, kSecond = 2 };  // rows of a plan entry

// The first kNumPolled are what the MMA warp waits for.
enum {
  kBarFull = 0, kBarRope = kBarFull + kUnits, kBarSRead = kBarRope + 2, kBarP, kBarQ, kBarQT, kBarOFree, kNumPolled,
  kBarEmpty = kNumPolled, kBarRopeFree = kBarEmpty + kUnits, kBarQFree = kBarRopeFree + 2, kBarQStage, kBarS, kBarPV, kBarPlan,
  kBarList = kBarPlan + kPlan, kNumBars = kBarList + kLists
};

struct Smem {
  static constexpr int q_off = 0;                                        // chunks kQTmem.. of Q
  static constexpr int ring_off = q_off + (9 - kQTmem) * kChunkBytes;
  static constexpr int rope_off = ring_off + kUnits * kUnitBytes;        // two slots of a tile's last chunk
  static constexpr int p_off = rope_off + 2 * kChunkBytes;               // [2 key blocks][64 heads][64 keys] of bf16
  static constexpr int bar_off = p_off + 2 * kChunkBytes;
  static constexpr int tmem_off = bar_off + 8 * kNumBars;
  static constexpr int plan_off = (tmem_off + 4 + 15) & ~15;             // int4 [kPlan]: item, tiles, length, -
  static constexpr int list_off = plan_off + 16 * kPlan;                 // int [kLists][128]: rows of a tile's keys, -1 where masked
  static constexpr int seen_off = list_off + kLists * kBN * 4;           // uint32 [kLists][4]: which are not
  static constexpr int max_off = seen_off + kLists * 16;                 // float [4][64]
  static constexpr int sum_off = max_off + 1024;                         // float [4][64]
  static constexpr int bytes = sum_off + 1024 + 1024;                    // + slack for the 1024-byte alignment
};
static_assert(Smem::bytes <= 232448, "pair attention: shared memory over the per-CTA limit");

// ---- cta_group::2 forms
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_result_addr, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result_addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_free2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
// arrives at `bar` of both CTAs once every product issued so far is done
__device__ __forceinline__ void commit2(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(uint16_t(3))
               : "memory");
}
__device__ __forceinline__ void mma2(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma2_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Loads into this CTA whose bytes are counted at a barrier of either CTA of the pair.
__device__ __forceinline__ void gather4(uint32_t dst, const CUtensorMap* map, int x, int4 y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst), "l"(map), "r"(x), "r"(y.x), "r"(y.y), "r"(y.z), "r"(y.w), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// This warp's 32 lanes x 8 consecutive columns of tensor memory.
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// Named barrier 2 over the softmax warps, plain and with an OR reduction.
__device__ __forceinline__ void group_sync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }
__device__ __forceinline__ bool group_sync_or(bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 2, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(uint32_t(x))
      : "memory");
  return r != 0;
}

// [32 rows][64 bytes] of shared memory (64-byte swizzle) to global memory, and the waits for this thread's stores: until
// shared memory has been read, until all is written.
__device__ __forceinline__ void tma_store_2d(uint32_t src, const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y), "r"(src)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// A place in the ring: slot and the parity of its use.
struct Ring {
  int slot, phase;
  __device__ __forceinline__ void add(int n) {  // n <= kUnits
    slot += n;
    if (slot >= kUnits) slot -= kUnits, phase ^= 1;
  }
  __device__ __forceinline__ void add_many(int n) {
    phase ^= (n / kUnits) & 1;
    add(n % kUnits);
  }
};

// One past the last visible entry of list[k_begin, j0), or 0: a warp, 1024 entries at a time, all requested before the first is
// looked at. (One by one, a row of 40 keys in a list of 2048 took 12 us more; 256 at a time 0.9.) A function of its own:
// inlined, launches that never come here were up to 5 % slower (40 rows x 1024 keys 24.1 -> 25.1 us).
__device__ __noinline__ int end_of_list(const int32_t* list, int k_begin, int j0, int len) {
  const int lane = threadIdx.x & 31;
  int bound = 0;
  for (; j0 > k_begin && bound == 0; j0 -= 1024) {
    int idx[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      const int j = j0 - 32 * (c + 1) + lane;
      idx[c] = -1;
      if (j >= k_begin) idx[c] = list[j];
    }
#pragma unroll
    for (int c = 0; c < 32; ++c)
      if (uint32_t(idx[c]) < uint32_t(len)) bound = max(bound, j0 - 32 * (c + 1) + lane + 1);
    bound = __reduce_max_sync(0xffffffffu, bound);
  }
  return bound;
}

struct Params {
  mla::Params m;
  int items;  // (row, block of 128 heads, split) triples
};

template <bool kBeside, bool kTwoRows>
__global__ void __launch_bounds__(kThreads, 1)
sparse_mla_pair_kernel(const __grid_constant__ CUtensorMap kv_map, const __grid_constant__ CUtensorMap q_map,
                       const __grid_constant__ CUtensorMap out_map, const Params pp) {
  const mla::Params& p = pp.m;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t s_ring = sbase + Smem::ring_off, s_rope = sbase + Smem::rope_off, s_q = sbase + Smem::q_off, s_p = sbase + Smem::p_off;
  auto bar = [&](int i) { return sbase + Smem::bar_off + 8u * uint32_t(i); };
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + Smem::tmem_off);
  volatile float* s_max = reinterpret_cast<volatile float*>(smem + Smem::max_off);
  volatile float* s_sum = reinterpret_cast<volatile float*>(smem + Smem::sum_off);
  const int4* s_plan = reinterpret_cast<const int4*>(smem + Smem::plan_off);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int rank = int(cluster_cta_rank());
  const int cid = blockIdx.x >> 1, clusters = gridDim.x >> 1;
  DSA_KTIME_BEGIN(2);

  if (tid == 0) {
    for (int i = 0; i < kNumBars; ++i) {
      const bool softmax = i == kBarQT || i == kBarSRead || i == kBarP || i == kBarOFree;
      mbar_init(bar(i), softmax ? 2 * kSoftWarps : i == kBarQStage ? kQTmem / 2 : 1);
    }
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc2(smem_u32(const_cast<uint32_t*>(s_tmem)), kTmemCols);
    tmem_relinquish2();
  }
  if (warp == kPlanWarp && lane == 0) {
    prefetch_tensor_map(&kv_map);
    prefetch_tensor_map(&q_map);
    prefetch_tensor_map(&out_map);
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the peer's barriers exist, its tensor memory is allocated
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);
  const uint32_t leader_bars = cluster_map(bar(0), 0);
  auto leader_bar = [&](int i) { return leader_bars + 8u * uint32_t(i); };

  if constexpr (!kBeside) pdl_wait();
  pdl_launch_dependents();

  // r: the row (kTwoRows: the first of two rows, the second CTA has the other), heads0: this CTA's 64 heads among all rows'
  const int hps = kTwoRows ? 1 : p.H / kHeads;
  struct Item { int r, split, k_begin, k_end; int64_t heads0; bool second; };
  auto item_of = [&](int i) {
    Item it;
    it.split = i % p.nsplit;
    int u = pp.items / p.nsplit - 1 - i / p.nsplit;  // last rows first: those of a prompt grow
    it.second = true;
    if constexpr (kTwoRows) {
      const int per_seq = (p.rows_per_seq + 1) / 2, seq = u / per_seq;
      u -= seq * per_seq;
      it.r = seq * p.rows_per_seq + 2 * u;
      it.second = 2 * u + 1 < p.rows_per_seq;
      it.heads0 = (int64_t(it.r) + rank) * 64;
    } else {
      it.r = u / hps;
      it.heads0 = int64_t(it.r) * p.H + u % hps * kHeads + rank * 64;
    }
    it.k_begin = it.split * p.keys_per_split;
    it.k_end = min(it.k_begin + p.keys_per_split, p.topk);
    return it;
  };
  bool failed = false;
  // the plan's entry n: item (-1: no more), tiles, length of the row whose list counts, which rows (kBoth, kFirst, kSecond)
  auto next_plan = [&](int n, int4& e) {
    if (__any_sync(0xffffffffu, !mbar_wait(bar(kBarPlan + (n & (kPlan - 1))), (n / kPlan) & 1))) {
      failed = true;
      return false;
    }
    e = s_plan[n & (kPlan - 1)];
    e.x = __shfl_sync(0xffffffffu, e.x, 0), e.y = __shfl_sync(0xffffffffu, e.y, 0);
    e.z = __shfl_sync(0xffffffffu, e.z, 0), e.w = __shfl_sync(0xffffffffu, e.w, 0);
    return e.x >= 0;
  };

  if (warp < kSoftWarps) {
    // ===================================================================== softmax, rescale, epilogue
    // Lane l of tensor memory: head l % 64, keys [64 (l / 64), ..) of a tile, value dims [256 (l / 64), ..). Of those keys and
    // dims a warp takes the first or the second half.
    const int quad = warp & 3, half = quad >> 1, group = warp >> 2, head = (quad & 1) * 32 + lane;
    const int part = 2 * half + group;  // quarter of a tile's keys
    const uint32_t tq = tmem + (uint32_t(quad * 32) << 16), ts = tq + kColS + 32u * group;
    const uint32_t s_prow = s_p + uint32_t(half) * kChunkBytes + uint32_t(head) * 128;
    int gt = 0;
    // item n's queries into tensor memory, in both lane halves (a product reads the half that its columns go to); every
    // score product of the item before is done: its last scores have been read
    auto queries = [&](int n) {
      if (group_sync_or(!mbar_wait(bar(kBarQStage), n & 1))) { failed = true; return; }
      const int unit = kQTmem / 2 * n + 8 * gt;  // units before this item's
#pragma unroll 1
      for (int c = group; c < kQTmem; c += 2) {
        const uint8_t* row = smem + Smem::ring_off + (unit + c / 2) % kUnits * kUnitBytes + (c & 1) * kChunkBytes;
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 x = *reinterpret_cast<const uint4*>(row + mla_tc::swz(head, i));
          v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
        }
        tmem_st_32x32(tq + kColQ + 32u * c, v);
      }
      tmem_st_wait();
      tc_fence_before();
      group_sync();
      if (lane == 0) arrive_at(leader_bar(kBarQT));
    };
    // (a wait that ran out is voted on: the group's barriers need all of it)
    auto next_item = [&](int n, int4& e) {
      const bool more = next_plan(n, e);
      if (group_sync_or(failed)) { failed = true; return false; }
      if (more) queries(n);
      return more && !failed;
    };
    int4 e;
    bool more = next_item(0, e);
    for (int n = 0; more && !failed; ++n) {
      const int tiles = e.y;
      float m_ref = -INFINITY, l_run = 0.f;
      for (int t = 0; t < tiles; ++t) {
        const int u = gt + t, list = kBarList + (u & (kLists - 1));
        // (one look at both barriers)
        if (!mbar_wait(bar(lane & 1 ? list : kBarS), (lane & 1 ? u / kLists : u) & 1)) failed = true;
        failed = __any_sync(0xffffffffu, failed);
        tc_fence_after();
        const uint32_t seen = *reinterpret_cast<volatile uint32_t*>(smem + Smem::seen_off + ((u & (kLists - 1)) * 4 + part) * 4);
        float x[32];  // this lane's 32 keys, -inf where masked; then its probabilities, two to a register
        {
          uint32_t raw[32];
          tmem_ld_32x32(ts, raw);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive_at(leader_bar(kBarSRead));
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(raw[i]);
          if (seen != 0xffffffffu) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (!((seen >> i) & 1u)) x[i] = -INFINITY;
          }
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], x[i]);
        const float m_loc = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;
        // No reference yet, or a maximum that ran away from it: the heads' quarters are compared.
        if (group_sync_or(failed || m_ref == -INFINITY || m_loc > m_ref + kRescaleLog2)) {
          s_max[part * 64 + head] = m_loc;
          if (group_sync_or(failed)) { failed = true; break; }
          float f = 1.f;
          const float m_first = fmaxf(s_max[head], s_max[64 + head]);
          const float m_tile = fmaxf(m_first, fmaxf(s_max[128 + head], s_max[192 + head]));
          // The maximum of the first 64 places of the first tile with a visible key, as the kernel of one CTA has it where its
          // first such tile is those 64: then the same roundings of p. The whole tile's where they are masked or it runs away.
          if (m_ref == -INFINITY) {
            m_ref = m_first == -INFINITY || m_tile > m_first + kRescaleLog2 ? m_tile : m_first;
          } else if (m_tile > m_ref + kRescaleLog2) {
            f = exp2f(m_ref - m_tile);
            l_run *= f;
            m_ref = m_tile;
          }
          if (__any_sync(0xffffffffu, f != 1.f)) {  // rare: scale this head's row of O
            if (t >= 1 && !mbar_wait(bar(kBarPV), (u - 1) & 1)) failed = true;
            failed = __any_sync(0xffffffffu, failed);
            tc_fence_after();
#pragma unroll 1
            for (int blk = 16 * group; blk < 16 * group + 16 && !failed; ++blk) {
              uint32_t o[8];
              tmem_ld_32x8(tq + kColO + 8u * blk, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tmem_st_32x8(tq + kColO + 8u * blk, o);
            }
            tmem_st_wait();
            tc_fence_before();
          }
          group_sync();  // (the maxima have been read)
        }
        const float mr = m_ref == -INFINITY ? 0.f : m_ref;  // every key so far masked: all p = 0
        // the row sum uses the rounded probabilities that the value product will see
        uint32_t pk[16];
        float ps[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(mla_tc::ex2_approx(fmaf(x[2 * i], p.scale_log2, -mr)),
                                                         mla_tc::ex2_approx(fmaf(x[2 * i + 1], p.scale_log2, -mr)));
          pk[i] = *reinterpret_cast<const uint32_t*>(&b);
          ps[0] += __uint_as_float(pk[i] << 16);
          ps[1] += __uint_as_float(pk[i] & 0xFFFF0000u);
        }
        l_run += ps[0] + ps[1];
        // P is single-buffered: the previous tile's value product must have read it
        if (u >= 1 && !mbar_wait(bar(kBarPV), (u - 1) & 1)) failed = true;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          st_shared_v4(s_prow + uint32_t(((4 * group + c) ^ (head & 7)) << 4),
                       make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]));
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at(leader_bar(kBarP));
      }
      gt += tiles;
      if (group_sync_or(failed)) { failed = true; break; }
      s_sum[part * 64 + head] = l_run;
      more = next_item(n + 1, e);
      // ---- result: the normalised bf16 rows (one split) or this split's partials
      if (!mbar_wait(bar(kBarPV), (gt - 1) & 1)) failed = true;
      if (group_sync_or(failed)) { failed = true; break; }
      tc_fence_after();
      const float l = (s_sum[head] + s_sum[64 + head]) + (s_sum[128 + head] + s_sum[192 + head]);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // (the item is read again: kept over the tiles, its numbers would cost registers)
      const volatile int* entry = reinterpret_cast<volatile int*>(smem + Smem::plan_off + 16 * (n & (kPlan - 1)));
      const Item done = item_of(entry[0]);
      const bool mine = !kTwoRows || entry[3] == kBoth || entry[3] == kFirst + rank;  // (else the other row's list went through)
      // first of this CTA's 64 rows of partials: [row][split][head]
      const int64_t pb = kTwoRows ? ((int64_t(done.r) + rank) * p.nsplit + done.split) * 64
                                  : (int64_t(done.r) * p.nsplit + done.split) * p.H + (done.heads0 - int64_t(done.r) * p.H);
      // 64 bytes of 32 rows at a time through this warp's 2 KB of the probabilities' place and out by TMA: 4400 cycles an item.
      // (Straight from the lanes, whose rows are a kilobyte or two apart, an instruction takes as many cycles as it has
      // lanes: 5700, and as much in the way of the others. Both in turn: 3 % slower for short rows.)
      const uint32_t s_stage = s_p + uint32_t(warp) * 2048u;
      const int srow = int((p.out ? done.heads0 : pb) + (quad & 1) * 32);
      auto put = [&](const uint32_t (&w)[16], int col) {
        if (lane == 0) bulk_wait_read();
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c)
          st_shared_v4(s_stage + uint32_t(lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)),
                       make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && mine) tma_store_2d(s_stage, &out_map, col, srow);
      };
#pragma unroll 1
      for (int blk = 4 * group; blk < 4 * group + 4; ++blk) {
        uint32_t o[32], w[16];
        tmem_ld_32x32(tq + kColO + 32u * blk, o);
        tmem_ld_wait();
        if (p.out) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
            w[i] = *reinterpret_cast<const uint32_t*>(&b);
          }
          put(w, 256 * half + 32 * blk);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = o[16 * j + i];
            put(w, 256 * half + 32 * blk + 16 * j);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_at(leader_bar(kBarOFree));
      if (!p.out && part == 0 && mine) {
        p.part_m[pb + head] = m_ref;
        p.part_l[pb + head] = l;
      }
      if (lane == 0) bulk_wait_read();
      group_sync();  // the probabilities' place and s_sum are free again
    }
    if (lane == 0) bulk_wait_all();
  } else {
    if (warp == kPlanWarp) {
      // ===================================================================== plan: items, their tiles, queries in shared memory
      const bool leader = elect_one();
      int n = 0;
      // entry n; the one in its place has been read by all, since the last score product of item n - 2 is done
      auto publish = [&](int item, int tiles, int len, int rows) {
        if (leader) {
          *reinterpret_cast<int4*>(smem + Smem::plan_off + 16 * (n & (kPlan - 1))) = make_int4(item, tiles, len, rows);
          mbar_arrive(bar(kBarPlan + (n & (kPlan - 1))));
        }
        __syncwarp();
      };
      auto list_of = [&](int r) { return p.indices ? p.indices + int64_t(r) * p.topk : nullptr; };
      auto length_of = [&](int r) {
        const int64_t len = p.seq_lens ? int64_t(p.seq_lens[r]) : p.ctx;
        return int(len < 0 ? 0 : (len > p.ctx ? p.ctx : len));
      };
      // where the last visible key of row r's part of the list ends; `last`: the list's last entries, requested together with the length
      auto tail_of = [&](const Item& it, int r) {
        const int32_t* list = list_of(r);
        return list && it.k_end - 32 + lane >= it.k_begin ? list[it.k_end - 32 + lane] : -1;
      };
      auto bound_of = [&](const Item& it, int r, int len, int last) {
        const int32_t* list = list_of(r);
        if (!list) return min(it.k_end, len);
        int bound = __reduce_max_sync(0xffffffffu, last >= 0 && last < len ? it.k_end - 31 + lane : 0);
        if (bound == 0) bound = end_of_list(list, it.k_begin, it.k_end - 32, len);
        return bound;
      };
      // kTwoRows: the bounds of both rows, and whether they nest: row r's visible keys are row r + 1's, in the same places, but
      // for one at most, and that one's value is finite. Then both go through the second one's list together. (The first row's
      // probability of the key is zero, and zero times an infinity would not be.) One pass over both lists, 16 loads under way.
      auto survey = [&](const Item& it, int len0, int len1, int& bound0, int& bound1) {
        const int32_t *list0 = list_of(it.r), *list1 = list_of(it.r + (it.second ? 1 : 0));
        int extras = 0, extra = -1;
        bool same = true;
        bound0 = bound1 = 0;
#pragma unroll 1
        for (int j0 = it.k_begin; j0 < it.k_end; j0 += 256) {
          int i0[8], i1[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int j = j0 + 32 * c + lane;
            i0[c] = i1[c] = -1;
            if (j < it.k_end) i0[c] = list0 ? list0[j] : j, i1[c] = list1 ? list1[j] : j;
          }
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int j = j0 + 32 * c + lane;
            const bool see0 = i0[c] >= 0 && i0[c] < len0, see1 = i1[c] >= 0 && i1[c] < len1;
            if (see0) bound0 = j + 1;
            if (see1) bound1 = j + 1;
            if (see0 && !(see1 && i0[c] == i1[c])) same = false;
            if (see1 && !see0) ++extras, extra = i1[c];
          }
        }
        bound0 = __reduce_max_sync(0xffffffffu, bound0), bound1 = __reduce_max_sync(0xffffffffu, bound1);
        if (!__all_sync(0xffffffffu, same) || __reduce_add_sync(0xffffffffu, extras) > 1) return false;
        extra = __reduce_max_sync(0xffffffffu, extra);
        bool finite = true;
        if (extra >= 0) {
          const uint8_t* row = p.kv + (int64_t(it.r / p.rows_per_seq) * p.kv_seq_stride + extra) * mla::kRowBytes;
#pragma unroll
          for (int c = 0; c < mla::kDV / 64; ++c) {  // (two value dims a word; the others do not enter the value product)
            const uint32_t w = reinterpret_cast<const uint32_t*>(row)[32 * c + lane];
            finite = finite && (w & 0x7F80u) != 0x7F80u && (w & 0x7F800000u) != 0x7F800000u;
          }
        }
        return __all_sync(0xffffffffu, finite) && bound1 > it.k_begin;
      };
      auto store_zeros = [&](const Item& it) {  // nothing visible: the plan does not mention the row
        const uint4 zero = make_uint4(0, 0, 0, 0);
        if (p.out) {
          uint4* dst = reinterpret_cast<uint4*>(p.out + it.heads0 * mla::kDV);
          for (int j = lane; j < 64 * mla::kDV / 8; j += 32) dst[j] = zero;
        } else {
          const int64_t pb = kTwoRows ? ((int64_t(it.r) + rank) * p.nsplit + it.split) * 64
                                      : (int64_t(it.r) * p.nsplit + it.split) * p.H + (it.heads0 - int64_t(it.r) * p.H);
          uint4* dst = reinterpret_cast<uint4*>(p.part_acc + pb * mla::kDV);
          for (int j = lane; j < 64 * mla::kDV / 4; j += 32) dst[j] = zero;
          for (int j = lane; j < 64; j += 32) p.part_m[pb + j] = -INFINITY, p.part_l[pb + j] = 0.f;
        }
      };
      auto tiles_of = [&](const Item& it, int bound) { return (max(bound - it.k_begin, 0) + kBN - 1) / kBN; };
      // puts an item into the plan and requests the rest of its queries
      auto enter = [&](int i, const Item& it, int tiles, int len, int rows) {
        publish(i, tiles, len, rows);
        if (n >= 1 && __any_sync(0xffffffffu, !mbar_wait(bar(kBarQFree), (n - 1) & 1))) return !(failed = true);
        if (leader) {
          if (rank == 0) mbar_arrive_expect_tx(bar(kBarQ), 2 * (9 - kQTmem) * kChunkBytes);
          const uint32_t at = leader_bar(kBarQ);
          for (int c = kQTmem; c < 9; ++c)
            tma_load_2d_pair(s_q + uint32_t(c - kQTmem) * kChunkBytes, &q_map, c * 64, int(it.heads0), at);
        }
        __syncwarp();
        ++n;
        return true;
      };
      for (int k = 0; k * clusters < pp.items && !failed; ++k) {
        // clusters take items in turn, every other time in reverse: the longer rows are spread over all
        const int i = k * clusters + ((k & 1) ? clusters - 1 - cid : cid);
        if (i >= pp.items) continue;
        const Item it = item_of(i);
        const int last = kTwoRows ? 0 : tail_of(it, it.r);
        const int len = length_of(it.r), len1 = kTwoRows && it.second ? length_of(it.r + 1) : 0;
        if constexpr (kTwoRows) {
          int bound, bound1;
          if (survey(it, len, len1, bound, bound1)) {
            if (!enter(i, it, tiles_of(it, bound1), len1, kBoth)) break;
            continue;
          }
          for (int row = 0; row < (it.second ? 2 : 1) && !failed; ++row) {
            const int tiles = tiles_of(it, row ? bound1 : bound);
            if (tiles > 0) enter(i, it, tiles, row ? len1 : len, row ? kSecond : kFirst);
            else if (rank == row) store_zeros(it);
          }
        } else {
          const int tiles = tiles_of(it, bound_of(it, it.r, len, last));
          if (tiles > 0) enter(i, it, tiles, len, kBoth);
          else store_zeros(it);
        }
      }
      if (!failed) publish(-1, 0, 0, kBoth);
    } else if (warp >= kGatherWarp0) {
      // ===================================================================== gather
      // Four warps bring unit j of a tile's keys and unit j of its values, 32 rows of one chunk each. The seventeenth lays out
      // the rows of the tiles and brings the last chunk of the keys.
      const int g = warp - kGatherWarp0, quad = g >> 2, chunk = (g >> 1) & 1, row0 = 32 * (g & 1);
      const bool leader = elect_one();
      Ring pos{0, 0};  // the item's first unit
      int gt = 0;      // tiles so far
      int4 e;
      for (int n = 0; !failed && next_plan(n, e); ++n) {
        const Item it = item_of(e.x);
        auto gather = [&](uint32_t dst, int x, uint32_t at, int u, int row0) {  // 32 rows of one chunk
          const int4* rows = reinterpret_cast<const int4*>(smem + Smem::list_off + ((u & (kLists - 1)) * kBN + row0) * 4);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int4 y = rows[q];
            if (leader) gather4(dst + 512u * q, &kv_map, x, y, at);
          }
          __syncwarp();
        };
        auto list_ready = [&](int u) {
          if (__any_sync(0xffffffffu, !mbar_wait(bar(kBarList + (u & (kLists - 1))), (u / kLists) & 1))) failed = true;
          return !failed;
        };
        auto unit = [&](const Ring& at, int x, int u, int block) {
          if (__any_sync(0xffffffffu, !mbar_wait(bar(kBarEmpty + at.slot), at.phase ^ 1))) return !(failed = true);
          if (rank == 0 && (g & 3) == 0 && leader) mbar_arrive_expect_tx(bar(kBarFull + at.slot), 2 * kUnitBytes);
          gather(s_ring + uint32_t(at.slot) * kUnitBytes + uint32_t(chunk) * kChunkBytes + uint32_t(row0) * 128, x + 64 * chunk,
                 leader_bar(kBarFull + at.slot), u, 64 * block + row0);
          return true;
        };
        if (g < kGatherWarps) {
          Ring at = pos;
          at.add(quad);
          // The part of the queries that goes to tensor memory passes through the ring. (A wait is for a parity:
          // a place's use before the last must be known to be over. Units are freed in order, and a warp's next place is at
          // most kUnits behind its last one, so it is.)
          if (quad < kQTmem / 2 && (g & 3) == 0) {
            if (__any_sync(0xffffffffu, !mbar_wait(bar(kBarEmpty + at.slot), at.phase ^ 1))) { failed = true; break; }
            if (leader) {
              mbar_arrive_expect_tx(bar(kBarQStage), kUnitBytes);
              for (int c = 0; c < 2; ++c)
                tma_load_2d(s_ring + uint32_t(at.slot) * kUnitBytes + uint32_t(c) * kChunkBytes, &q_map, 128 * quad + 64 * c,
                            int(it.heads0), bar(kBarQStage));
            }
            __syncwarp();
          }
          at.add(kQTmem / 2);
          if (!list_ready(gt) || !unit(at, 128 * quad, gt, rank)) break;
          for (int u = gt; u < gt + e.y; ++u) {
            at.add(4);
            if (u + 1 < gt + e.y) {
              if (!list_ready(u + 1) || !unit(at, 128 * quad, u + 1, rank)) break;
              at.add(4);
            }
            if (!unit(at, 256 * rank + 128 * (quad & 1), u, quad >> 1)) break;
          }
        } else {
          // The rows of a tile for everybody, once the products of the scores two tiles before are done: the value product four
          // tiles before, the last to need the place's rows, was issued before those. Then the tile's last chunk.
          const int64_t seq_row = int64_t(it.r / p.rows_per_seq) * p.kv_seq_stride;
          // kTwoRows: both CTAs go through one list, but the first CTA's row sees what its own list says
          const int lrow = it.r + (kTwoRows && e.w != kFirst ? 1 : 0);
          const bool own = kTwoRows && e.w == kBoth && rank == 0;
          int own_len = 0;
          if (own) {
            const int64_t len = p.seq_lens ? int64_t(p.seq_lens[it.r]) : p.ctx;
            own_len = int(len < 0 ? 0 : (len > p.ctx ? p.ctx : len));
          }
          auto load = [&](int r, int t, int (&idx)[4]) {
            const int32_t* list = p.indices ? p.indices + int64_t(r) * p.topk : nullptr;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int j = it.k_begin + t * kBN + 32 * i + lane;
              idx[i] = -1;
              if (t < e.y && j < it.k_end) idx[i] = list ? list[j] : j;
            }
          };
          int idx[4], mine[4];
          load(lrow, 0, idx);
          if (own) load(it.r, 0, mine);
          for (int t = 0; t < e.y && !failed; ++t) {
            const int u = gt + t, b = u & 1, l = u & (kLists - 1);
            if (__any_sync(0xffffffffu, !mbar_wait(bar(kBarRopeFree + b), ((u >> 1) & 1) ^ 1))) { failed = true; break; }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const bool ok = idx[i] >= 0 && idx[i] < e.z;
              const uint32_t seen = __ballot_sync(0xffffffffu, own ? mine[i] >= 0 && mine[i] < own_len : ok);
              *reinterpret_cast<volatile int*>(smem + Smem::list_off + (l * kBN + 32 * i + lane) * 4) = ok ? int(seq_row + idx[i]) : -1;
              if (lane == 0) *reinterpret_cast<volatile uint32_t*>(smem + Smem::seen_off + (l * 4 + i) * 4) = seen;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kBarList + l));
            if (rank == 0 && leader) mbar_arrive_expect_tx(bar(kBarRope + b), 2 * kChunkBytes);
            load(lrow, t + 1, idx);
            if (own) load(it.r, t + 1, mine);
            gather(s_rope + uint32_t(b) * kChunkBytes, 512, leader_bar(kBarRope + b), u, 64 * rank);
            gather(s_rope + uint32_t(b) * kChunkBytes + kChunkBytes / 2, 512, leader_bar(kBarRope + b), u, 64 * rank + 32);
          }
        }
        gt += e.y;
        pos.add_many(kQTmem / 2 + 8 * e.y);
      }
    } else if (warp == kMmaWarp) {
      // ===================================================================== MMA issue (the pair's first CTA)
      if (rank == 0) {
        const bool leader = elect_one();
        constexpr uint32_t idesc_qk = idesc_bf16_f32(128, kBN, false, false);
        constexpr uint32_t idesc_pv = idesc_bf16_f32(128, 256, false, true);
        int slot = 0, gt = 0;
        // One look tests every barrier that this warp ever waits for, a lane each: bit i of `ready` says that the next phase of
        // barrier i is complete, bit i of `phases` is its parity. (A wait of its own for each unit, ready or not, cost 200
        // cycles, and the products of a unit take 260.)
        static_assert(kNumPolled <= 32 && kBarFull == 0, "a lane per barrier");
        uint32_t ready = 0, phases = 0;
        auto wait = [&](int b) {
          unsigned long long t0 = 0;
          for (uint32_t i = 0; !((ready >> b) & 1u); ++i) {
            ready |= __ballot_sync(0xffffffffu, lane < kNumPolled && mbar_test(bar(lane), (phases >> lane) & 1u));
            if ((i & 255u) == 255u) {  // bounded, as mbar_wait is
              const unsigned long long now = __shfl_sync(0xffffffffu, wall_ns(), 0);
              if (t0 == 0) t0 = now;
              else if (now - t0 > kWaitLimitNs) return !(failed = true);
            }
          }
          ready &= ~(1u << b), phases ^= 1u << b;
          tc_fence_after();
          return true;
        };
        auto advance = [&]() { slot = slot + 1 == kUnits ? 0 : slot + 1; };
        auto scores = [&](int u) {  // S of tile u (counted over all items)
          const uint32_t d = tmem + kColS;
          if (u >= 1 && !wait(kBarSRead)) return false;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (!wait(kBarFull + slot)) return false;
            if (leader) {
              const uint64_t b0 = smem_desc_k128(s_ring + uint32_t(slot) * kUnitBytes);
#pragma unroll
              for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                  const uint64_t b = b0 + uint64_t((c * kChunkBytes >> 4) + 2 * ks);
                  if (2 * j + c < kQTmem) mma2_ts(d, tmem + kColQ + 32u * (2 * j + c) + 8u * ks, b, idesc_qk, (j | c | ks) ? 1u : 0u);
                  else mma2(d, smem_desc_k128(s_q + uint32_t(2 * j + c - kQTmem) * kChunkBytes) + uint64_t(2 * ks), b, idesc_qk, 1u);
                }
              commit2(bar(kBarEmpty + slot));
            }
            __syncwarp();
            advance();
          }
          if (!wait(kBarRope + (u & 1))) return false;
          if (leader) {
            const uint64_t b0 = smem_desc_k128(s_rope + uint32_t(u & 1) * kChunkBytes);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              mma2(d, smem_desc_k128(s_q + uint32_t(8 - kQTmem) * kChunkBytes) + uint64_t(2 * ks), b0 + uint64_t(2 * ks), idesc_qk, 1u);
            commit2(bar(kBarRopeFree + (u & 1)));
            commit2(bar(kBarS));
          }
          __syncwarp();
          return true;
        };
        auto values = [&](int u, bool first) {
          if (!wait(kBarP)) return false;
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (!wait(kBarFull + slot)) return false;
              if (leader) {
                const uint64_t v0 = smem_desc_mn128(s_ring + uint32_t(slot) * kUnitBytes, kChunkBytes, 1024);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                  mma2(tmem + kColO + 128u * i, smem_desc_k128(s_p + uint32_t(b) * kChunkBytes) + uint64_t(2 * ks),
                       v0 + uint64_t(ks * (2048 >> 4)),
                       idesc_pv, (first && b == 0 && ks == 0) ? 0u : 1u);
                commit2(bar(kBarEmpty + slot));
              }
              __syncwarp();
              advance();
            }
          if (leader) commit2(bar(kBarPV));
          __syncwarp();
          return true;
        };
        int4 e;
        for (int n = 0; !failed && next_plan(n, e); ++n) {
          if (!wait(kBarQT) || !wait(kBarQ)) break;
#pragma unroll
          for (int i = 0; i < kQTmem / 2; ++i) {  // the queries' units are free, in the ring's order: behind the item before
            if (leader) commit2(bar(kBarEmpty + slot));
            advance();
          }
          __syncwarp();
          if (!scores(gt)) break;
          for (int t = 0; t < e.y; ++t) {
            if (t + 1 < e.y && !scores(gt + t + 1)) break;
            if (t + 1 == max(e.y - 1, 1)) {  // every score product of the item has been issued
              if (leader) commit2(bar(kBarQFree));
              __syncwarp();
            }
            if (t == 0 && n >= 1 && !wait(kBarOFree)) break;
            if (!values(gt + t, t == 0)) break;
          }
          gt += e.y;
        }
      }
    }
  }

  if (failed) {
    atomicOr(&g_device_status, kStatusAttnTimeout);
    drain_after_timeout();  // let outstanding copies and products drain
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // neither CTA leaves while the other still signals its barriers
  cluster_wait();
  if (warp == kMmaWarp) tmem_free2(tmem, kTmemCols);
  if constexpr (kBeside) pdl_wait();
  DSA_KTIME_END(2);
}

}  // namespace mla_pair
}  // namespace dsa
