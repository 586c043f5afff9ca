// Split-K sparse MLA decode on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// Same contract and the same split-K partials as sparse_mla.cuh (reference:
// kernels/cuda_fused_sparse_splitk.py:282-530 attention warps, :996-1045 merge),
// for head counts that are a multiple of 64. One CTA = (query row, block of 64
// heads, one split of the index list); 64-key tiles:
//
//   S   [64 heads x 64 keys]  = Q K^T      A = Q   (K-major),  B = K tile (K-major)
//   O^T [512 dims x 64 heads] += V^T P^T   A = V^T (MN-major), B = P      (K-major)
//
// Both products read the SAME shared-memory image of the gathered latent rows:
// nine 64-dim chunks of [64 keys][128 B] with the 128-byte swizzle. For Q K^T a
// chunk is a K-major B operand; for V^T P^T the first eight chunks are an
// MN-major A operand (dims contiguous), so no transposed copy is ever made.
// O^T puts the 512 value dims on the 128 TMEM lanes (4 blocks of 64 columns) and
// the heads on columns: 256 of the 512 columns. S takes 64, and the first 384 dims
// of Q the other 192, as a TMEM A operand (rows 64..127 of the 128-row MMA are
// whatever the lanes hold; nobody reads the score rows that they feed).
//
// What bounds it. At N = 64 an MMA with both operands in shared memory takes 49 cycles
// (6 KB at 128 B per cycle), with A in TMEM 33, so a tile costs 24 x 33 + 12 x 49 + 16 x 49
// = 2160 cycles of the tensor core and as much of the shared memory; a tile takes 2900 - 3300,
// the rest being the hand-offs S -> softmax (1700 cycles) -> O^T -> next rows (a thousand
// cycles behind the free slot) of which only two or three tiles are under way. Hence:
//   * the MMA warp stays converged (elect_one() around the instructions). Under `lane == 0`
//     each instruction cost 63 - 95 cycles of moving operands to uniform registers, which
//     looked like the tensor core's rate: 1026 -> 877 us for 1024 rows of 128 heads x 2048 keys;
//   * Q in TMEM frees shared memory for three slots of a tile's first six chunks (and two of the
//     rest), whose rows travel a tile ahead; -> 851 us with four chunks in two slots;
//   * the value product goes first whenever it is ready, dims 384..511 (the part with two slots)
//     before the others; the first rows of a CTA go out before the list's length is known, and
//     twelve warps write the result instead of four -> 817 us. (Batch 32 of 128 heads, bf16 rows
//     51.6 -> 44.0, fp8 rows 55.6 -> 49.2; 700-token prompt, 64 heads 103 -> 86 us.)
//   * rows are launched last first: those of a prompt grow, and the long ones must not be the tail.
// Tried: two S buffers with four chunks of Q in TMEM (901 us), a fixed order S(t + 1), O(t) (874;
// a ready value product then waits for rows: 46 us at batch 32), looking for work after every chunk
// (1220: each look costs 300 cycles of a busy shared memory), two issuing warps (852: their
// instructions alternate, and the value product ends with the score product).
//
// Warp roles (480 threads): a warp reaches the TMEM lane quadrant (warp % 4).
// Warps 0,1 and 4,5 run the softmax on the 64 real S rows (thread = head; warps 0,1
// take key columns 0..31, warps 4,5 columns 32..63) after warps 0,1 have moved Q into TMEM;
// warps 0-3 rescale O^T; warp 6 allocates TMEM and issues the MMAs; warps 7-14 gather
// rows (eight threads per row; with four gather warps the fp8 conversion paced the
// kernel: 63 us against 56 us at batch 32, bf16 rows unchanged): 16-byte asynchronous
// copies straight into the swizzled image (bf16 rows) or load / dequantise / store (fp8
// rows, fp8 -> f32, x group scale, round to bf16; :1181-1196); warps 0-11 write the result.
//
// Softmax reference point: the row maximum of the first visible tile is kept as
// the reference m for the whole split; a later tile only forces a rescale of O^T
// (rare path: all four lane-quadrant warps scale the 64 head columns in TMEM) when
// it exceeds m by more than 2^kRescaleLog2. Probabilities are floating point, so
// a stale reference costs no precision; the split's (m, l, O) stay consistent
// and the merge kernel renormalises them.
//
// Tile size: four 32-key ring slots (the same bytes as two 64-key slots, three
// tiles in flight instead of one) were built and measured 1.5x SLOWER: the
// per-tile fixed latencies (mbarrier hand-offs, tensor-memory load, proxy
// fences, the softmax group barrier) do not shrink with the tile.
#pragma once

#include "sparse_mla.cuh"

#ifndef DSA_MLA_TC_PROD_WARPS
#define DSA_MLA_TC_PROD_WARPS 8
#endif

namespace dsa {
namespace mla_tc {

constexpr int kHG = 64;                        // heads per CTA
constexpr int kBN = 64;                        // keys per tile
constexpr int kChunks = mla::kD / 64;          // 9 chunks of 64 dims (128 B of bf16)
constexpr int kChunkBytes = 64 * 128;          // [64 rows][128 B]
constexpr int kTileBytes = kChunks * kChunkBytes;  // 73,728
constexpr int kProdWarps = DSA_MLA_TC_PROD_WARPS;  // gather warps: 4 or 8
constexpr int kThreads = 224 + 32 * kProdWarps;
constexpr int kSoftThreads = 192;              // warps 0-5: softmax / rescale group
constexpr int kMmaWarp = 6;                    // issues the products (and owns the tensor-memory allocation)
constexpr int kProducerWarp0 = 7;
constexpr int kFirstChunks = 6;                // chunks of a tile's first part (three slots; the rest of a tile: two)
constexpr int kFirstBytes = kFirstChunks * kChunkBytes, kRestBytes = kTileBytes - kFirstBytes;
constexpr int kProducers = 32 * kProdWarps;
constexpr int kEpiGroups = kThreads / 128;     // groups of four warps that write the result
constexpr int kRowsPerPass = 4 * kProdWarps;    // 8 threads per row
constexpr int kPasses = kBN / kRowsPerPass;     // rows of a tile per gather thread
constexpr float kRescaleLog2 = 40.f;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0;                  // S: 64 columns
constexpr uint32_t kColO = 64;                // four O^T blocks of 64 columns
constexpr uint32_t kColQ = 320;                // the first kQTmem chunks of Q as bf16, 32 columns each
constexpr int kQTmem = 6;
#ifndef DSA_MLA_TC_MIN_TILES
#define DSA_MLA_TC_MIN_TILES 128  // (a build flag, for measuring the crossover)
#endif
// Fewer 64 x 64 tiles than this: the mma.sync kernel. With the merge, each with its own best split (us, this kernel /
// mma.sync): 32 tiles 11.6 / 9.3 (bf16 rows), 14.0 / 11.9 (fp8); 64 of one row 12.0 / 9.7, 14.8 / 12.3; 96 (3 rows of 64
// heads) 12.0 / 13.5, 14.5 / 18.6; 128 12.6 / 15.5, 15.1 / 20.7; 256 14.5 / 22.4, 17.4 / 32.1. (Between 64 and 128 tiles
// the line lies by the rows; 64 tiles of two rows are 11.4 / 11.4 and 12.0 / 14.0.)
constexpr int kMinTiles = DSA_MLA_TC_MIN_TILES;

struct Smem {
  static constexpr int q_off = 0;
  static constexpr int k_off = q_off + (kChunks - kQTmem) * kChunkBytes;  // chunks kQTmem.. of Q (the others are in tensor memory)
  static constexpr int rest_off = k_off + 3 * kFirstBytes;
  static constexpr int p_off = rest_off + 2 * kRestBytes;
  static constexpr int misc_off = p_off + kHG * 128;
  static constexpr int bar_off = misc_off;             // 16 mbarriers
  static constexpr int tmem_off = misc_off + 136;
  static constexpr int flag_off = misc_off + 140;      // int [2]
  static constexpr int valid_off = misc_off + 148;     // uint32 [2 stages][producer warps]
  static constexpr int bound_off = misc_off + 248;     // int: end of the split's last visible key
  static constexpr int factor_off = misc_off + 256;    // float [64]
  static constexpr int max_off = misc_off + 512;       // float [2 parities][2 halves][64]
  static constexpr int bytes = misc_off + 1536 + 1024;  // + slack for the 1024-byte alignment
};
static_assert(Smem::bytes <= 232448, "tcgen05 sparse MLA: shared memory over the per-CTA limit");

// First / Rest: the two parts of a tile have landed; RestFree / Free: the value product has read the second
// part / everything; SFull / SRead: scores computed / read; PFull: probabilities stored; OFull: all done.
enum {
  kBarQ = 0, kBarFirst = 1, kBarRest = 4, kBarRestFree = 6, kBarFree = 8, kBarSFull = 11, kBarSRead = 12, kBarPFull = 13, kBarOFull = 14,
  kBarQT = 15 /* queries in tensor memory */, kNumBars = 16
};

// Named barrier 2 over the 192 threads of warps 0-5, plain and with an OR reduction.
__device__ __forceinline__ void group_sync() { asm volatile("bar.sync 2, 192;" ::: "memory"); }
__device__ __forceinline__ bool group_sync_or(bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 2, 192, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(uint32_t(x))
      : "memory");
  return r != 0;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Byte offset of 16-byte unit `u` (0..7) of row `row` inside a swizzled chunk.
__device__ __forceinline__ uint32_t swz(int row, int u) { return uint32_t(row * 128 + ((u ^ (row & 7)) << 4)); }

template <bool kBeside>  // as in mla_partials_body
__global__ void __launch_bounds__(kThreads, 1)
sparse_mla_tc_kernel(const mla::Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t s_q = sbase + Smem::q_off;
  const uint32_t s_k = sbase + Smem::k_off;
  // shared-memory address that chunk c of tile t has as its place
  const auto chunk_at = [&](int t, int c) {
    return c < kFirstChunks ? s_k + uint32_t(t % 3) * kFirstBytes + uint32_t(c) * kChunkBytes
                            : s_k + 3u * kFirstBytes + uint32_t(t & 1) * kRestBytes + uint32_t(c - kFirstChunks) * kChunkBytes;
  };
  const uint32_t s_p = sbase + Smem::p_off;
  const uint32_t bars = sbase + Smem::bar_off;
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + Smem::tmem_off);
  volatile int* s_flag = reinterpret_cast<volatile int*>(smem + Smem::flag_off);
  volatile uint32_t* s_validw = reinterpret_cast<volatile uint32_t*>(smem + Smem::valid_off);
  int* s_bound = reinterpret_cast<int*>(smem + Smem::bound_off);
  volatile float* s_factor = reinterpret_cast<volatile float*>(smem + Smem::factor_off);
  volatile float* s_max = reinterpret_cast<volatile float*>(smem + Smem::max_off);
  auto bar = [&](int i) { return bars + 8u * uint32_t(i); };

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // (warp-uniform)
  const int split = blockIdx.x, hg = blockIdx.y, r = gridDim.z - 1 - blockIdx.z;
  DSA_KTIME_BEGIN(2);
  const int scta = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  (void)scta;

  if (tid == 0) {
    mbar_init(bar(kBarQ), kProducers);
    mbar_init(bar(kBarQT), kHG);
    for (int s = 0; s < 3; ++s) {
      mbar_init(bar(kBarFirst + s), kProducers);
      mbar_init(bar(kBarFree + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(kBarRest + s), kProducers);
      mbar_init(bar(kBarRestFree + s), 1);
      s_flag[s] = 0;
    }
    mbar_init(bar(kBarSFull), 1);
    mbar_init(bar(kBarSRead), 2 * kHG);
    mbar_init(bar(kBarPFull), 2 * kHG);
    mbar_init(bar(kBarOFull), 1);
    *s_bound = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(s_tmem)), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);

  if constexpr (!kBeside) pdl_wait();  // the selection, the queries and the lengths may come from the previous kernel
  pdl_launch_dependents();

  const int seq = r / p.rows_per_seq;
  int64_t len = p.seq_lens ? int64_t(p.seq_lens[r]) : p.ctx;
  len = len < 0 ? 0 : (len > p.ctx ? p.ctx : len);
  const int k_begin = split * p.keys_per_split;
  const int k_end = min(k_begin + p.keys_per_split, p.topk);
  bool failed = false;
  float m_ref = -INFINITY, l_run = 0.f;  // softmax
  DSA_STAMP(scta, 14);

  const int ptid = tid - kProducerWarp0 * 32;
  const int v8 = ptid & 7, rsub = ptid >> 3;  // gather: 8 threads per row, kRowsPerPass rows per pass
  const int row_bytes = p.kv_fp8 ? mla::kFp8Row : mla::kRowBytes;
  const uint8_t* kv_seq = p.kv + int64_t(seq) * p.kv_seq_stride * row_bytes;
  int64_t idx_next[kPasses];  // gather: selection entries of this thread's rows of the next tile
  // rows of tile t handled by this thread (nullptr: masked key) and the tile's validity bits
  auto resolve = [&](const uint8_t* (&src)[kPasses], uint32_t& vword) {
    vword = 0;
#pragma unroll
    for (int k = 0; k < kPasses; ++k) {
      const bool ok = idx_next[k] >= 0 && idx_next[k] < len;
      src[k] = ok ? kv_seq + idx_next[k] * row_bytes : nullptr;
      const uint32_t b = __ballot_sync(0xffffffffu, ok);
      vword |= (((b >> 0) & 1u) | (((b >> 8) & 1u) << 1) | (((b >> 16) & 1u) << 2) | (((b >> 24) & 1u) << 3)) << (4 * k);
    }
  };
  const uint8_t *src[kPasses], *nsrc[kPasses];
  uint32_t vword = 0, nvword = 0;
  auto copy_chunks = [&](int t, int c0, int c1, const uint8_t* (&from)[kPasses]) {
#pragma unroll
    for (int k = 0; k < kPasses; ++k) {
      const int row = rsub + kRowsPerPass * k;
      if (from[k]) {
#pragma unroll
        for (int c = c0; c < c1; ++c) cp_async16(chunk_at(t, c) + swz(row, v8), from[k] + c * 128 + v8 * 16);
      } else {
        // masked key: its row must be finite because 0 * NaN would poison V^T P^T
#pragma unroll
        for (int c = c0; c < c1; ++c) st_shared_v4(chunk_at(t, c) + swz(row, v8), make_uint4(0, 0, 0, 0));
      }
    }
    cp_async_commit();
  };
  if (warp >= kProducerWarp0) {
#pragma unroll
    for (int k = 0; k < kPasses; ++k) {
      const int j = k_begin + rsub + kRowsPerPass * k;
      idx_next[k] = -1;
      if (j < k_end) idx_next[k] = p.indices ? int64_t(p.indices[int64_t(r) * p.topk + j]) : int64_t(j);
    }
    // queries of this head block: [64 heads][1152 B] -> swizzled chunks; those on their way to tensor memory
    // rest in the third slot until tile 2 needs it
    const uint8_t* qsrc = reinterpret_cast<const uint8_t*>(p.q + (int64_t(r) * p.H + hg * kHG) * mla::kD);
#pragma unroll
    for (int k = 0; k < kPasses; ++k) {
      const int row = rsub + kRowsPerPass * k;
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        cp_async16((c < kQTmem ? chunk_at(2, c) : s_q + uint32_t(c - kQTmem) * kChunkBytes) + swz(row, v8),
                   qsrc + row * mla::kRowBytes + c * 128 + v8 * 16);
    }
    cp_async_commit();
    if (!p.kv_fp8) {  // the first rows go out before anything else is known about the list
      resolve(src, vword);
      copy_chunks(0, 0, kFirstChunks, src);
    }
  }
  // Where the split's last visible key ends: the padding behind it (a row with fewer keys than the list
  // has entries, as most rows of a prompt) costs no tiles. The look at the list runs beside the query's
  // way into shared memory, which the first product waits for anyway. (4099-token prompt, top-2048,
  // 128 heads: a quarter of the tiles.)
  int n_tiles;
  if (p.indices) {
    int bound = 0;
#pragma unroll 4
    for (int j = k_begin + tid; j < k_end; j += kThreads) {
      const int idx = p.indices[int64_t(r) * p.topk + j];
      if (idx >= 0 && idx < len) bound = j + 1;
    }
    bound = __reduce_max_sync(0xffffffffu, bound);
    if (lane == 0 && bound > 0) atomicMax(s_bound, bound);
    __syncthreads();
    n_tiles = (max(*s_bound - k_begin, 0) + kBN - 1) / kBN;
  } else {
    n_tiles = (max(int(min(int64_t(k_end), len)) - k_begin, 0) + kBN - 1) / kBN;
  }

  if (warp >= kProducerWarp0) {
    // ===================================================================== gather
    // selection entries of this thread's four rows of tile t (-1 past the split)
    auto load_idx = [&](int t, int64_t (&idx)[kPasses]) {
#pragma unroll
      for (int k = 0; k < kPasses; ++k) {
        const int j = k_begin + t * kBN + rsub + kRowsPerPass * k;
        idx[k] = -1;
        if (t < n_tiles && j < k_end) idx[k] = p.indices ? int64_t(p.indices[int64_t(r) * p.topk + j]) : int64_t(j);
      }
    };
    auto publish_queries = [&]() {
      fence_proxy_async_smem();
      mbar_arrive(bar(kBarQ));
    };
    if (!p.kv_fp8) {
      load_idx(1, idx_next);
      cp_async_wait_pending<1>();
      publish_queries();
      // The first part of tile t + 1 is requested behind the second part of tile t: its slot is free by
      // then, and its way is hidden behind a whole tile.
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t & 1;
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 0);
        resolve(nsrc, nvword);
        load_idx(t + 2, idx_next);  // in flight during the waits below
        cp_async_wait_all();
        fence_proxy_async_smem();
        mbar_arrive(bar(kBarFirst + t % 3));
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 1);
        // (the outcome of a wait is made warp-uniform: the loop contains warp votes)
        if (__any_sync(0xffffffffu, t >= 2 && !mbar_wait(bar(kBarRestFree + s), ((t >> 1) - 1) & 1))) { failed = true; break; }
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 3);
        if (lane == 0) s_validw[s * kProdWarps + (warp - kProducerWarp0)] = vword;
        copy_chunks(t, kFirstChunks, kChunks, src);
        if (t + 1 < n_tiles) {
          if (__any_sync(0xffffffffu, t == 1 ? !mbar_wait(bar(kBarQT), 0) : t >= 2 && !mbar_wait(bar(kBarFree + (t + 1) % 3), ((t - 2) / 3) & 1))) {
            failed = true;
            break;
          }
          copy_chunks(t + 1, 0, kFirstChunks, nsrc);
          cp_async_wait_pending<1>();
        } else {
          cp_async_wait_all();
        }
        fence_proxy_async_smem();
        mbar_arrive(bar(kBarRest + s));
#pragma unroll
        for (int k = 0; k < kPasses; ++k) src[k] = nsrc[k];
        vword = nvword;
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 4);
      }
    } else {
      // fp8 rows: 512 e4m3 | 4 fp32 group scales | 64 bf16 rope. Unit u = v8 + 8 g of the
      // e4m3 part belongs to scale group g and expands to bf16 units 2u, 2u + 1. The raw
      // bytes of tile t + 1 are requested into registers as soon as tile t is stored, so
      // they travel while the slot of tile t + 1 is still being read by the tensor core.
      uint4 raw[kPasses][4], rope[kPasses], sc4[kPasses];
      auto request = [&]() {
        const uint8_t* src[kPasses];
        resolve(src, vword);
#pragma unroll
        for (int k = 0; k < kPasses; ++k) {
          if (src[k]) {
#pragma unroll
            for (int g = 0; g < 4; ++g) raw[k][g] = ld_global_nc_v4(src[k] + (v8 + 8 * g) * 16);
            sc4[k] = ld_global_nc_v4(src[k] + 512);
            rope[k] = ld_global_nc_v4(src[k] + 528 + v8 * 16);
          } else {
#pragma unroll
            for (int g = 0; g < 4; ++g) raw[k][g] = make_uint4(0, 0, 0, 0);
            sc4[k] = make_uint4(0, 0, 0, 0);
            rope[k] = make_uint4(0, 0, 0, 0);
          }
        }
      };
      if (n_tiles > 0) {
        request();
        load_idx(1, idx_next);
      }
      cp_async_wait_all();
      publish_queries();
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t & 1;
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 0);
        auto store_group = [&](int k, int g, float scale) {
          const int row = rsub + kRowsPerPass * k, c = 2 * g + (v8 >> 2), u = 2 * (v8 & 3);
          const uint2 d0 = mla::dequant4(raw[k][g].x, scale), d1 = mla::dequant4(raw[k][g].y, scale);
          const uint2 d2 = mla::dequant4(raw[k][g].z, scale), d3 = mla::dequant4(raw[k][g].w, scale);
          // (lanes 0..3 of a row store the even units of one chunk while lanes 4..7 store the odd ones of the next:
          // the same units of both lie in the same banks)
          const uint4 even = make_uint4(d0.x, d0.y, d1.x, d1.y), odd = make_uint4(d2.x, d2.y, d3.x, d3.y);
          const bool hi = v8 >= 4;
          st_shared_v4(chunk_at(t, c) + swz(row, hi ? u + 1 : u), hi ? odd : even);
          st_shared_v4(chunk_at(t, c) + swz(row, hi ? u : u + 1), hi ? even : odd);
        };
        static_assert(kFirstChunks == 6, "the first part of an fp8 tile is scale groups 0, 1 and 2");
        if (__any_sync(0xffffffffu, t == 2 ? !mbar_wait(bar(kBarQT), 0) : t >= 3 && !mbar_wait(bar(kBarFree + t % 3), (t / 3 - 1) & 1))) {
          failed = true;
          break;
        }
#pragma unroll
        for (int k = 0; k < kPasses; ++k) {
          store_group(k, 0, __uint_as_float(sc4[k].x));
          store_group(k, 1, __uint_as_float(sc4[k].y));
          store_group(k, 2, __uint_as_float(sc4[k].z));
        }
        fence_proxy_async_smem();
        mbar_arrive(bar(kBarFirst + t % 3));
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 1);
        if (__any_sync(0xffffffffu, t >= 2 && !mbar_wait(bar(kBarRestFree + s), ((t >> 1) - 1) & 1))) { failed = true; break; }
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 3);
        if (lane == 0) s_validw[s * kProdWarps + (warp - kProducerWarp0)] = vword;
#pragma unroll
        for (int k = 0; k < kPasses; ++k) {
          store_group(k, 3, __uint_as_float(sc4[k].w));
          st_shared_v4(chunk_at(t, 8) + swz(rsub + kRowsPerPass * k, v8), rope[k]);
        }
        fence_proxy_async_smem();
        mbar_arrive(bar(kBarRest + s));
        DSA_STAMP_IF(ptid == 0 && t == 4, scta, 4);
        if (t + 1 < n_tiles) {
          request();
          load_idx(t + 2, idx_next);
        }
      }
    }
    cp_async_wait_all();  // never leave with a copy in flight
  } else if (warp == kMmaWarp) {
    // ===================================================================== MMA issue
    // One warp issues both products, whichever is ready, the value product first: its completion is what
    // the next rows wait for, those of the second part only for dims 384..511. The tensor core queues some
    // of the instructions, so looking for the next part costs it little.
    // S(t) waits until the softmax has read S(t - 1) out of the only buffer.
    const bool leader = elect_one();
    n_tiles = __shfl_sync(0xffffffffu, n_tiles, 0);
    constexpr uint32_t idesc_qk = idesc_bf16_f32(128, kBN, false, false);
    constexpr uint32_t idesc_pv = idesc_bf16_f32(128, kHG, true, false);
    static_assert(kQTmem == kFirstChunks, "the first part of a tile meets the queries in tensor memory");
    auto ready = [&](int b, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test(bar(b), parity)) != 0; };
    if (n_tiles > 0) failed = __any_sync(0xffffffffu, !mbar_wait(bar(kBarQT), 0));
    int ts = 0, part = 0, to = 0;  // next score product and its next part, next value product
    uint32_t idle = 0;
    unsigned long long t0 = 0;
#pragma unroll 1
    while (to < n_tiles && !failed) {
      if (to < ts && ready(kBarPFull, to & 1)) {
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const int j = (jj + 3) & 3;
#pragma unroll
            for (int ks = 0; ks < kBN / 16; ++ks)
              tc_mma_f16(tmem + kColO + 64u * j, smem_desc_mn128(chunk_at(to, 2 * j) + uint32_t(ks) * 2048u, kChunkBytes, 1024),
                         smem_desc_k128(s_p) + uint64_t(2 * ks), idesc_pv, (to > 0 || ks > 0) ? 1u : 0u);
            if (jj == 0) tc_commit(bar(kBarRestFree + (to & 1)));
          }
          tc_commit(bar(kBarFree + to % 3));
          if (to == n_tiles - 1) tc_commit(bar(kBarOFull));
        }
        __syncwarp();
        DSA_STAMP_IF(leader && to == 4, scta, 8);
        ++to;
        idle = 0, t0 = 0;
      } else if (ts < n_tiles && part == 0 && (ts == 0 || ready(kBarSRead, (ts - 1) & 1)) && ready(kBarFirst + ts % 3, (ts / 3) & 1)) {
        tc_fence_after();
        DSA_STAMP_IF(leader && ts == 4, scta, 5);
        if (leader) {
#pragma unroll
          for (int c = 0; c < kFirstChunks; ++c)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tc_mma_f16_ts(tmem + kColS, tmem + kColQ + uint32_t(32 * c + 8 * ks), smem_desc_k128(chunk_at(ts, c)) + uint64_t(2 * ks),
                            idesc_qk, (c | ks) ? 1u : 0u);
        }
        __syncwarp();
        part = 1;
        idle = 0, t0 = 0;
      } else if (ts < n_tiles && part == 1 && ready(kBarRest + (ts & 1), (ts >> 1) & 1)) {
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int c = kFirstChunks; c < kChunks; ++c)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tc_mma_f16(tmem + kColS, smem_desc_k128(s_q + uint32_t(c - kQTmem) * kChunkBytes) + uint64_t(2 * ks),
                         smem_desc_k128(chunk_at(ts, c)) + uint64_t(2 * ks), idesc_qk, 1u);
          tc_commit(bar(kBarSFull));
        }
        __syncwarp();
        DSA_STAMP_IF(leader && ts == 4, scta, 6);
        part = 0;
        ++ts;
        idle = 0, t0 = 0;
      } else if ((++idle & 255u) == 0u) {  // bounded, as mbar_wait is
        const unsigned long long now = wall_ns();
        if (t0 == 0) t0 = now;
        failed = __any_sync(0xffffffffu, now - t0 > kWaitLimitNs);
      }
    }
  } else if (warp < 6) {
    // ===================================================================== softmax, rescale, epilogue
    const int quad = warp & 3;                   // TMEM lanes [32 quad, 32 quad + 32)
    const int half = warp >> 2;                  // key columns [32 half, 32 half + 32) of a tile
    const uint32_t tq = tmem + (uint32_t(quad * 32) << 16);
    const bool soft = quad < 2;                  // lanes 0..63 hold the 64 real S rows
    const int head = quad * 32 + lane;
    if (warp < 2 && n_tiles > 0) {
      // the first kQTmem chunks of Q into tensor memory (rows 64..127 stay as they are: the score rows that
      // they feed are read by nobody)
      failed = __any_sync(0xffffffffu, !mbar_wait(bar(kBarQ), 0));
#pragma unroll
      for (int c = 0; c < kQTmem; ++c) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 x = *reinterpret_cast<const uint4*>(smem + (chunk_at(2, c) - sbase) + swz(head, i));
          v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
        }
        tmem_st_32x32(tq + kColQ + 32u * c, v);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar(kBarQT));
    }
    for (int t = 0; t < n_tiles; ++t) {          // left only through the uniform vote below
      const int s = t & 1;
      float x[32];
      if (soft) {
        // (tcgen05.ld is warp-collective, so the outcome of the wait is made warp-uniform)
        // key j of the tile was staged by producer warp (j % kRowsPerPass) >> 2 in its pass
        // j / kRowsPerPass: bit 4 pass + (j & 3) of that warp's word (read while the scores are computed)
        constexpr int kHalfPasses = kPasses / 2;  // passes that make up 32 keys
        uint32_t vw[kProdWarps], vall = 0xFFFFFFFFu;
        failed = __any_sync(0xffffffffu, failed || !mbar_wait(bar(kBarRest + s), (t >> 1) & 1));
#pragma unroll
        for (int w = 0; w < kProdWarps; ++w) {
          vw[w] = s_validw[s * kProdWarps + w] >> (4 * kHalfPasses * half);
          vall &= vw[w];
        }
        failed = __any_sync(0xffffffffu, failed || !mbar_wait(bar(kBarSFull), t & 1));
        tc_fence_after();
        DSA_STAMP_IF(tid == 0 && t == 4, scta, 9);
        float m_loc = -INFINITY;
        if (!failed) {
          uint32_t raw[32];
          tmem_ld_32x32(tq + kColS + 32u * half, raw);
          tmem_ld_wait();
          tc_fence_before();
          mbar_arrive(bar(kBarSRead));
          // x keeps the raw dot products (-inf for masked keys); the softmax scale (> 0) is
          // applied to the maximum here and folded into the exponent's multiply-add below
          if ((vall & ((1u << (4 * kHalfPasses)) - 1u)) == (1u << (4 * kHalfPasses)) - 1u) {  // every key of the half-tile visible
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(raw[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const bool ok = (vw[(i % kRowsPerPass) >> 2] >> ((i / kRowsPerPass) * 4 + (i & 3))) & 1u;
              x[i] = ok ? __uint_as_float(raw[i]) : -INFINITY;
            }
          }
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], x[i]);
          m_loc = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;
          if (m_ref != -INFINITY && m_loc > m_ref + kRescaleLog2) s_flag[s] = 1;
        }
        s_max[(s * 2 + half) * kHG + head] = m_loc;
      }
      if (group_sync_or(failed)) { failed = true; break; }
      DSA_STAMP_IF(tid == 0 && t == 4, scta, 10);
      float m_tile = -INFINITY;
      if (soft) m_tile = fmaxf(s_max[(s * 2) * kHG + head], s_max[(s * 2 + 1) * kHG + head]);
      if (s_flag[s]) {
        // rare: some head's maximum ran away from its reference; scale its O^T column
        if (__any_sync(0xffffffffu, t >= 1 && !mbar_wait(bar(kBarFree + (t + 2) % 3), ((t - 1) / 3) & 1)))
          failed = true;
        tc_fence_after();
        if (soft) {
          float f = 1.f;
          if (m_ref != -INFINITY && m_tile > m_ref + kRescaleLog2) {
            f = exp2f(m_ref - m_tile);
            l_run *= f;
            m_ref = m_tile;
          }
          if (half == 0) s_factor[head] = f;
        }
        group_sync();
        if (warp < 4 && !failed) {
#pragma unroll 1
          for (int blk = 0; blk < 8; ++blk) {
            uint32_t o[32];
            tmem_ld_32x32(tq + kColO + 32u * blk, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * s_factor[(blk & 1) * 32 + i]);
            tmem_st_32x32(tq + kColO + 32u * blk, o);
          }
          tmem_st_wait();
        }
        tc_fence_before();
        group_sync();
        if (tid == 0) s_flag[s] = 0;
      }
      if (soft && !failed) {
        if (m_ref == -INFINITY) m_ref = m_tile;
        const float mr = m_ref == -INFINITY ? 0.f : m_ref;  // every key so far masked: all p = 0
        // the row sum uses the rounded probabilities that the value product will see
        uint32_t pk[16];
        float psum0 = 0.f, psum1 = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(ex2_approx(fmaf(x[2 * i], p.scale_log2, -mr)),
                                                         ex2_approx(fmaf(x[2 * i + 1], p.scale_log2, -mr)));
          pk[i] = *reinterpret_cast<const uint32_t*>(&b);
          psum0 += __uint_as_float(pk[i] << 16);
          psum1 += __uint_as_float(pk[i] & 0xFFFF0000u);
        }
        l_run += psum0 + psum1;
        DSA_STAMP_IF(tid == 0 && t == 4, scta, 11);
        // P is single-buffered: the previous tile's value product must have read it
        if (t >= 1 && !mbar_wait(bar(kBarFree + (t + 2) % 3), ((t - 1) / 3) & 1)) failed = true;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          st_shared_v4(s_p + uint32_t(head * 128 + (((half * 4 + u) ^ (head & 7)) << 4)),
                       make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]));
        fence_proxy_async_smem();
        tc_fence_before();
        mbar_arrive(bar(kBarPFull));
        DSA_STAMP_IF(tid == 0 && t == 4, scta, 12);
        DSA_STAMP_IF(tid == 0 && t == 5, scta, 13);
      }
    }
    DSA_STAMP(scta, 2);
    // the two column halves of a head add their sums
    if (soft && half == 1) s_factor[head] = l_run;
    group_sync();
    if (soft && half == 0) {
      l_run += s_factor[head];
      s_factor[head] = l_run > 0.f ? 1.f / l_run : 0.f;  // (read only by this thread above)
    }
  }
  __syncthreads();

  if (warp < 4 * kEpiGroups) {
    // ---- partials of this split: O^T (lane = value dim, column = head), reference m, sum l; or,
    // when there is only one split, the normalised bf16 result itself (what the merge kernel would
    // make of the partials: 256 KB less traffic per row and 128 heads, and one launch less). Every warp
    // reaches the lane quadrant (warp % 4): the column blocks are shared out over three groups of four
    // (one group: 4100 cycles of a CTA's 75 000 at 24 tiles).
    const int quad = warp & 3;
    const uint32_t tq = tmem + (uint32_t(quad * 32) << 16);
    const int64_t pbase = (int64_t(r) * p.nsplit + split) * p.H + hg * kHG;
    bool have = n_tiles > 0 && !__any_sync(0xffffffffu, failed);
    if (__any_sync(0xffffffffu, have && !mbar_wait(bar(kBarOFull), 0))) have = false, failed = true;
    tc_fence_after();
    DSA_STAMP(scta, 7);
#pragma unroll 1
    for (int blk = warp >> 2; blk < 8; blk += kEpiGroups) {
      uint32_t o[32];
      if (have) {
        tmem_ld_32x32(tq + kColO + 32u * blk, o);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0u;
      }
      const int dim = (blk >> 1) * 128 + quad * 32 + lane;
      if (p.out) {
        __nv_bfloat16* dst = p.out + (int64_t(r) * p.H + hg * kHG + (blk & 1) * 32) * mla::kDV + dim;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          dst[i * mla::kDV] = __float2bfloat16_rn(__uint_as_float(o[i]) * s_factor[(blk & 1) * 32 + i]);
      } else {
        float* dst = p.part_acc + (pbase + (blk & 1) * 32) * mla::kDV + dim;
#pragma unroll
        for (int i = 0; i < 32; ++i) dst[int64_t(i) * mla::kDV] = __uint_as_float(o[i]);
      }
    }
    if (tid < kHG && !p.out) {
      p.part_m[pbase + tid] = have ? m_ref : -INFINITY;
      p.part_l[pbase + tid] = have ? l_run : 0.f;
    }
  }

  if (failed) {
    atomicOr(&g_device_status, kStatusAttnTimeout);
    drain_after_timeout();  // let outstanding copies and MMAs drain
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, kTmemCols);
  if constexpr (kBeside) pdl_wait();
  DSA_STAMP(scta, 15);
  DSA_KTIME_END(2);
}

}  // namespace mla_tc
}  // namespace dsa
