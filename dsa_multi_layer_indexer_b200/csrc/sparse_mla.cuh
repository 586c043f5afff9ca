// Split-K sparse MLA decode over the selected latent rows, plus the
// log-sum-exp merge of the split partials.
//
//   out[r,h,:] = softmax_j(scale * q[r,h,:] . kv[idx_j,:]) . kv[idx_j,:512]
//
// Same arithmetic as the reference's attention warps and combine kernel
// (kernels/cuda_fused_sparse_splitk.py:282-530, :996-1045; host form
// ref_sparse_mla :2950-2966): bf16 operands, fp32 accumulation, base-2 online
// softmax, probabilities rounded to bf16 before the value product.
//
// One CTA = (query row, one or two blocks of 16 heads, one split of the index list). The
// 1152-byte latent rows are gathered with one bulk asynchronous copy per row
// (TMA engine, completion counted on an mbarrier) into padded shared-memory
// rows, so the gather costs one instruction per row instead of 72 16-byte
// copies per row. FP8 latent rows (656 B) are staged the same way and
// dequantised into the bf16 tile exactly as the reference does
// (fp8 -> f32, x group scale, round to bf16; :1181-1196).
//
// What bounds it (one 64-key bf16 tile per CTA, cycles after the dependency wait; 16 heads alone on an SM / two such CTAs on it):
// selection entries 900, rows and queries landed 2400-3400 / 3550 (an SM gets 45-61 bytes a cycle from L2), scores 1250 / 2280
// and values 750 / 1170 (shared-memory reads: 148 and 65 KB a CTA), maximum, softmax and their barriers 600 / 800, partials
// 1280-1390 / 1500, and 200 / 920 until the CTA's last warp has stored and added up.
#pragma once


#include "common.cuh"

namespace dsa {
namespace mla {

constexpr int kD = DSA_LATENT_DIM;       // 576
constexpr int kDV = DSA_VALUE_DIM;       // 512
constexpr int kHB = DSA_HEAD_BLOCK;      // heads of a block
constexpr int kBN = 64;                  // keys per tile
constexpr int kSlices = 8;               // groups of eight keys of a tile, each summed by itself
constexpr int kRowBytes = kD * 2;        // 1152
constexpr int kRowPitch = kRowBytes + 16;  // 1168: 8 consecutive rows hit 8 distinct bank groups
constexpr int kPPitch = (kBN + 8) * 2;   // bf16 probabilities, padded the same way
constexpr int kFp8Row = DSA_FP8_LATENT_ROW;

struct Params {
  const __nv_bfloat16* q;
  const uint8_t* kv;
  const int32_t* indices;
  const int32_t* seq_lens;
  float* part_acc;
  float* part_m;
  float* part_l;
  int64_t kv_seq_stride;  // rows per cached sequence
  int64_t ctx;            // dense mode: key capacity
  int rows_per_seq;
  int H;
  int topk;
  int nsplit;
  int keys_per_split;
  int kv_fp8;
  float scale_log2;       // sm_scale * log2(e)
  __nv_bfloat16* out;     // one split only: the normalised result goes here and no partials are written
};

// MT blocks of 16 heads share a CTA's gathered rows, NB tiles are on their way or in use at once.
template <int MT, int NB>
struct SmemLayout {
  static constexpr int q_off = 0;
  static constexpr int k_off = q_off + MT * kHB * kRowPitch;
  static constexpr int p_off = k_off + NB * kBN * kRowPitch;
  static constexpr int red_off = p_off + MT * kHB * kPPitch;             // float [2][8][16 MT]
  static constexpr int swap_off = red_off + 2 * kSlices * MT * kHB * 4;  // float4 [8][MT][32]
  static constexpr int valid_off = swap_off + (MT == 1 ? 0 : kSlices * MT * 32 * 16);  // int [NB][64] (four warps swap nothing)
  static constexpr int bar_off = valid_off + NB * kBN * 4;               // 1 + 2 NB mbarriers
  static constexpr int bytes = (bar_off + 8 * (1 + 2 * NB) + 15) & ~15;
};
// Two CTAs of one head block (and 1 KB of the system's each) fit the 196 KB configuration that the scan and the top-k run
// in. An SM is drained before its configuration changes: at 101 KB a CTA, which takes the 228 KB one, a layer of 128 heads
// and 512 keys took 19.1 us instead of 17.2, its two-stream form 12.9 instead of 10.3.
static_assert(2 * (SmemLayout<1, 1>::bytes + 1024) <= 196 * 1024, "sparse MLA: two CTAs of one head block share an SM");
static_assert(SmemLayout<2, 2>::bytes <= 232448, "sparse MLA: shared memory over the per-CTA limit");

// Barrier over the attention CTA's W warps (named barrier 1: in the fused launch others may have left).
template <int W>
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory"); }
// The same barrier that also ORs a flag over the threads: every thread gets the same answer.
template <int W>
__device__ __forceinline__ bool cta_any(bool flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(uint32_t(flag)), "n"(32 * W)
      : "memory");
  return r != 0;
}
// Barrier of the two warps that share a key group (named barriers 2..5).
__device__ __forceinline__ void pair_sync(int key_group) {
  asm volatile("bar.sync %0, 64;" ::"r"(2 + key_group) : "memory");
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 4 packed e4m3 -> 4 bf16 with one fp32 scale: fp8 -> f16 (exact) -> f32 -> * s -> bf16 RN
__device__ __forceinline__ uint2 dequant4(uint32_t w, float s) {
  const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w & 0xFFFFu), __NV_E4M3);
  const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w >> 16), __NV_E4M3);
  const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&lo));
  const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  const __nv_bfloat162 b01 = __floats2bfloat162_rn(f01.x * s, f01.y * s);
  const __nv_bfloat162 b23 = __floats2bfloat162_rn(f23.x * s, f23.y * s);
  uint2 r;
  r.x = *reinterpret_cast<const uint32_t*>(&b01);
  r.y = *reinterpret_cast<const uint32_t*>(&b23);
  return r;
}

// One 64-key tile for the 16 MT heads of a CTA of W = 4 or 8 warps: S = Q K^T on bf16 tensor cores,
// base-2 online softmax across the warps, P rounded to bf16, O += P V.
// Scores: of eight warps (dh, kg) multiplies keys [16 kg, 16 kg + 16) with half dh of the dims; the two warps of
// a key group then swap, so that each holds the sums of eight keys for the softmax. Of four warps each does both
// halves and holds sixteen keys: the same sums, added in the same order. Values: warp w owns 512 / W columns.
// `landed` is this thread's outcome of its wait for the tile; where one ran out, all threads leave together
// with false. Contains two block barriers.
template <int MT, int W>
__device__ __forceinline__ bool attend_tile(const uint8_t* s_q, const uint8_t* s_k, uint8_t* s_p,
                                            float* s_red, float4* s_swap, const int* s_valid, float scale_log2,
                                            bool landed, int warp, int lane, float (&m_run)[MT][2],
                                            float (&l_run)[MT][8 / W][2], float (&acc)[MT][kDV / 8 / W][4]) {
  constexpr int kRows = MT * kHB, NS = kSlices / W;  // NS slices of eight keys per warp
  const int g = lane >> 2, t4 = lane & 3, kg = warp & 3, dh = warp >> 2;  // (dh = 0 of four warps)
  float x[MT][NS][4];
  {
    const uint32_t a_base = smem_u32(s_q + (lane & 15) * kRowPitch + (lane >> 4) * 16) + dh * kD;  // (half a row: kD bytes)
    const uint32_t b_base = smem_u32(s_k + (kg * 16 + (lane & 7) + 8 * (lane >> 4)) * kRowPitch +
                                     ((lane >> 3) & 1) * 16) + dh * kD;
    float sc[NS][MT][2][4];  // [half of the dims][head block][slice]
#pragma unroll
    for (int hf = 0; hf < NS; ++hf)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[hf][mt][0][e] = sc[hf][mt][1][e] = 0.f;
#pragma unroll 3
    for (int k0 = 0; k0 < kD / 2; k0 += 16) {
#pragma unroll
      for (int hf = 0; hf < NS; ++hf) {
        uint32_t b[4];
        ldsm_x4(b_base + hf * kD + k0 * 2, b);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          uint32_t a[4];
          ldsm_x4(a_base + hf * kD + mt * kHB * kRowPitch + k0 * 2, a);
          mma_bf16(sc[hf][mt][0], a, b[0], b[1]);
          mma_bf16(sc[hf][mt][1], a, b[2], b[3]);
        }
      }
    }
    if constexpr (W == 8) {  // this warp keeps keys [16 kg + 8 dh, + 8)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float4 give;
        give.x = dh ? sc[0][mt][0][0] : sc[0][mt][1][0];
        give.y = dh ? sc[0][mt][0][1] : sc[0][mt][1][1];
        give.z = dh ? sc[0][mt][0][2] : sc[0][mt][1][2];
        give.w = dh ? sc[0][mt][0][3] : sc[0][mt][1][3];
        s_swap[(warp * MT + mt) * 32 + lane] = give;
      }
      pair_sync(kg);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const float4 o = s_swap[((warp ^ 4) * MT + mt) * 32 + lane];
        x[mt][0][0] = (dh ? sc[0][mt][1][0] : sc[0][mt][0][0]) + o.x;
        x[mt][0][1] = (dh ? sc[0][mt][1][1] : sc[0][mt][0][1]) + o.y;
        x[mt][0][2] = (dh ? sc[0][mt][1][2] : sc[0][mt][0][2]) + o.z;
        x[mt][0][3] = (dh ? sc[0][mt][1][3] : sc[0][mt][0][3]) + o.w;
      }
    } else {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int n = 0; n < NS; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[mt][n][e] = sc[0][mt][n][e] + sc[NS - 1][mt][n][e];
    }
  }
  // scale, mask, tile max per head row (rows g and g + 8 of a block); slice `dh + n` of the key group
  const auto column = [&](int n) { return kg * 16 + (dh + n) * 8 + t4 * 2; };
#pragma unroll
  for (int n = 0; n < NS; ++n) {
    const bool v0 = s_valid[column(n)] != 0, v1 = s_valid[column(n) + 1] != 0;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      x[mt][n][0] = v0 ? x[mt][n][0] * scale_log2 : -INFINITY;
      x[mt][n][1] = v1 ? x[mt][n][1] * scale_log2 : -INFINITY;
      x[mt][n][2] = v0 ? x[mt][n][2] * scale_log2 : -INFINITY;
      x[mt][n][3] = v1 ? x[mt][n][3] * scale_log2 : -INFINITY;
    }
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    float tmax[2] = {fmaxf(x[mt][0][0], x[mt][0][1]), fmaxf(x[mt][0][2], x[mt][0][3])};
#pragma unroll
    for (int n = 1; n < NS; ++n) {
      tmax[0] = fmaxf(tmax[0], fmaxf(x[mt][n][0], x[mt][n][1]));
      tmax[1] = fmaxf(tmax[1], fmaxf(x[mt][n][2], x[mt][n][3]));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      tmax[i] = fmaxf(tmax[i], __shfl_xor_sync(0xffffffffu, tmax[i], 1));
      tmax[i] = fmaxf(tmax[i], __shfl_xor_sync(0xffffffffu, tmax[i], 2));
    }
    if (t4 == 0) {
      s_red[warp * kRows + mt * kHB + g] = tmax[0];
      s_red[warp * kRows + mt * kHB + g + 8] = tmax[1];
    }
  }
  if (cta_any<W>(!landed)) return false;
  float alpha[MT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = mt * kHB + g + 8 * i;
      float m = m_run[mt][i];
#pragma unroll
      for (int w = 0; w < W; ++w) m = fmaxf(m, s_red[w * kRows + row]);
      alpha[mt][i] = (m == -INFINITY) ? 1.f : exp2f(m_run[mt][i] - m);
      m_run[mt][i] = m;
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      float pr[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float m = m_run[mt][e >> 1];
        pr[e] = (m == -INFINITY) ? 0.f : exp2f(x[mt][n][e] - m);
      }
      const __nv_bfloat162 p01 = __floats2bfloat162_rn(pr[0], pr[1]);
      const __nv_bfloat162 p23 = __floats2bfloat162_rn(pr[2], pr[3]);
      // the row sum uses the rounded probabilities that P.V will see; each thread keeps the sum of its own keys,
      // the CTA's are added up once, at the end
      l_run[mt][n][0] = l_run[mt][n][0] * alpha[mt][0] + (__bfloat162float(p01.x) + __bfloat162float(p01.y));
      l_run[mt][n][1] = l_run[mt][n][1] * alpha[mt][1] + (__bfloat162float(p23.x) + __bfloat162float(p23.y));
      *reinterpret_cast<__nv_bfloat162*>(s_p + (mt * kHB + g) * kPPitch + column(n) * 2) = p01;
      *reinterpret_cast<__nv_bfloat162*>(s_p + (mt * kHB + g + 8) * kPPitch + column(n) * 2) = p23;
    }
  }
  cta_sync<W>();
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int i = 0; i < kDV / 8 / W; ++i) {
      acc[mt][i][0] *= alpha[mt][0];
      acc[mt][i][1] *= alpha[mt][0];
      acc[mt][i][2] *= alpha[mt][1];
      acc[mt][i][3] *= alpha[mt][1];
    }

  // ---- O += P V: warp w owns value columns [512 / W w, 512 / W (w + 1))
  {
    const uint32_t a_base = smem_u32(s_p + (lane & 15) * kPPitch + (lane >> 4) * 16);
    const uint32_t b_base = smem_u32(s_k + ((lane & 7) + 8 * ((lane >> 3) & 1)) * kRowPitch +
                                     (warp * (kDV / W) + 8 * (lane >> 4)) * 2);
#pragma unroll
    for (int ks = 0; ks < kBN / 16; ++ks) {
      uint32_t a[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) ldsm_x4(a_base + mt * kHB * kPPitch + ks * 32, a[mt]);
#pragma unroll
      for (int np = 0; np < kDV / 16 / W; ++np) {
        uint32_t b[4];
        ldsm_x4_t(b_base + ks * 16 * kRowPitch + np * 32, b);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_bf16(acc[mt][2 * np], a[mt], b[0], b[1]);
          mma_bf16(acc[mt][2 * np + 1], a[mt], b[2], b[3]);
        }
      }
    }
  }
  return true;
}

// Every thread's sums of its own keys, the four lanes of a head row added up, where sum_of can read them
// behind a block barrier.
template <int MT, int W>
__device__ __forceinline__ void post_sums(float* s_red, int warp, int lane, const float (&l_run)[MT][8 / W][2]) {
  float* s_sum = s_red + kSlices * MT * kHB;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int n = 0; n < kSlices / W; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float s = l_run[mt][n][i];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if ((lane & 3) == 0) s_sum[(warp + 4 * n) * MT * kHB + mt * kHB + (lane >> 2) + 8 * i] = s;
      }
}
template <int MT>
__device__ __forceinline__ float sum_of(const float* s_red, int row) {
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < kSlices; ++w) s += s_red[(kSlices + w) * MT * kHB + row];
  return s;
}

// Dequantises a staged fp8 tile in place: the 656 staged bytes of a row sit at
// the END of that row's 1152-byte bf16 slot (offset 496), so no separate staging
// buffer is needed and the fp8 path keeps two CTAs per SM. Expanding a chunk
// overwrites bytes other threads may still have to read, so the tile is done in
// three passes of "load into registers, barrier, store", ordered so that a pass
// only overwrites sources of chunks already expanded or loaded:
//   chunks 0..15  read [496,752)   write [0,512)
//   chunks 16..23 read [752,880)   write [512,768)
//   chunks 24..31 + rope read [880,1152) write [768,1152)
// The four group scales sit at [1008,1024) and are read before the last stores.
constexpr int kFp8StageOff = kRowBytes - kFp8Row;  // 496
template <int FIRST, int NDEQ, int NROPE, int W>
__device__ __forceinline__ void dequant_pass(uint8_t* s_k, const int* s_valid, int tid) {
  constexpr int kPerRow = NDEQ + NROPE, kThreads = 32 * W;
  constexpr int kPer = (kBN * kPerRow) / kThreads;
  static_assert((kBN * kPerRow) % kThreads == 0, "items must divide evenly");
  uint4 raw[kPer];
  float sc[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int i = tid + u * kThreads, row = i / kPerRow, k = i - row * kPerRow;
    const uint8_t* src = s_k + row * kRowPitch + kFp8StageOff;
    raw[u] = make_uint4(0, 0, 0, 0);
    sc[u] = 0.f;
    if (s_valid[row]) {
      if (k < NDEQ) {
        raw[u] = *reinterpret_cast<const uint4*>(src + (FIRST + k) * 16);
        sc[u] = *reinterpret_cast<const float*>(src + 512 + ((FIRST + k) >> 3) * 4);
      } else {
        raw[u] = *reinterpret_cast<const uint4*>(src + 528 + (k - NDEQ) * 16);
      }
    }
  }
  cta_sync<W>();
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int i = tid + u * kThreads, row = i / kPerRow, k = i - row * kPerRow;
    if (!s_valid[row]) continue;  // masked rows were cleared at gather time
    uint8_t* rowp = s_k + row * kRowPitch;
    if (k < NDEQ) {
      const int c = FIRST + k;
      const uint2 d0 = dequant4(raw[u].x, sc[u]), d1 = dequant4(raw[u].y, sc[u]);
      const uint2 d2 = dequant4(raw[u].z, sc[u]), d3 = dequant4(raw[u].w, sc[u]);
      *reinterpret_cast<uint4*>(rowp + c * 32) = make_uint4(d0.x, d0.y, d1.x, d1.y);
      *reinterpret_cast<uint4*>(rowp + c * 32 + 16) = make_uint4(d2.x, d2.y, d3.x, d3.y);
    } else {
      *reinterpret_cast<uint4*>(rowp + 1024 + (k - NDEQ) * 16) = raw[u];
    }
  }
}
template <int W>
__device__ __forceinline__ void dequant_tile_inplace(uint8_t* s_k, const int* s_valid, int tid) {
  dequant_pass<0, 16, 0, W>(s_k, s_valid, tid);
  dequant_pass<16, 8, 0, W>(s_k, s_valid, tid);
  dequant_pass<24, 8, 8, W>(s_k, s_valid, tid);
}

// Body of the split-K partials for CTA (split, hg, r); `smem` is the CTA's
// dynamic shared memory. Threads 0..32 W - 1 take part.
// kBeside: the launch does not depend on the kernel enqueued just before it (under the lagged
// schedule the attention reads the PREVIOUS layer's selection while this layer's top-k runs), so
// it releases its own dependents and starts at once, beside that kernel, and waits for it only
// before it exits: it still completes after it, and the next kernel's wait covers both.
// kDirect: the split is the only one and writes the result itself.
// MT: blocks of 16 heads per CTA; hg counts blocks of 16 MT heads. NB: row buffers (one block: one, since two CTAs share an SM
// and cover each other's gathers). kMayExpand: rows may be fp8. A launch over bf16 rows carries no code for that: one row of
// 64 heads 21.7 -> 21.45 us a layer, 8 of 16 heads chained 21.8 -> 20.85, 16 of 32 37.6 -> 37.0; fp8 rows in an instantiation of
// their own were slower (one row of 128 heads 23.65 -> 24.0: the 32-head form then spills 112 bytes).
template <bool kBeside, bool kDirect, bool kMayExpand, int MT, int W, int NB>
__device__ __forceinline__ void mla_partials_body(const Params& p, const int split, const int hg, const int r,
                                                  uint8_t* smem) {
  constexpr int kRowsPerWarp = kBN / W;  // latent rows of a tile that a warp requests
  using L = SmemLayout<MT, NB>;
  constexpr int kHeads = MT * kHB;
  uint8_t* s_q = smem + L::q_off;
  uint8_t* s_k = smem + L::k_off;
  uint8_t* s_p = smem + L::p_off;
  float* s_red = reinterpret_cast<float*>(smem + L::red_off);
  float4* s_swap = reinterpret_cast<float4*>(smem + L::swap_off);
  int* s_valid = reinterpret_cast<int*>(smem + L::valid_off);
  const uint32_t bar_q = smem_u32(smem + L::bar_off);
  const auto bar_k = [&](int buf, int half) { return bar_q + 8u * uint32_t(1 + 2 * buf + half); };  // rows 0..31, 32..63 of a tile

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  DSA_KTIME_BEGIN(2);
  const int seq = r / p.rows_per_seq;
  const bool fp8 = kMayExpand && p.kv_fp8;
  const int row_bytes = fp8 ? kFp8Row : kRowBytes;
  const uint8_t* kv_seq = p.kv + int64_t(seq) * p.kv_seq_stride * row_bytes;

  if (tid == 0) {
    mbar_init(bar_q, W);
    for (int i = 0; i < 2 * NB; ++i) mbar_init(bar_k(i >> 1, i & 1), W / 2);
    mbar_fence_init();
  }
  cta_sync<W>();
  if constexpr (!kBeside) pdl_wait();  // the selection, the queries and the lengths may come from the previous kernel
  pdl_launch_dependents();
  // The first tile's selection entries are requested before the row's length is looked at: two
  // loads in flight together instead of two trips to global memory one after the other.
  const int k_begin = split * p.keys_per_split;
  const int k_end = min(k_begin + p.keys_per_split, p.topk);
  const int n_tiles = (max(k_end - k_begin, 0) + kBN - 1) / kBN;
  const int my_row = warp * kRowsPerWarp + lane;  // (lanes 0..kRowsPerWarp - 1)
  const auto entry = [&](int tile) {
    const int j = k_begin + tile * kBN + my_row;
    if (lane >= kRowsPerWarp || j >= k_end) return -1;
    return p.indices ? int(p.indices[int64_t(r) * p.topk + j]) : j;
  };
  int idx_next = entry(0);
  // (32 bits, as the entries have: with 64 the 32-head form spilled 28 bytes and the one that shares a launch with the scan 4)
  const int ctx = int(min(p.ctx, int64_t(0x7FFFFFFF)));
  const int len = p.seq_lens ? min(max(p.seq_lens[r], 0), ctx) : ctx;

  // Gather up to 64 latent rows: one bulk copy per valid row, shared out over all warps. (A warp issues its lanes'
  // copies one after the other, 60 cycles each: from two warps the 64 took 1900 cycles whether one CTA or two shared the SM.
  // 16-byte asynchronous copies by all threads instead were slower still: 4608 of them per tile.)
  const auto gather = [&](int tile) {
    const int buf = NB == 1 ? 0 : tile & 1;
    const int idx = idx_next;
    const bool ok = idx >= 0 && idx < len;
    const uint32_t seen = __ballot_sync(0xffffffffu, ok);
    const uint32_t bar = bar_k(buf, warp / (W / 2));
    uint8_t* dst = s_k + (buf * kBN + my_row) * kRowPitch;
    if (lane < kRowsPerWarp) {
      s_valid[buf * kBN + my_row] = ok;
      if (!ok) {
        // masked key: its row must be finite because 0 * NaN would poison P.V
        uint4* z = reinterpret_cast<uint4*>(dst);
        for (int i = 0; i < kRowBytes / 16; ++i) z[i] = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async_smem();  // earlier generic reads of these rows precede the async writes
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_expect_tx(bar, uint32_t(__popc(seen)) * uint32_t(row_bytes));
    __syncwarp();
    if (ok) {
      if (fp8)  // staged at the end of the row's own slot, expanded in place below
        bulk_g2s(smem_u32(dst + kFp8StageOff), kv_seq + int64_t(idx) * kFp8Row, kFp8Row, bar);
      else
        bulk_g2s(smem_u32(dst), kv_seq + int64_t(idx) * kRowBytes, kRowBytes, bar);
    }
    idx_next = entry(tile + 1);
  };
  // Queries of the head blocks, rows of 1152 B: in front of the latent rows with 16 heads (128 heads over 1024 keys, a layer:
  // 19.5 us, behind them 19.75; beside the scan of one launch 28.55 and 28.85), behind them with 32, whose rows are twice as
  // many for as many copies (3 rows of 64 heads: 13.4 us, in front 13.6).
  if (MT > 1 && n_tiles > 0) gather(0);
  {
    constexpr int kPerWarp = kHeads / W;
    if (lane == 0) mbar_arrive_expect_tx(bar_q, kPerWarp * kRowBytes);
    __syncwarp();
    if (lane < kPerWarp) {
      const int h = warp * kPerWarp + lane;
      bulk_g2s(smem_u32(s_q + h * kRowPitch), p.q + (int64_t(r) * p.H + hg * kHeads + h) * kD, kRowBytes, bar_q);
    }
  }
  if (MT == 1 && n_tiles > 0) gather(0);

  const int g = lane >> 2, t4 = lane & 3;
  float m_run[MT][2], l_run[MT][kSlices / W][2];
  float acc[MT][kDV / 8 / W][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    m_run[mt][0] = m_run[mt][1] = -INFINITY;
#pragma unroll
    for (int n = 0; n < kSlices / W; ++n) l_run[mt][n][0] = l_run[mt][n][1] = 0.f;
#pragma unroll
    for (int i = 0; i < kDV / 8 / W; ++i) acc[mt][i][0] = acc[mt][i][1] = acc[mt][i][2] = acc[mt][i][3] = 0.f;
  }
  bool timed_out = false;

  for (int tile = 0; tile < n_tiles; ++tile) {
    const int buf = NB == 1 ? 0 : tile & 1, parity = (NB == 1 ? tile : tile >> 1) & 1;
    if (NB > 1 && tile + 1 < n_tiles) gather(tile + 1);  // (its slot was read before the last barrier)
    uint8_t* tile_k = s_k + buf * kBN * kRowPitch;
    const int* valid = s_valid + buf * kBN;
    // A warp waits for the half of the tile that its key group lies in; each thread runs its own clock, so the
    // threads agree on leaving at the softmax's barrier (fp8 rows: here) and nobody is left alone at a later one.
    bool landed = tile > 0 || mbar_wait(bar_q, 0);
    if (!mbar_wait(bar_k(buf, (warp >> 1) & 1), parity)) landed = false;
    if (fp8) {
      if (!mbar_wait(bar_k(buf, ((warp >> 1) & 1) ^ 1), parity)) landed = false;
      timed_out = cta_any<W>(!landed);
      if (timed_out) break;
      dequant_tile_inplace<W>(tile_k, valid, tid);
      cta_sync<W>();
    }
    timed_out = !attend_tile<MT, W>(s_q, tile_k, s_p, s_red, s_swap, valid, p.scale_log2, landed, warp, lane, m_run, l_run, acc);
    if (timed_out) break;
    if (tile + 1 < n_tiles) {
      cta_sync<W>();  // the K tile and P are free for the next gather
      if (NB == 1) gather(tile + 1);
    }
  }

  if (n_tiles == 0) timed_out = cta_any<W>(!mbar_wait(bar_q, 0));  // never leave with a copy in flight
  if (timed_out) {
    atomicOr(&g_device_status, kStatusAttnTimeout);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      m_run[mt][0] = m_run[mt][1] = -INFINITY;
#pragma unroll
      for (int n = 0; n < kSlices / W; ++n) l_run[mt][n][0] = l_run[mt][n][1] = 0.f;
    }
    drain_after_timeout();  // let outstanding copies land
  }
  post_sums<MT, W>(s_red, warp, lane, l_run);

  if constexpr (kDirect) {  // the only split: what the merge kernel would make of its partials
    cta_sync<W>();
    __nv_bfloat16* out = p.out + (int64_t(r) * p.H + hg * kHeads) * kDV;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const float l0 = sum_of<MT>(s_red, mt * kHB + g), l1 = sum_of<MT>(s_red, mt * kHB + g + 8);
      const float inv0 = l0 > 0.f ? 1.f / l0 : 0.f, inv1 = l1 > 0.f ? 1.f / l1 : 0.f;
#pragma unroll
      for (int i = 0; i < kDV / 8 / W; ++i) {
        __nv_bfloat16* dst = out + (mt * kHB + g) * kDV + warp * (kDV / W) + i * 8 + t4 * 2;
        *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(acc[mt][i][0] * inv0, acc[mt][i][1] * inv0);
        *reinterpret_cast<__nv_bfloat162*>(dst + 8 * kDV) = __floats2bfloat162_rn(acc[mt][i][2] * inv1, acc[mt][i][3] * inv1);
      }
    }
    if constexpr (kBeside) pdl_wait();
    DSA_KTIME_END(2);
    return;
  }
  // ---- partials of this split: unnormalised accumulator, running max (base 2), sum. The 32 MT KB take 1300-1500
  // cycles with 16 heads, 2050-2400 with 32 (25-32 bytes a cycle and SM); the sums' barrier waits in their shadow.
  const int64_t pbase = (int64_t(r) * p.nsplit + split) * p.H + hg * kHeads;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    float* dst = p.part_acc + (pbase + mt * kHB + g) * kDV + warp * (kDV / W) + t4 * 2;
#pragma unroll
    for (int i = 0; i < kDV / 8 / W; ++i) {
      *reinterpret_cast<float2*>(dst + i * 8) = make_float2(acc[mt][i][0], acc[mt][i][1]);
      *reinterpret_cast<float2*>(dst + 8 * kDV + i * 8) = make_float2(acc[mt][i][2], acc[mt][i][3]);
    }
    if (warp == 0 && t4 == 0) {
      p.part_m[pbase + mt * kHB + g] = m_run[mt][0];
      p.part_m[pbase + mt * kHB + g + 8] = m_run[mt][1];
    }
  }
  cta_sync<W>();
  if (tid < kHeads) p.part_l[pbase + tid] = sum_of<MT>(s_red, tid);
  if constexpr (kBeside) pdl_wait();
  DSA_KTIME_END(2);
}

// (instantiations of their own: the direct form's code costs a step 0.1 us)
// (registers: what leaves room for the merge kernel's CTAs, which wait beside this kernel's; nothing waits beside the direct
// form: one fp8 tile of 16 heads 7.6 us with 242 registers, 7.95 with 168)
template <bool kBeside, bool kDirect, bool kMayExpand, int MT, int W, int NB>
__global__ void __launch_bounds__(32 * W, MT == 1 ? (kDirect ? 2 : 3) : kDirect ? 1 : 2)
sparse_mla_partials_kernel(const Params p) {
  extern __shared__ __align__(16) uint8_t mla_smem[];
  mla_partials_body<kBeside, kDirect, kMayExpand, MT, W, NB>(p, blockIdx.x, blockIdx.y, blockIdx.z, mla_smem);
}

// ------------------------------------------------------------------------------
// out = sum_s acc_s 2^(m_s - m) / sum_s l_s 2^(m_s - m); splits with m = -inf
// (no visible key) are skipped, a row with none yields zeros. One CTA per (row,
// head, 1 / kParts of the columns) of 1..4 groups of 128 / kParts threads (the launch picks min(nsplit, 4)):
// group g folds splits g, g + ngrp, ... with all loads of a chunk of eight splits in
// flight at once, then the groups' results are merged in a fixed order, the same for every kParts.
// Bound by two dependent trips to L2 and by the 61 bytes a cycle that an SM gets from there.
template <int kParts, bool kUnrolled>
__global__ void __launch_bounds__(512 / kParts)
sparse_mla_combine_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_m,
                          const float* __restrict__ part_l, __nv_bfloat16* __restrict__ out, int H,
                          int nsplit) {
  constexpr int kCols = kDV / kParts, kGroup = kCols / 4;  // columns of a CTA; threads of a group, four columns each
  __shared__ float s_m[4], s_l[4];
  __shared__ __align__(16) float s_o[4][kCols];
  const int h = blockIdx.x / kParts, c0 = (blockIdx.x % kParts) * kCols, r = blockIdx.y;
  const int tid = threadIdx.x % kGroup, grp = threadIdx.x / kGroup;
  const int ngrp = blockDim.x / kGroup;  // 1..4, each taking every ngrp-th split
  // Final loops unrolled: 0.1-0.2 us less with part of the columns per CTA. With all of them it takes 64 registers instead
  // of 74, and two such CTAs share an SM: with more pairs than SMs that is a wave less (2 rows of 128 heads, 32 splits,
  // attention + merge 13.0 instead of 14.3 us), with fewer a layer of 128 heads takes 25.2 instead of 24.5, though the merge
  // alone is as fast; presumably the next launch's CTAs then come to lie beside these.
  const int groups = kUnrolled ? 4 : ngrp;
  DSA_KTIME_BEGIN(3);
  pdl_wait();
  pdl_launch_dependents();
  const float* pm = part_m + int64_t(r) * nsplit * H + h;
  const float* pl = part_l + int64_t(r) * nsplit * H + h;
  const float* pa = part_acc + (int64_t(r) * nsplit * H + h) * kDV + c0 + tid * 4;
  float mg = -INFINITY, lg = 0.f;
  float4 og = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = grp; s0 < nsplit; s0 += 8 * ngrp) {
    float ms[8], ls[8];
    float4 a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int sp = s0 + ngrp * u;
      const bool ok = sp < nsplit;
      ms[u] = ok ? pm[int64_t(sp) * H] : -INFINITY;
      ls[u] = ok ? pl[int64_t(sp) * H] : 0.f;
      a[u] = ok ? *reinterpret_cast<const float4*>(pa + int64_t(sp) * H * kDV) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float m_new = mg;
#pragma unroll
    for (int u = 0; u < 8; ++u) m_new = fmaxf(m_new, ms[u]);
    if (m_new != -INFINITY) {
      const float keep = (mg == -INFINITY) ? 0.f : exp2f(mg - m_new);
      lg *= keep;
      og.x *= keep;
      og.y *= keep;
      og.z *= keep;
      og.w *= keep;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float e = (ms[u] == -INFINITY) ? 0.f : exp2f(ms[u] - m_new);
        lg = fmaf(ls[u], e, lg);
        og.x = fmaf(a[u].x, e, og.x);
        og.y = fmaf(a[u].y, e, og.y);
        og.z = fmaf(a[u].z, e, og.z);
        og.w = fmaf(a[u].w, e, og.w);
      }
    }
    mg = m_new;
  }
  if (tid == 0) {
    s_m[grp] = mg;
    s_l[grp] = lg;
  }
  *reinterpret_cast<float4*>(&s_o[grp][tid * 4]) = og;
  __syncthreads();
  if (grp == 0) {
    float m = s_m[0];
#pragma unroll
    for (int gi = 1; gi < groups; ++gi) m = gi < ngrp ? fmaxf(m, s_m[gi]) : m;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    if (m != -INFINITY) {
#pragma unroll
      for (int gi = 0; gi < groups; ++gi) {
        if (gi >= ngrp) break;
        const float e = (s_m[gi] == -INFINITY) ? 0.f : exp2f(s_m[gi] - m);
        const float4 a = *reinterpret_cast<const float4*>(&s_o[gi][tid * 4]);
        l = fmaf(s_l[gi], e, l);
        o.x = fmaf(a.x, e, o.x);
        o.y = fmaf(a.y, e, o.y);
        o.z = fmaf(a.z, e, o.z);
        o.w = fmaf(a.w, e, o.w);
      }
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    __nv_bfloat162 lo = __floats2bfloat162_rn(o.x * inv, o.y * inv);
    __nv_bfloat162 hi = __floats2bfloat162_rn(o.z * inv, o.w * inv);
    uint2 pk;
    pk.x = *reinterpret_cast<uint32_t*>(&lo);
    pk.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(out + (int64_t(r) * H + h) * kDV + c0 + tid * 4) = pk;
  }
  DSA_KTIME_END(3);
}

// The same merge for many (row, head) pairs: one thread per four output columns, kUnroll splits' loads
// in flight at once, no shared memory; splits are folded in ascending order, kUnroll at a time. L2-bound:
// 16.8 MB of partials (512 pairs x 16 splits) in 3.3 us, where a CTA per pair with its loads spread over
// four thread groups takes 8.0.
template <int kUnroll>
__global__ void __launch_bounds__(128)
sparse_mla_combine_flat_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_m,
                               const float* __restrict__ part_l, __nv_bfloat16* __restrict__ out, int H,
                               int nsplit) {
  DSA_KTIME_BEGIN(3);
  pdl_wait();
  pdl_launch_dependents();
  const int64_t pair = blockIdx.x;  // row * H + head
  const int64_t r = pair / H, h = pair % H;
  const int c4 = threadIdx.x;
  float m = -INFINITY, l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < nsplit; s0 += kUnroll) {
    float ms[kUnroll], ls[kUnroll];
    float4 a[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const bool ok = s0 + u < nsplit;
      const int64_t row = (r * nsplit + s0 + u) * H + h;
      ms[u] = ok ? part_m[row] : -INFINITY;
      ls[u] = ok ? part_l[row] : 0.f;
      a[u] = ok ? *reinterpret_cast<const float4*>(part_acc + row * kDV + c4 * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float m_new = m;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) m_new = fmaxf(m_new, ms[u]);
    if (m_new == -INFINITY) continue;
    if (s0 > 0) {
      const float keep = (m == -INFINITY) ? 0.f : exp2f(m - m_new);
      l *= keep;
      o.x *= keep;
      o.y *= keep;
      o.z *= keep;
      o.w *= keep;
    }
    m = m_new;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const float e = (ms[u] == -INFINITY) ? 0.f : exp2f(ms[u] - m);
      l = fmaf(ls[u], e, l);
      o.x = fmaf(a[u].x, e, o.x);
      o.y = fmaf(a[u].y, e, o.y);
      o.z = fmaf(a[u].z, e, o.z);
      o.w = fmaf(a[u].w, e, o.w);
    }
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  __nv_bfloat162 lo = __floats2bfloat162_rn(o.x * inv, o.y * inv);
  __nv_bfloat162 hi = __floats2bfloat162_rn(o.z * inv, o.w * inv);
  uint2 pk;
  pk.x = *reinterpret_cast<uint32_t*>(&lo);
  pk.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(out + pair * kDV + c4 * 4) = pk;
  DSA_KTIME_END(3);
}

// fp32 attention for any head / latent width: one CTA per (row, head), keys in
// chunks of 128 with an online softmax. indices == nullptr attends [0, len).
__global__ void __launch_bounds__(128)
sparse_mla_f32_kernel(const float* __restrict__ q, const float* __restrict__ kv,
                      const int32_t* __restrict__ indices, const int32_t* __restrict__ seq_lens,
                      float* __restrict__ out, int rows_per_seq, int H, int qk_dim, int v_dim,
                      int topk, float sm_scale, int64_t kv_seq_stride, int64_t ctx) {
  extern __shared__ float s_f[];  // q[qk_dim] | p[128] | idx[128] (as int) | red[8]
  float* s_qv = s_f;
  float* s_pv = s_f + qk_dim;
  int* s_idx = reinterpret_cast<int*>(s_pv + 128);
  float* s_r = reinterpret_cast<float*>(s_idx + 128);
  const int h = blockIdx.x, r = blockIdx.y, tid = threadIdx.x;
  const int seq = r / rows_per_seq;
  int64_t len = seq_lens ? int64_t(seq_lens[r]) : ctx;
  len = len < 0 ? 0 : (len > ctx ? ctx : len);
  const float* kvs = kv + int64_t(seq) * kv_seq_stride * qk_dim;
  for (int i = tid; i < qk_dim; i += 128) s_qv[i] = q[(int64_t(r) * H + h) * qk_dim + i];
  const int64_t n_keys = indices ? int64_t(topk) : len;
  float m_run = -INFINITY, l_run = 0.f;
  float o[4] = {0.f, 0.f, 0.f, 0.f};  // value columns tid, tid+128, ...
  __syncthreads();
  for (int64_t c0 = 0; c0 < n_keys; c0 += 128) {
    const int64_t j = c0 + tid;
    int64_t idx = -1;
    if (j < n_keys) idx = indices ? int64_t(indices[int64_t(r) * topk + j]) : j;
    const bool ok = idx >= 0 && idx < len;
    float s = -INFINITY;
    if (ok) {
      const float* kr = kvs + idx * qk_dim;
      float d = 0.f;
      for (int i = 0; i < qk_dim; ++i) d = fmaf(s_qv[i], kr[i], d);
      s = d * sm_scale;
    }
    // chunk max
    float mx = s;
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
    if ((tid & 31) == 0) s_r[tid >> 5] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(s_r[0], s_r[1]), fmaxf(s_r[2], s_r[3]));
    const float m_new = fmaxf(m_run, mx);
    const float pj = (ok && m_new != -INFINITY) ? expf(s - m_new) : 0.f;
    s_pv[tid] = pj;
    s_idx[tid] = ok ? int(idx) : -1;
    float ps = pj;
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, of);
    if ((tid & 31) == 0) s_r[4 + (tid >> 5)] = ps;
    __syncthreads();
    ps = s_r[4] + s_r[5] + s_r[6] + s_r[7];
    const float alpha = (m_new == -INFINITY) ? 1.f : expf(m_run - m_new);
    l_run = l_run * alpha + ps;
    m_run = m_new;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] *= alpha;
    for (int jj = 0; jj < 128; ++jj) {
      const int id = s_idx[jj];
      if (id < 0) continue;
      const float pw = s_pv[jj];
      const float* vr = kvs + int64_t(id) * qk_dim;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int col = tid + c * 128;
        if (col < v_dim) o[c] = fmaf(pw, vr[col], o[c]);
      }
    }
    __syncthreads();
  }
  const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int col = tid + c * 128;
    if (col < v_dim) out[(int64_t(r) * H + h) * v_dim + col] = o[c] * inv;
  }
}

// The same for many rows (full-sequence layers): one CTA per (row, block of eight heads). A tile of 16
// latent rows is gathered into shared memory once for the eight heads (padded rows: conflict-free
// 16-byte reads); a thread owns one (head, key) pair of the scores and every 128th value column of the
// result for all eight heads. The kernel above gathers every row once per head and waits for a chunk of
// 128 keys whatever the list's length: 66 us for 1024 rows x 8 heads x 16 keys x 80 against 12 us.
constexpr int kF32Heads = 8, kF32Keys = 16, kF32Threads = kF32Heads * kF32Keys;
__host__ __device__ inline int f32_rows_pitch(int qk_dim) { return (qk_dim + 7) / 8 * 8 + 4; }
inline size_t f32_rows_smem(int qk_dim) {
  return (size_t(kF32Heads + kF32Keys) * f32_rows_pitch(qk_dim) + kF32Heads * kF32Keys + 2 * kF32Heads) * 4;
}
__global__ void __launch_bounds__(kF32Threads)
sparse_mla_f32_rows_kernel(const float* __restrict__ q, const float* __restrict__ kv,
                           const int32_t* __restrict__ indices, const int32_t* __restrict__ seq_lens,
                           float* __restrict__ out, int rows_per_seq, int H, int qk_dim, int v_dim,
                           int topk, float sm_scale, int64_t kv_seq_stride, int64_t ctx) {
  extern __shared__ __align__(16) float s_fr[];
  const int pitch = f32_rows_pitch(qk_dim), dp = (qk_dim + 3) & ~3;
  float* s_q = s_fr;                               // [8][pitch]
  float* s_k = s_q + kF32Heads * pitch;            // [16][pitch]
  float* s_p = s_k + kF32Keys * pitch;             // [16 keys][8 heads]
  float* s_alpha = s_p + kF32Heads * kF32Keys;     // [8]
  float* s_inv = s_alpha + kF32Heads;              // [8]
  const int tid = threadIdx.x, key = tid & 15, head = tid >> 4;
  const int r = blockIdx.x, h0 = blockIdx.y * kF32Heads, heads = min(kF32Heads, H - h0);
  const int seq = r / rows_per_seq;
  int64_t len = seq_lens ? int64_t(seq_lens[r]) : ctx;
  len = len < 0 ? 0 : (len > ctx ? ctx : len);
  const float* kvs = kv + int64_t(seq) * kv_seq_stride * qk_dim;
  for (int i = tid; i < kF32Heads * dp; i += kF32Threads) {
    const int h = i / dp, d = i - h * dp;
    s_q[h * pitch + d] = (h < heads && d < qk_dim) ? q[(int64_t(r) * H + h0 + h) * qk_dim + d] : 0.f;
  }
  const int64_t n_keys = indices ? int64_t(topk) : len;
  float m_run = -INFINITY, l_run = 0.f;            // of this thread's head (equal in its 16 lanes)
  float o[kF32Heads][4] = {};                      // value columns tid, tid + 128, ... of every head
  for (int64_t c0 = 0; c0 < n_keys; c0 += kF32Keys) {
    // every thread looks at entry c0 + key, so that the 16 entries are known to each half-warp
    const int64_t j = c0 + key;
    int64_t idx = -1;
    if (j < n_keys) idx = indices ? int64_t(indices[int64_t(r) * topk + j]) : j;
    const bool ok = idx >= 0 && idx < len;
    const uint32_t any = __ballot_sync(0xffffffffu, ok);
    if ((any & 0xFFFFu) == 0u) continue;           // (the same 16 entries in both halves of every warp)
    __syncthreads();                               // the previous tile and its probabilities have been read
    for (int k = head; k < kF32Keys; k += kF32Heads) {  // 16 threads per latent row
      const int64_t at = __shfl_sync(0xffffffffu, ok ? idx : int64_t(-1), k);
      for (int d = key; d < dp; d += 16) s_k[k * pitch + d] = (at >= 0 && d < qk_dim) ? kvs[at * qk_dim + d] : 0.f;
    }
    __syncthreads();
    float s = 0.f;
    const float *qr = s_q + head * pitch, *kr = s_k + key * pitch;
#pragma unroll 4
    for (int d = 0; d < dp; d += 4) {
      const float4 a = *reinterpret_cast<const float4*>(qr + d), b = *reinterpret_cast<const float4*>(kr + d);
      s = fmaf(a.x, b.x, s);
      s = fmaf(a.y, b.y, s);
      s = fmaf(a.z, b.z, s);
      s = fmaf(a.w, b.w, s);
    }
    s = ok ? s * sm_scale : -INFINITY;
    float mx = s;
#pragma unroll
    for (int of = 8; of > 0; of >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, of));
    const float m_new = fmaxf(m_run, mx);
    const float pj = (ok && m_new != -INFINITY) ? expf(s - m_new) : 0.f;
    float ps = pj;
#pragma unroll
    for (int of = 8; of > 0; of >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, of);
    const float alpha = (m_new == -INFINITY) ? 1.f : expf(m_run - m_new);
    l_run = l_run * alpha + ps;
    m_run = m_new;
    s_p[key * kF32Heads + head] = pj;
    if (key == 0) s_alpha[head] = alpha;
    __syncthreads();
    float al[kF32Heads];
#pragma unroll
    for (int h = 0; h < kF32Heads; ++h) al[h] = s_alpha[h];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int col = tid + c * 128;
      if (col >= v_dim) break;
#pragma unroll
      for (int h = 0; h < kF32Heads; ++h) o[h][c] *= al[h];
#pragma unroll 4
      for (int k = 0; k < kF32Keys; ++k) {
        const float v = s_k[k * pitch + col];
        const float4 p0 = *reinterpret_cast<const float4*>(s_p + k * kF32Heads);
        const float4 p1 = *reinterpret_cast<const float4*>(s_p + k * kF32Heads + 4);
        o[0][c] = fmaf(p0.x, v, o[0][c]);
        o[1][c] = fmaf(p0.y, v, o[1][c]);
        o[2][c] = fmaf(p0.z, v, o[2][c]);
        o[3][c] = fmaf(p0.w, v, o[3][c]);
        o[4][c] = fmaf(p1.x, v, o[4][c]);
        o[5][c] = fmaf(p1.y, v, o[5][c]);
        o[6][c] = fmaf(p1.z, v, o[6][c]);
        o[7][c] = fmaf(p1.w, v, o[7][c]);
      }
    }
  }
  if (key == 0) s_inv[head] = l_run > 0.f ? 1.f / l_run : 0.f;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int col = tid + c * 128;
    if (col >= v_dim) break;
#pragma unroll
    for (int h = 0; h < kF32Heads; ++h)
      if (h < heads) out[(int64_t(r) * H + h0 + h) * v_dim + col] = o[h][c] * s_inv[h];
  }
}

}  // namespace mla
}  // namespace dsa
