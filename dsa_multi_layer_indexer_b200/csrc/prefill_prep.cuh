// Full-sequence counterpart of decode_prep.cuh: what lies between the projection GEMMs of a prompt
// and the scan / attention kernels, in two launches.
//
//   prefill_latents_kernel   behind the GEMM that reads x_norm: RMSNorm of the query latent, RMSNorm +
//                            RoPE of the latent cache row, RoPE (+ e4m3 quantisation) of the index key;
//                            the last two go straight to their rows of the caches;
//   prefill_queries_kernel   behind the GEMM that reads c_q: RoPE of the MLA query heads into the rope
//                            part of the absorbed query (the GEMM with W_UK writes the other 512
//                            columns itself), RoPE (+ e4m3 quantisation, scale folded into the head
//                            weight) of the indexer heads.
//
// (src/lagged_indexer_dsa/dsa_layer.py:87-143, rope.py:52-84.) Every product and sum is rounded to the
// element type on its own, as the elementwise operations of the reference are, so the results are those
// of the unfused chain bit for bit (the two norms aside: another summation order).
//
// Bound: HBM. At 4099 tokens x 128 + 64 heads the pair moves about 350 MB (54 us at the copy peak); the
// chain of torch launches it replaces (two multiplications, negation, concatenations, addition, copies,
// conversions per operand, and torch.cat of the 604 MB query) took 7.0 ms per layer there.
#pragma once

#include "decode_prep.cuh"

namespace dsa {
namespace prep {

struct LatentsParams {
  const void* qa;            // [rows] x q_rank, row stride qa_stride (nullptr: skipped)
  const void* kv_a;          // [rows] x (kv_rank + rope_dim) (nullptr: skipped)
  const void* ik;            // [rows] x idx_dim (nullptr: skipped)
  const void* q_norm_w;
  const void* kv_norm_w;
  const void* mla_cos;       // [seq, rope_dim]
  const void* mla_sin;
  const void* idx_cos;       // [seq, idx_dim]
  const void* idx_sin;
  void* c_q;                 // [rows, q_rank]
  void* kv_out;              // row (b, s) at b * kv_cap + s, kv_rank + rope_dim wide
  void* ik_out;              // e4m3 rows (ik_scale given) or rows of T, at b * ik_cap + s
  float* ik_scale;
  int64_t qa_stride, kv_a_stride, ik_stride, kv_cap, ik_cap, rows;
  int seq, q_rank, kv_rank, rope_dim, idx_dim, interleave;
  float eps;
};

struct QueriesParams {
  const void* q;             // element (row, head, i) at row * q_stride + head * q_head_stride + i; rope part from `nope`
  const void* iq;            // [rows] x Hidx * idx_dim, row stride iq_stride (nullptr: skipped)
  const void* w;             // [rows] x Hidx, row stride w_stride
  const void* mla_cos;
  const void* mla_sin;
  const void* idx_cos;
  const void* idx_sin;
  void* q_full;              // [rows, H, kv_rank + rope_dim]: the rope part is written here (nullptr: skipped)
  void* index_q;             // e4m3 (index_w given) or T, [rows, Hidx, idx_dim]
  float* index_w;            // [rows, Hidx]
  int64_t q_stride, q_head_stride, iq_stride, w_stride, rows;
  int seq, H, Hidx, nope, kv_rank, rope_dim, idx_dim, interleave;
};

template <typename T>
__device__ __forceinline__ float rounded(float v) { return to_f32<T>(from_f32<T>(v)); }

// x * cos + partner * sin with the roundings of three separate operations.
template <typename T>
__device__ __forceinline__ float rope_one(float x, float partner, float c, float s) {
  return rounded<T>(__fadd_rn(rounded<T>(__fmul_rn(x, c)), rounded<T>(__fmul_rn(partner, s))));
}

// The rotated element i of a d-wide vector in global memory (any even d).
template <typename T>
__device__ __forceinline__ float rope_at(const T* src, const T* cosr, const T* sinr, int i, int d, bool interleave) {
  const int half = d >> 1;
  float partner;
  if (interleave) partner = (i & 1) ? to_f32<T>(src[i - 1]) : -to_f32<T>(src[i + 1]);
  else partner = i < half ? -to_f32<T>(src[i + half]) : to_f32<T>(src[i - half]);
  return rope_one<T>(to_f32<T>(src[i]), partner, to_f32<T>(cosr[i]), to_f32<T>(sinr[i]));
}

// Four consecutive bf16 values as floats (8-byte aligned source).
__device__ __forceinline__ void load4(const __nv_bfloat16* src, float (&v)[4]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(src);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  v[0] = lo.x, v[1] = lo.y, v[2] = hi.x, v[3] = hi.y;
}

// RoPE of dims [4 lane, 4 lane + 4) of a 128-wide bf16 vector held four per lane.
__device__ __forceinline__ void rope128_bf16(float (&v)[4], const float (&c)[4], const float (&s)[4], int lane,
                                             bool interleave) {
  float p[4];
  if (interleave) {
    p[0] = -v[1], p[1] = v[0], p[2] = -v[3], p[3] = v[2];
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, v[j], 16);
      p[j] = lane < 16 ? -other : other;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = rope_one<__nv_bfloat16>(v[j], p[j], c[j], s[j]);
}

// One warp: y = x * rsqrt(mean(x^2) + eps) * w over n elements, fp32 math, one rounding.
template <typename T>
__device__ __forceinline__ void warp_rmsnorm(const T* x, const T* w, T* y, int n, float eps, int lane) {
  constexpr int kVec = 16 / int(sizeof(T));
  float ss = 0.f;
  const bool vec = n % kVec == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) |
                                      reinterpret_cast<uintptr_t>(y)) & 15u) == 0;
  if (vec) {
#pragma unroll 2
    for (int i = lane * kVec; i < n; i += 32 * kVec) {
      const uint4 raw = *reinterpret_cast<const uint4*>(x + i);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int j = 0; j < kVec; ++j) ss = fmaf(to_f32<T>(e[j]), to_f32<T>(e[j]), ss);
    }
  } else {
    for (int i = lane; i < n; i += 32) ss = fmaf(to_f32<T>(x[i]), to_f32<T>(x[i]), ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float inv = rsqrtf(ss / float(n) + eps);
  if (vec) {
#pragma unroll 2
    for (int i = lane * kVec; i < n; i += 32 * kVec) {  // (the second read hits L1)
      const uint4 raw = *reinterpret_cast<const uint4*>(x + i), wraw = *reinterpret_cast<const uint4*>(w + i);
      const T* e = reinterpret_cast<const T*>(&raw);
      const T* we = reinterpret_cast<const T*>(&wraw);
      uint4 o;
      T* oe = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int j = 0; j < kVec; ++j) oe[j] = from_f32<T>(to_f32<T>(e[j]) * inv * to_f32<T>(we[j]));
      *reinterpret_cast<uint4*>(y + i) = o;
    }
  } else {
    for (int i = lane; i < n; i += 32) y[i] = from_f32<T>(to_f32<T>(x[i]) * inv * to_f32<T>(w[i]));
  }
}

// One warp per (row, item): item 0 the query latent, 1 the latent cache row, 2 the index key.
constexpr int kLatentWarps = 6;
template <typename T>
__global__ void __launch_bounds__(kLatentWarps * 32)
prefill_latents_kernel(const LatentsParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t unit = int64_t(blockIdx.x) * kLatentWarps + (threadIdx.x >> 5);
  const int64_t row = unit / 3;
  const int item = int(unit - row * 3);
  if (row >= p.rows) return;
  const int64_t b = row / p.seq;
  const int s = int(row - b * p.seq);
  if (item == 0) {
    if (p.qa)
      warp_rmsnorm<T>(static_cast<const T*>(p.qa) + row * p.qa_stride, static_cast<const T*>(p.q_norm_w),
                      static_cast<T*>(p.c_q) + row * p.q_rank, p.q_rank, p.eps, lane);
  } else if (item == 1) {
    if (!p.kv_a) return;
    const T* src = static_cast<const T*>(p.kv_a) + row * p.kv_a_stride;
    T* dst = static_cast<T*>(p.kv_out) + (b * p.kv_cap + s) * (p.kv_rank + p.rope_dim);
    warp_rmsnorm<T>(src, static_cast<const T*>(p.kv_norm_w), dst, p.kv_rank, p.eps, lane);
    const T* cr = static_cast<const T*>(p.mla_cos) + int64_t(s) * p.rope_dim;
    const T* sr = static_cast<const T*>(p.mla_sin) + int64_t(s) * p.rope_dim;
    for (int i = lane; i < p.rope_dim; i += 32)
      dst[p.kv_rank + i] = from_f32<T>(rope_at<T>(src + p.kv_rank, cr, sr, i, p.rope_dim, false));
  } else {
    if (!p.ik) return;
    const T* src = static_cast<const T*>(p.ik) + row * p.ik_stride;
    const T* cr = static_cast<const T*>(p.idx_cos) + int64_t(s) * p.idx_dim;
    const T* sr = static_cast<const T*>(p.idx_sin) + int64_t(s) * p.idx_dim;
    const int64_t at = b * p.ik_cap + s;
    if (p.ik_scale) {  // 128 wide (checked by the host)
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = rope_at<T>(src, cr, sr, 4 * lane + j, 128, p.interleave != 0);
      float scale;
      const uint32_t packed = quant128(v, scale);
      reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.ik_out) + at * 128)[lane] = packed;
      if (lane == 0) p.ik_scale[at] = scale;
    } else {
      T* dst = static_cast<T*>(p.ik_out) + at * p.idx_dim;
      for (int i = lane; i < p.idx_dim; i += 32) dst[i] = from_f32<T>(rope_at<T>(src, cr, sr, i, p.idx_dim, p.interleave != 0));
    }
  }
}

// bf16, production widths: one CTA per token; a warp keeps its lanes' table entries in registers and
// walks every eighth head, two heads in flight.
constexpr int kQueryWarps = 8;
__global__ void __launch_bounds__(kQueryWarps * 32)
prefill_queries_bf16_kernel(const QueriesParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = blockIdx.x;
  const int s = int(row % p.seq);
  if (p.iq) {
    float c[4], sn[4];
    load4(static_cast<const __nv_bfloat16*>(p.idx_cos) + int64_t(s) * 128 + 4 * lane, c);
    load4(static_cast<const __nv_bfloat16*>(p.idx_sin) + int64_t(s) * 128 + 4 * lane, sn);
    const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(p.iq) + row * p.iq_stride + 4 * lane;
    const __nv_bfloat16* wr = static_cast<const __nv_bfloat16*>(p.w) + row * p.w_stride;
    uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.index_q) + row * p.Hidx * 128) + lane;
#pragma unroll 2
    for (int h = warp; h < p.Hidx; h += kQueryWarps) {
      float v[4];
      load4(src + h * 128, v);
      rope128_bf16(v, c, sn, lane, p.interleave != 0);
      float scale;
      const uint32_t packed = quant128(v, scale);
      dst[h * 32] = packed;
      if (lane == 0) p.index_w[row * p.Hidx + h] = scale * __bfloat162float(wr[h]);
    }
  }
  if (p.q_full) {
    // 64 rope dims: 16 lanes per head (four dims each, partner in lane ^ 8), two heads per warp step
    const int sub = lane & 15;
    float c[4], sn[4];
    load4(static_cast<const __nv_bfloat16*>(p.mla_cos) + int64_t(s) * 64 + 4 * sub, c);
    load4(static_cast<const __nv_bfloat16*>(p.mla_sin) + int64_t(s) * 64 + 4 * sub, sn);
    const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(p.q) + row * p.q_stride + p.nope + 4 * sub;
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.q_full) + row * p.H * DSA_LATENT_DIM + DSA_VALUE_DIM + 4 * sub;
#pragma unroll 2
    for (int h0 = 2 * warp; h0 < p.H; h0 += 2 * kQueryWarps) {
      const int h = h0 + (lane >> 4);
      const bool in = h < p.H;
      float v[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
      if (in) load4(src + int64_t(h) * p.q_head_stride, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, v[j], 8);
        o[j] = rope_one<__nv_bfloat16>(v[j], sub < 8 ? -other : other, c[j], sn[j]);
      }
      if (in) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), d = __floats2bfloat162_rn(o[2], o[3]);
        uint2 pk;
        pk.x = *reinterpret_cast<const uint32_t*>(&a);
        pk.y = *reinterpret_cast<const uint32_t*>(&d);
        *reinterpret_cast<uint2*>(dst + int64_t(h) * DSA_LATENT_DIM) = pk;
      }
    }
  }
}

// fp32 rows of any width: one thread per element.
__global__ void __launch_bounds__(256)
prefill_queries_f32_kernel(const QueriesParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t row = blockIdx.x;
  const int s = int(row % p.seq);
  if (p.iq) {
    const float* src = static_cast<const float*>(p.iq) + row * p.iq_stride;
    float* dst = static_cast<float*>(p.index_q) + row * p.Hidx * p.idx_dim;
    const float* cr = static_cast<const float*>(p.idx_cos) + int64_t(s) * p.idx_dim;
    const float* sr = static_cast<const float*>(p.idx_sin) + int64_t(s) * p.idx_dim;
    for (int t = threadIdx.x; t < p.Hidx * p.idx_dim; t += 256) {
      const int h = t / p.idx_dim, i = t - h * p.idx_dim;
      dst[t] = rope_at<float>(src + h * p.idx_dim, cr, sr, i, p.idx_dim, p.interleave != 0);
    }
  }
  if (p.q_full) {
    const float* src = static_cast<const float*>(p.q) + row * p.q_stride + p.nope;
    const int width = p.kv_rank + p.rope_dim;
    float* dst = static_cast<float*>(p.q_full) + row * p.H * width + p.kv_rank;
    const float* cr = static_cast<const float*>(p.mla_cos) + int64_t(s) * p.rope_dim;
    const float* sr = static_cast<const float*>(p.mla_sin) + int64_t(s) * p.rope_dim;
    for (int t = threadIdx.x; t < p.H * p.rope_dim; t += 256) {
      const int h = t / p.rope_dim, i = t - h * p.rope_dim;
      dst[int64_t(h) * width + i] = rope_at<float>(src + int64_t(h) * p.q_head_stride, cr, sr, i, p.rope_dim, false);
    }
  }
}

}  // namespace prep
}  // namespace dsa
