// Backward preprocess for rows that vectors can read: delta = rowsum(dO * O) and, optionally, the bf16 copy of dO.  A launch of its own
// (bma_api.cu), or the CTAs behind the slot tables of the backward scratch (bwd_slots.cu).
#pragma once

#include <algorithm>

#include "common.cuh"

namespace bma {

inline bool rows_of_16_bytes(const bma_tensor& t) {
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.stride_b % 4 == 0 && t.stride_l % 4 == 0 && t.stride_h % 4 == 0;
}
inline bool preprocess_vectors(const bma_attn_args& a, const void* out) {
  return a.d % 4 == 0 && rows_of_16_bytes(a.o) && rows_of_16_bytes(a.d_o) && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
}
inline int preprocess_rows4_ctas(const bma_attn_args& a) {
  const int64_t units = (int64_t)a.B * a.Hq * ((a.N + 3) / 4);
  return (int)std::min<int64_t>((units + 7) / 8, kSms * 32);
}

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u);
  v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
}

// Streaming form for d <= 128 with vector accesses: one warp takes FOUR consecutive queries of one
// (batch, head), issues all eight 16-byte loads per lane before it uses any of them, and writes the four
// delta values as one 16-byte line, so that the [B, Hq, N] delta array is written in whole sectors
// (one warp per row wrote 4 bytes per 32-byte sector).  Bound by HBM: reads |O| + |dO|, writes the bf16
// copy of dO and delta.
template <typename TO, typename TDO>
__device__ __forceinline__ void preprocess_rows4(const bma_attn_args& a, __nv_bfloat16* __restrict__ do_bf16, int cta, int ctas) {
  const int lane = threadIdx.x & 31;
  const int warps = (blockDim.x >> 5);
  const int64_t nq4 = (a.N + 3) / 4;
  const int64_t units = (int64_t)a.B * a.Hq * nq4;
  const int c = lane * 4;
  const bool act = c < a.d;
  for (int64_t u = (int64_t)cta * warps + (threadIdx.x >> 5); u < units; u += (int64_t)ctas * warps) {
    const int q0 = (int)(u % nq4) * 4;
    const int h = (int)((u / nq4) % a.Hq);
    const int b = (int)(u / (nq4 * a.Hq));
    float gv[4][4], ov[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = q0 + i;
      if (act && q < a.N) {
        load4(static_cast<const TDO*>(a.d_o.ptr) + (int64_t)b * a.d_o.stride_b + (int64_t)q * a.d_o.stride_l + (int64_t)h * a.d_o.stride_h + c, gv[i]);
        load4(static_cast<const TO*>(a.o.ptr) + (int64_t)b * a.o.stride_b + (int64_t)q * a.o.stride_l + (int64_t)h * a.o.stride_h + c, ov[i]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) { gv[i][e] = 0.f; ov[i][e] = 0.f; }
      }
    }
    // With a bf16 copy, delta is taken from the ROUNDED cotangent -- the values the dP = dO V^T product of the backward
    // kernels sees -- so that dP - delta cancels where it should (a row that attends one key has dS = 0 exactly; with
    // the float32 cotangent in delta and the bf16 one in dP the difference of the two roundings would survive).
    float acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = q0 + i;
      if (do_bf16) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(gv[i][0], gv[i][1]), hi = __floats2bfloat162_rn(gv[i][2], gv[i][3]);
        uint2 w;
        w.x = *reinterpret_cast<uint32_t*>(&lo);
        w.y = *reinterpret_cast<uint32_t*>(&hi);
        gv[i][0] = __uint_as_float(w.x << 16); gv[i][1] = __uint_as_float(w.x & 0xffff0000u);
        gv[i][2] = __uint_as_float(w.y << 16); gv[i][3] = __uint_as_float(w.y & 0xffff0000u);
        if (act && q < a.N) *reinterpret_cast<uint2*>(do_bf16 + (((int64_t)b * a.N + q) * a.Hq + h) * a.d + c) = w;
      }
      acc[i] = fmaf(gv[i][0], ov[i][0], fmaf(gv[i][1], ov[i][1], fmaf(gv[i][2], ov[i][2], gv[i][3] * ov[i][3])));
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
    }
    float* dst = a.delta + ((int64_t)b * a.Hq + h) * a.N + q0;
    if (lane == 0) {
      if (q0 + 3 < a.N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (q0 + i < a.N) dst[i] = acc[i];
      }
    }
  }
}

}  // namespace bma
