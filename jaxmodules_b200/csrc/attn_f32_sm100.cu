// float32 attention (forward, dK/dV, dQ) on the sm_100a tensor core.
//
// A float32 value between 2^-110 and 3.38e38 in magnitude is the exact sum of three bfloat16 values (8 + 8 + 8 significand bits),
// and a product of two bfloat16 values is exact in the float32 accumulator.  Every operand is therefore carried as three bf16 planes hi + mid + lo, and
// every matrix product is the sum of the six plane products whose weight reaches 2^-24 of the result:
//     x y  ~  lo hi + hi lo + mid mid + mid hi + hi mid + hi hi        (dropped: mid lo, lo mid, lo lo <= 2^-24 |x y|)
// issued smallest terms first.  Six passes at the bf16 rate leave 270 TFLOP/s of the measured tensor peak, against
// 72 TFLOP/s of the FP32 FMA pipes (and the 14 - 19 the FP32 tile kernels of attn_simt.cu reach).
//
// Accuracy is held to that of an FP32 FMA chain: the tensor core truncates when it adds to its accumulator, so accumulations
// are short there -- the plane products of one 64-wide tile (of the padded head dimension, 64 or 128, for S and dP) -- and O,
// dQ, dK and dV are summed over the tiles in registers, with rounded FP32 adds.  Against float64 the 2-norm error is 1.4e-7 - 3.5e-7 (causal, B=2 L=2048 H=16 d=64; the FP32 tile
// kernels: 4.1e-7 - 8.5e-7).
//
// Measured there: forward 110 us (tile kernels 861), dK/dV 171 (1383), dQ 133 (1357), the two splits 21 each; forward with
// d=128, N=L=1500, 16 heads: 134 us (1139).
//
// One split kernel writes the planes of Q, K, V (and dO) into the caller's workspace as [3, B, L, H, DP] bf16, DP = 64 or
// 128 columns (zero padded), from where TMA fetches them; splitting inside the attention kernels would repeat the
// conversion for every tile that reads the operand.
//
// Where a product has only 64 columns of output per operand (64 keys, 64 queries, 64 head columns) the hi and mid planes
// of its B operand are stacked to N = 128: a 128x64x16 MMA takes 53 cycles, a 128x128x16 one 64.  The two accumulator
// halves are added when they are read.
//
// Order: such a sum is a chain of 64- and 128-column MMAs into the same columns, issued by one thread with nothing between
// them, and the first of a region overwrites it.  PTX promises the order of tcgen05.mma pairs of one accumulator and one
// shape; that pairs of different shapes run in the order of issue too is how the tensor core of an SM works through the
// MMAs of a CTA, not a written rule.  A swap would lose whole products (2^-8 of the result or more, and not the same twice):
// every float32 test would see it, and tests/test_gpu_kernel_variants.py repeats calls for it.  One shape throughout would cost
// 256 cycles per 16-deep step with 128 columns (and a zero plane behind every lo plane, a third more shared memory for the
// operand), 318 with 64, instead of 234.
//
// Tensor memory columns hold the accumulators of a tile and then, over the columns that the reading thread has just
// consumed, the three planes of P or dS as A operands (per 16 keys: 8 columns hi, 8 mid, and 8 lo in the other half).
// Every mbarrier wait is bounded; on a timeout the thread records an error code and unwinds.

#include "common.cuh"
#include "ptx_sm100.cuh"
#include "simt_tiles.cuh"

namespace bma {
namespace {

using namespace ptx;

constexpr int BM = 128;                          // rows of a tile (queries forward / dQ, keys dK/dV)
constexpr int BH = 64;                           // columns of a half tile (keys forward / dQ, queries dK/dV)
constexpr int kThreads = 384;                    // two warpgroups of row threads, one of single-warp roles
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kRowBox = BM * 128;           // one [128 x 64] bf16 box
constexpr uint32_t kHalfBox = BH * 128;          // one [64 x 64] bf16 box
constexpr int kMaxKvFwd = 4096, kMaxKvBwd = 1024;

__device__ __forceinline__ void setmaxnreg_inc_208() { asm volatile("setmaxnreg.inc.sync.aligned.u32 208;"); }
__device__ __forceinline__ void setmaxnreg_dec_80() { asm volatile("setmaxnreg.dec.sync.aligned.u32 80;"); }

// x = hi + mid + lo, exactly, for two neighbouring values (packed like an MMA operand).  The row threads work on pairs throughout: the
// packed FP32 instructions round like the scalar ones and take one issue slot for two.
__device__ __forceinline__ float2 minus_hi(float2 x, uint32_t hi) {
  return __ffma2_rn(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), make_float2(-1.f, -1.f), x);
}
__device__ __forceinline__ void split3(float2 x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x.x, x.y);
  x = minus_hi(x, hi);
  mid = pack_bf16(x.x, x.y);
  x = minus_hi(x, mid);
  lo = pack_bf16(x.x, x.y);
}
// Sum of the two halves of an accumulator region, columns 2j and 2j + 1.
__device__ __forceinline__ float2 halves(const uint32_t* r0, const uint32_t* r1, int j) {
  return __fadd2_rn(make_float2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1])),
                    make_float2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1])));
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// Plane p of the A operand of k-step ks (16 keys or queries) inside a 128-column accumulator region.
__device__ __forceinline__ uint32_t plane_col(int p, int ks) { return p == 2 ? 64 + 16 * ks : 16 * ks + 8 * p; }

// Stores the planes of 32 consecutive values (k-steps ks0, ks0 + 1) over the columns they came from.
__device__ __forceinline__ void store_planes32(uint32_t region, int ks0, const float2* v) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    uint32_t hm[16], lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) split3(v[u * 8 + j], hm[j], hm[8 + j], lo[j]);
    tmem_st16(region + 16 * (ks0 + u), hm);
    tmem_st8(region + 64 + 16 * (ks0 + u), lo);
  }
}

// ---- plane products ---------------------------------------------------------------------------------------------
// region[0, 64) and region[64, 128) <- A B^T with B of 64 rows, K-major: A planes at a[0..2], B planes stacked in shared
// memory (hi, mid, lo of 64 rows each, kHalfBox apart), one 64-column box of both per `boxes` step.
constexpr uint32_t kIdescN64 = make_idesc_bf16(BM, 64, 0, 0), kIdescN128 = make_idesc_bf16(BM, 128, 0, 0);
constexpr uint32_t kIdescN64T = make_idesc_bf16(BM, 64, 0, 1), kIdescN128T = make_idesc_bf16(BM, 128, 0, 1);

template <int BOXES>
__device__ __forceinline__ void product_rows(bool leader, uint32_t region, uint64_t a_hi, uint64_t b_hi) {
  constexpr uint32_t kAPlane = (BOXES * kRowBox) >> 4, kBPlane = kHalfBox >> 4;
  auto a_off = [](int ks) { return (uint32_t)(((ks >> 2) * kRowBox + (ks & 3) * 32) >> 4); };
  auto b_off = [](int ks) { return (uint32_t)(((ks >> 2) * 3 * kHalfBox + (ks & 3) * 32) >> 4); };
  if (!leader) return;
#pragma unroll
  for (int ks = 0; ks < BOXES * 4; ++ks) mma_ss(region, a_hi + 2 * kAPlane + a_off(ks), b_hi + b_off(ks), kIdescN64, ks > 0);
#pragma unroll
  for (int ks = 0; ks < BOXES * 4; ++ks) mma_ss(region + 64, a_hi + a_off(ks), b_hi + 2 * kBPlane + b_off(ks), kIdescN64, ks > 0);
#pragma unroll
  for (int ks = 0; ks < BOXES * 4; ++ks) mma_ss(region, a_hi + kAPlane + a_off(ks), b_hi + b_off(ks), kIdescN128, 1);
#pragma unroll
  for (int ks = 0; ks < BOXES * 4; ++ks) mma_ss(region, a_hi + a_off(ks), b_hi + b_off(ks), kIdescN128, 1);
}

// region <- P B with the planes of P [128 x 64] in tensor memory at `p` and B [64 x DP] read MN-major (planes DP/64 boxes
// of [64 x 64] each).  DP 64: the hi and mid planes of B side by side, two halves to be added; DP 128: one sum.
template <int BOXES>
__device__ __forceinline__ void product_cols(bool leader, uint32_t region, uint32_t p, uint64_t b_hi) {
  constexpr uint32_t kBPlane = (BOXES * kHalfBox) >> 4;
  if (!leader) return;
  auto b_off = [](int ks) { return (uint32_t)(ks * (2048 >> 4)); };
  if constexpr (BOXES == 1) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(region, p + plane_col(2, ks), b_hi + b_off(ks), kIdescN64T, ks > 0);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(region + 64, p + plane_col(0, ks), b_hi + 2 * kBPlane + b_off(ks), kIdescN64T, ks > 0);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(region, p + plane_col(1, ks), b_hi + b_off(ks), kIdescN128T, 1);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(region, p + plane_col(0, ks), b_hi + b_off(ks), kIdescN128T, 1);
  } else {
    constexpr int kTerms[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};   // (plane of P, plane of B)
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        mma_ts(region, p + plane_col(kTerms[t][0], ks), b_hi + kTerms[t][1] * kBPlane + b_off(ks), kIdescN128T, (t > 0) || (ks > 0));
  }
}

// ---- splitting ----------------------------------------------------------------------------------------------------
struct SplitJob {
  bma_tensor t;
  uint8_t* out;      // [3, B, L, H, DP] bf16
  int L, H;
};
struct SplitParams {
  SplitJob job[4];
  int B, d;
  bma_tensor o;          // backward: with `delta`, delta = rowsum(dO * O) on the way through dO (job 3)
  float* delta;          // null: the caller's
  int jobs;              // blockIdx.y == jobs: the block lists of a mask of interval terms, both sides, where the caller has none
  bma_block_lists lists;
  bma_mask_spec spec;
  const uint8_t* used;   // null, or one byte per kv block [used_B, NKV] (jobs 1 and 2, K and V): 0 = no list names it
  int used_B, NKV;
};

// used[b', kj] = 1 where a list of batch entry b' names kv block kj (a kv-side list; backward: or a q-side list of kj has an
// entry), else 0.  One CTA per batch entry of the lists.
__global__ void __launch_bounds__(256) used_blocks_kernel(bma_block_lists l, bma_mask_spec spec, bool backward, uint8_t* __restrict__ used) {
  __shared__ uint8_t mark[kMaxKvFwd];
  for (int i = threadIdx.x; i < l.NKV; i += 256) mark[i] = 0;
  __syncthreads();
  const int rows = l.H * l.NQ, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (!l.kv_num)
    for (int i = threadIdx.x; i < l.NKV; i += 256)
      for (int qi = 0; qi < l.NQ; ++qi) mark[i] |= interval_class(spec, qi, i, BM, BM) != 0;
  for (int r = warp; r < rows && l.kv_num; r += 8) {
    const int64_t row = (int64_t)blockIdx.x * rows + r;
    const int nfull = l.full_kv_num[row], npart = l.kv_num[row];
    for (int i = lane; i < nfull; i += 32) mark[l.full_kv_idx[row * l.NKV + i]] = 1;
    for (int i = lane; i < npart; i += 32) mark[l.kv_idx[row * l.NKV + i]] = 1;
  }
  if (backward && l.q_num)
    for (int i = threadIdx.x; i < l.H * l.NKV; i += 256)
      if (l.q_num[(int64_t)blockIdx.x * l.H * l.NKV + i] + l.full_q_num[(int64_t)blockIdx.x * l.H * l.NKV + i] > 0) mark[i % l.NKV] = 1;
  __syncthreads();
  for (int i = threadIdx.x; i < l.NKV; i += 256) used[(int64_t)blockIdx.x * l.NKV + i] = mark[i];
}

// Block lists of a mask of interval terms: a warp per row of either side.
__device__ __forceinline__ void write_lists(const bma_block_lists& l, const bma_mask_spec& spec) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1;
  for (int r = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5); r < l.NQ + l.NKV; r += (int)gridDim.x * 8) {
    const bool q_side = r >= l.NQ;
    const int row = q_side ? r - l.NQ : r, width = q_side ? l.NQ : l.NKV;
    int32_t* full = (q_side ? l.full_q_idx : l.full_kv_idx) + (int64_t)row * width;
    int32_t* part = (q_side ? l.q_idx : l.kv_idx) + (int64_t)row * width;
    int nfull = 0, npart = 0;
    for (int base = 0; base < width; base += 32) {
      const int j = base + lane;
      const int c = j >= width ? 0 : q_side ? interval_class(spec, j, row, BM, BM) : interval_class(spec, row, j, BM, BM);
      const unsigned mf = __ballot_sync(0xffffffffu, c == 2), mp = __ballot_sync(0xffffffffu, c == 1);
      if (c == 2) full[nfull + __popc(mf & below)] = j;
      if (c == 1) part[npart + __popc(mp & below)] = j;
      nfull += __popc(mf);
      npart += __popc(mp);
    }
    if (lane == 0) {
      (q_side ? l.full_q_num : l.full_kv_num)[row] = nfull;
      (q_side ? l.q_num : l.kv_num)[row] = npart;
    }
  }
}

// One thread per 8 columns: 32 bytes in, three 16-byte lines out.  Backward the same launch takes delta = rowsum(dO * O) and writes the
// block lists that the caller left to it: launches of their own, 2.6 and 3 us of the device and 8 - 10 of the host each (2 x 128 tokens, 8 heads,
// forward and backward: the call 154 -> 143 us; 2 x 2048, 16 heads, where O and dO were read in a pass of their own: 533 -> 526).  Bound by HBM (4 bytes read, 6 written per element), or
// by launch latency where the tensors are small.
template <int DP>
__global__ void __launch_bounds__(256) split_kernel(const SplitParams p) {
  if ((int)blockIdx.y == p.jobs) {
    write_lists(p.lists, p.spec);
    return;
  }
  const SplitJob& job = p.job[blockIdx.y];
  constexpr int kChunks = DP / 8;
  const bool take_delta = blockIdx.y == 3 && p.delta != nullptr, o_f32 = p.o.dtype == BMA_DTYPE_F32;
  const int64_t n = (int64_t)p.B * job.L * job.H * kChunks;
  const bool f32 = job.t.dtype == BMA_DTYPE_F32;
  const bool vec = f32 && (reinterpret_cast<uintptr_t>(job.t.ptr) & 15) == 0 && ((job.t.stride_b | job.t.stride_l | job.t.stride_h) & 3) == 0;
  uint4* out = reinterpret_cast<uint4*>(job.out);
  auto split8 = [&](int64_t i) {
    const int c = (int)(i % kChunks) * 8;
    const int64_t row = i / kChunks;
    const int h = (int)(row % job.H);
    const int l = (int)((row / job.H) % job.L);
    const int b = (int)(row / ((int64_t)job.H * job.L));
    const int64_t off = (int64_t)b * job.t.stride_b + (int64_t)l * job.t.stride_l + (int64_t)h * job.t.stride_h + c;
    float v[8];
    if (vec && c + 8 <= p.d) {
      const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(job.t.ptr) + off);
      const float4 x = src[0], y = src[1];
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[e] = 0.f;
        if (c + e < p.d)
          v[e] = f32 ? static_cast<const float*>(job.t.ptr)[off + e] : to_float(static_cast<const __nv_bfloat16*>(job.t.ptr)[off + e]);
      }
    }
    uint32_t w[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split3(make_float2(v[2 * e], v[2 * e + 1]), w[0][e], w[1][e], w[2][e]);
#pragma unroll
    for (int q = 0; q < 3; ++q) out[q * n + i] = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
    if (take_delta) {
      // Sums in the order of bwd_preprocess_rows4_kernel (four columns, then a tree over the columns' highest bits first), bit for bit: next to a
      // huge key, dS is the rounding of delta alone, and what a tile that is done again makes of it is that of the FP32 tile kernels.
      const int64_t at = (int64_t)b * p.o.stride_b + (int64_t)l * p.o.stride_l + (int64_t)h * p.o.stride_h + c;
      float s[2] = {0.f, 0.f};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (c + 4 * u >= p.d) continue;
        float o4[4];
        if (o_f32) {
          const float4 x = *reinterpret_cast<const float4*>(static_cast<const float*>(p.o.ptr) + at + 4 * u);
          o4[0] = x.x; o4[1] = x.y; o4[2] = x.z; o4[3] = x.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) o4[e] = to_float(static_cast<const __nv_bfloat16*>(p.o.ptr)[at + 4 * u + e]);
        }
        s[u] = fmaf(v[4 * u], o4[0], fmaf(v[4 * u + 1], o4[1], fmaf(v[4 * u + 2], o4[2], v[4 * u + 3] * o4[3])));
      }
      const int lane = threadIdx.x & 31;   // (the kChunks lanes of a row are all here or all past the end)
      const unsigned group = ((1u << kChunks) - 1) << (lane & ~(kChunks - 1));
#pragma unroll
      for (int off = kChunks / 2; off; off /= 2) {
        s[0] += __shfl_xor_sync(group, s[0], off);
        s[1] += __shfl_xor_sync(group, s[1], off);
      }
      if ((lane & (kChunks - 1)) == 0) p.delta[((int64_t)b * job.H + h) * job.L + l] = s[0] + s[1];
    }
  };
  if (!p.used || blockIdx.y == 0 || blockIdx.y == 3) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) split8(i);
    return;
  }
  // K and V: a kv block at a time, in pieces of 1024 lines so that a few blocks fill the chip as well
  constexpr int kPiece = 1024;
  const int parts = (BM * job.H * kChunks + kPiece - 1) / kPiece;
  for (int64_t w = blockIdx.x; w < (int64_t)p.B * p.NKV * parts; w += gridDim.x) {
    const int64_t blk = w / parts;
    const int b = (int)(blk / p.NKV), l0 = (int)(blk % p.NKV) * BM, at = (int)(w % parts) * kPiece;
    if (!__ldg(p.used + (int64_t)(p.used_B == 1 ? 0 : b) * p.NKV + l0 / BM)) continue;
    const int64_t first = ((int64_t)b * job.L + l0) * job.H * kChunks;
    const int end = min(at + kPiece, min(BM, job.L - l0) * job.H * kChunks);
    for (int i = at + (int)threadIdx.x; i < end; i += blockDim.x) split8(first + i);
  }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

struct F32Params {
  bma_attn_args a;
  bma_mask_spec spec;
  bma_block_lists l;
  float scale_log2;
  int* status;
  LaunchOrder order;
  int parts;       // CTAs of a cluster that share a walk
  int first;       // forward: number of tiles, in launch order, that an earlier launch has done
};

// ---- results that are not finite ----------------------------------------------------------------------------------
// The planes of an infinity, a NaN or a finite value above bfloat16's largest (3.39e38) are not numbers, and neither is
// any sum that such a value, or an overflow of the products, reaches.  A CTA that finds one among its results
// does its block row again with the FP32 tile functions, whose results these are then: two rows of 64-tiles over the same
// lists, on the 256 row threads, in the shared memory of the CTA.  (Written behind the kernel's end so that the
// main path pays one multiply-add per result for it; a second launch over flagged tiles cost 4 - 12 us a call.)
__device__ __forceinline__ void note_finite(float& z, float v) { z = fmaf(v, 0.f, z); }   // NaN from the first such v

struct RowSync {   // the 256 row threads
  static __device__ __forceinline__ void sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
  static __device__ __forceinline__ bool any(bool x) {
    uint32_t r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, 256, p;\n selp.u32 %0, 1, 0, q;\n}" : "=r"(r) : "r"((uint32_t)x) : "memory");
    return r != 0;
  }
};
enum RedoPass { REDO_FWD, REDO_DKDV, REDO_DQ };
template <RedoPass PASS, int DC>
__device__ __noinline__ void redo_row(float* smem, const F32Params& fp, int tile128, int h, int b) {
  const SimtParams p{fp.a, fp.spec, fp.l, fp.scale_log2};
  const bool do_f32 = fp.a.d_o.dtype == BMA_DTYPE_F32;
  for (int half = 0; half < 2; ++half) {
    const int tile = 2 * tile128 + half;
    if (tile * TQ >= (PASS == REDO_DKDV ? fp.a.L : fp.a.N)) return;
    RowSync::sync();   // the shared memory is free: its last readers have arrived here
    if constexpr (PASS == REDO_FWD) {
      fwd_tile<float, DC, true, RowSync>(smem, p, tile, h, b);
    } else if constexpr (PASS == REDO_DKDV) {
      if (do_f32) dkdv_tile<float, float, DC, true, RowSync>(smem, p, tile, h, b);
      else dkdv_tile<float, __nv_bfloat16, DC, true, RowSync>(smem, p, tile, h, b);
    } else {
      if (do_f32) dq_tile<float, float, DC, true, RowSync>(smem, p, tile, h, b);
      else dq_tile<float, __nv_bfloat16, DC, true, RowSync>(smem, p, tile, h, b);
    }
  }
}

// Merged kv list of one query tile in shared memory, ascending, every block once: kv tile | partial << 15.
// Called by all threads of the CTA between two __syncthreads of its own; returns the number of entries.
template <int MAX>
struct KvList {
  uint16_t entry[MAX];
  uint8_t cls[MAX];
  int count;
};
template <int MAX>
__device__ __forceinline__ int build_kv_list(KvList<MAX>& s, const bma_block_lists& l, const bma_mask_spec& spec, int b, int h, int qi) {
  const int NKV = l.NKV, lane = threadIdx.x & 31;
  const int64_t lrow = ((int64_t)(l.B == 1 ? 0 : b) * l.H + (l.H == 1 ? 0 : h)) * l.NQ + qi;
  if (l.kv_num) {
    for (int i = threadIdx.x; i < NKV; i += kThreads) s.cls[i] = 0;
    __syncthreads();
    const int nfull = l.full_kv_num[lrow], npart = l.kv_num[lrow];
    for (int i = threadIdx.x; i < nfull; i += kThreads) s.cls[l.full_kv_idx[lrow * NKV + i]] = 2;
    for (int i = threadIdx.x; i < npart; i += kThreads) s.cls[l.kv_idx[lrow * NKV + i]] = 1;
  } else {   // no lists: a mask of interval terms, whose blocks are known from the indices
    for (int i = threadIdx.x; i < NKV; i += kThreads) s.cls[i] = (uint8_t)interval_class(spec, qi, i, BM, BM);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int count = 0;
    for (int base = 0; base < NKV; base += 32) {
      const int j = base + lane;
      const int c = j < NKV ? s.cls[j] : 0;
      const unsigned m = __ballot_sync(0xffffffffu, c != 0);
      if (c) s.entry[count + __popc(m & ((1u << lane) - 1))] = (uint16_t)(j | (c == 1 ? 0x8000 : 0));
      count += __popc(m);
    }
    if (lane == 0) s.count = count;
  }
  __syncthreads();
  return s.count;
}

// Allowed-key bits of query row q for the 64 keys from k0 (two words).
__device__ __forceinline__ void row_bits64(const bma_mask_spec& spec, int b, int h, int q, int k0, uint32_t (&bits)[2]) {
  const MaskView mv = make_mask_view(spec, b, h);
  int jlo, jhi;
  row_interval(mv, q, k0, jlo, jhi);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int lo = max(jlo - c * 32, 0), hi = min(jhi - c * 32, 31);
    bits[c] = (lo <= hi) ? ((0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) : 0u;
    if (bits[c] && (mv.flags & kTableTerms)) bits[c] &= table_bits_row32(mv, q, k0 + c * 32);
  }
}

// Probabilities of 32 columns: those that `bits` does not allow become 0.
__device__ __forceinline__ void keep_allowed(float2* pr, uint32_t bits) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (!((bits >> (2 * j)) & 1u)) pr[j].x = 0.f;
    if (!((bits >> (2 * j + 1)) & 1u)) pr[j].y = 0.f;
  }
}

// 128 rows of `cols` staged floats (row pitch `pitch`) to a [*, *, *, d] tensor, whole rows per warp.
template <int NT>
__device__ __forceinline__ void store_rows(const float* stage, int pitch, const bma_tensor& t, int b, int l0, int lmax, int h, int d, int tid) {
  const int rows = min(BM, lmax - l0);
  const bool vec = (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && ((t.stride_b | t.stride_l | t.stride_h) & 3) == 0 && (d & 3) == 0;
  const int64_t base = (int64_t)b * t.stride_b + (int64_t)l0 * t.stride_l + (int64_t)h * t.stride_h;
  if (vec) {
    const int per = d / 4;
    for (int i = tid; i < rows * per; i += NT) {
      const int r = i / per, c = (i - r * per) * 4;
      const float4 v = *reinterpret_cast<const float4*>(stage + r * pitch + c);
      const int64_t off = base + (int64_t)r * t.stride_l + c;
      if (t.dtype == BMA_DTYPE_F32) *reinterpret_cast<float4*>(static_cast<float*>(t.ptr) + off) = v;
      else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(t.ptr) + off) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
    }
  } else {
    for (int i = tid; i < rows * d; i += NT) {
      const int r = i / d, c = i - r * d;
      const int64_t off = base + (int64_t)r * t.stride_l + c;
      if (t.dtype == BMA_DTYPE_F32) static_cast<float*>(t.ptr)[off] = stage[r * pitch + c];
      else static_cast<__nv_bfloat16*>(t.ptr)[off] = __float2bfloat16_rn(stage[r * pitch + c]);
    }
  }
}

// Rows of a gradient whose tile's walk is shared out over the CTAs of a cluster: the sum of the partials that each has staged at `stage`, the rows
// dealt out over the CTAs, four columns to one of the 256 row threads; a result that is not finite is noted in the first CTA.
template <int COLS>
__device__ __noinline__ void sum_rows(const float* stage, int pitch, const bma_tensor& t, int b, int l0, int lmax, int h, int d, int parts, int part, int* not_finite) {
  const bool vec = (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && ((t.stride_b | t.stride_l | t.stride_h) & 3) == 0 && (d & 3) == 0;
  float z = 0.f;
#pragma unroll 1
  for (int i = threadIdx.x; i < (BM + parts - 1) / parts * (COLS / 4); i += 256) {
    const int row = part + parts * (i / (COLS / 4)), c = (i % (COLS / 4)) * 4;
    if (row >= BM || l0 + row >= lmax || c >= d) continue;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int src = 0; src < parts; ++src) {
      const float4 v = cluster_ld4(cluster_addr(stage + row * pitch + c, (uint32_t)src));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    note_finite(z, (s.x + s.y) + (s.z + s.w));
    float* dst = static_cast<float*>(t.ptr) + (int64_t)b * t.stride_b + (int64_t)(l0 + row) * t.stride_l + (int64_t)h * t.stride_h + c;
    if (vec) {
      *reinterpret_cast<float4*>(dst) = s;
    } else {
      const float e4[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e < d) dst[e] = e4[e];
    }
  }
  if (!(z == 0.f)) cluster_st(cluster_addr(not_finite, 0), 1);
}

// Rows of a tile whose key list is shared out over the CTAs of a cluster: the weighted sum of their partials (two per CTA: [2][BM] rows
// of DP + 4 floats at `stage`, maximum and sum at `ml`) relative to their common maximum.  Half a warp per row, eight warps, the rows
// dealt out over the CTAs; a result that is not finite is noted in the first CTA.
template <int DP>
__device__ __noinline__ void sum_parts(const float* stage, const float* ml, int* not_finite, const F32Params& p, int parts, int part, int q0, int h, int b) {
  const bma_attn_args& a = p.a;
  const int lane = threadIdx.x & 31, c = lane & 15, warp = threadIdx.x >> 5, sources = 2 * parts;
  constexpr int kPitch = DP + 4;
  const bool vec = (reinterpret_cast<uintptr_t>(a.o.ptr) & 15) == 0 && ((a.o.stride_b | a.o.stride_l | a.o.stride_h) & 3) == 0 && (a.d & 3) == 0;
  float z = 0.f;
#pragma unroll 1
  for (int i0 = warp * 2; i0 * parts < BM; i0 += 16) {
    const int i = part + parts * (i0 + (lane >> 4)), q = q0 + i;
    const bool valid = i < BM && q < a.N;
    float m = -INFINITY, l = 0.f;
    if (valid && c < sources) {
      const uint32_t at = cluster_addr(ml + (c & 1) * 2 * BM + i, (uint32_t)(c >> 1));
      m = cluster_ld(at);
      l = cluster_ld(at + BM * (uint32_t)sizeof(float));
    }
    float mt = m;
#pragma unroll
    for (int off = 8; off; off >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, off));
    const float f = ex2(m - (mt == -INFINITY ? 0.f : mt));
    float lt = l * f;
#pragma unroll
    for (int off = 8; off; off >>= 1) lt += __shfl_xor_sync(0xffffffffu, lt, off);
    float4 acc[DP / 64];
#pragma unroll
    for (int u = 0; u < DP / 64; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* mine = stage + (valid ? i : 0) * kPitch + c * 4;
#pragma unroll 4
    for (int src = 0; src < sources; ++src) {
      const uint32_t at = cluster_addr(mine + (src & 1) * BM * kPitch, (uint32_t)(src >> 1));
      const float w = __shfl_sync(0xffffffffu, f, src, 16);
#pragma unroll
      for (int u = 0; u < DP / 64; ++u) {
        const float4 v = cluster_ld4(at + u * 256);
        acc[u].x = fmaf(v.x, w, acc[u].x); acc[u].y = fmaf(v.y, w, acc[u].y); acc[u].z = fmaf(v.z, w, acc[u].z); acc[u].w = fmaf(v.w, w, acc[u].w);
      }
    }
    if (!valid) continue;
    if (c == 0 && a.lse) a.lse[((int64_t)b * a.Hq + h) * a.N + q] = lt > 0.f ? (mt + log2f(lt)) * kLn2 : -INFINITY;
    const float inv = lt > 0.f ? 1.f / lt : 0.f;   // (0 for a NaN as well: then a sum below is not finite)
#pragma unroll
    for (int u = 0; u < DP / 64; ++u) {
      float o4[4] = {acc[u].x * inv, acc[u].y * inv, acc[u].z * inv, acc[u].w * inv};
      note_finite(z, (o4[0] + o4[1]) + (o4[2] + o4[3]));
      const int col = u * 64 + c * 4;
      const int64_t off = (int64_t)b * a.o.stride_b + (int64_t)q * a.o.stride_l + (int64_t)h * a.o.stride_h + col;
      if (vec && col < a.d) {
        if (a.o.dtype == BMA_DTYPE_F32) *reinterpret_cast<float4*>(static_cast<float*>(a.o.ptr) + off) = make_float4(o4[0], o4[1], o4[2], o4[3]);
        else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.o.ptr) + off) = make_uint2(pack_bf16(o4[0], o4[1]), pack_bf16(o4[2], o4[3]));
      } else if (!vec) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (col + e >= a.d) break;
          if (a.o.dtype == BMA_DTYPE_F32) static_cast<float*>(a.o.ptr)[off + e] = o4[e];
          else static_cast<__nv_bfloat16*>(a.o.ptr)[off + e] = __float2bfloat16_rn(o4[e]);
        }
      }
    }
  }
  if (!(z == 0.f)) cluster_st(cluster_addr(not_finite, 0), 1);
}

// =================================================================================================================
// Forward: one CTA per (128-query tile, query head, batch).  Each listed kv tile is cut into two halves of 64 keys;
// warpgroup x (thread = query row) runs its own online softmax over the halves x of all tiles, so that the two
// warpgroups ping-pong on the tensor core without waiting for one another, and the two partial results are merged in
// shared memory at the end.
//   warp 8: K planes, warp 10: V planes and Q planes (TMA), warp 9: MMA issue.
//   TMEM per warpgroup: S (then the planes of P) 128 columns, P V of one half tile 128 columns.
// =================================================================================================================
enum {
  FB_Q = 0, FB_S0, FB_S1, FB_P0, FB_P1, FB_O0, FB_O1, FB_OFREE0, FB_OFREE1, FB_SYNC, FB_K_FULL, FB_K_FREE = FB_K_FULL + 3,
  FB_V_FULL = FB_K_FREE + 3, FB_V_FREE = FB_V_FULL + 3, FB_NUM = FB_V_FREE + 3
};

template <int DP>
struct __align__(1024) FwdSmem {
  static constexpr int kBoxes = DP / 64;
  static constexpr int kStages = DP == 64 ? 3 : 1;   // 128 columns: 96 KB of Q planes leave room for one half tile each of K and V
  uint8_t q[3][kBoxes][kRowBox];
  uint8_t k[kStages][kBoxes][3][kHalfBox];
  uint8_t v[kStages][3][kBoxes][kHalfBox];
  float ml[2][2][BM];                                // running maximum and sum of the two halves
  KvList<kMaxKvFwd> list;
  uint64_t bar[FB_NUM];
  uint32_t tmem_base;
  int not_finite;
};

static_assert(fwd_smem<4>() <= sizeof(FwdSmem<64>) && fwd_smem<8>() <= sizeof(FwdSmem<128>), "a tile is done again in the same shared memory");

// KB: with a key bias, or a scale that is not positive: for a negative one the maximum of the scores is not that of the scaled ones, and a scale of 0
// would make a NaN of a score that the mask has set to -inf before it is scaled (its tile would be done again with FP32 arithmetic).
// SHARED: the CTAs of a cluster share a tile's keys; an instance of its own, since the part costs the plain kernel registers (4 x 4096 tokens,
// 16 heads, causal: the call 1 437 us with it, 1 408 without at 128 head columns, 765 and 757 at 64).
template <int DP, bool KB, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
f32_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ F32Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  using Smem = FwdSmem<DP>;
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  constexpr int kBoxes = Smem::kBoxes, kStages = Smem::kStages;
  const bma_attn_args& a = p.a;
  const int parts = SHARED ? p.parts : 1;
  int qi, h;
  cta_of(p.order, (SHARED ? p.first : 0) + (int)blockIdx.x / parts, qi, h);
  qi = p.order.tiles - 1 - qi;
  const int b = h / a.Hq;
  h -= b * a.Hq;
  const int hk = h / (a.Hq / a.Hkv);
  const int q0 = qi * BM;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, wg = warp >> 2;

  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_device_error(p.status, 601);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < FB_NUM; ++i) {
      uint32_t count = 1;
      if (i == FB_P0 || i == FB_P1 || i == FB_OFREE0 || i == FB_OFREE1) count = 128;
      if (i == FB_SYNC) count = 256;
      mbar_init(&sm.bar[i], count);
    }
    sm.not_finite = 0;
    fence_barrier_init();
  }
  if (warp == 8) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  const int listed = build_kv_list(sm.list, p.l, p.spec, b, h, qi);
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  // this CTA's part of the list
  const int part = (int)blockIdx.x % parts, t0 = listed * part / parts, T = listed * (part + 1) / parts - t0;
  const uint16_t* entry = sm.list.entry + t0;
  // half tiles per warpgroup: the second half of the last tile may lie past the end of the keys
  const int T0 = T;
  const int T1 = (T > 0 && (int)(entry[T - 1] & 0x7fff) * 128 + BH >= a.L) ? T - 1 : T;

  if (wg == 2) {
    setmaxnreg_dec_80();
    if (warp == 8 && lane == 0 && T > 0) {
      // ------------------------------------------------------------ K planes
      bool ok = true;
      int i = 0;
      for (int n = 0; n < T && ok; ++n)
        for (int x = 0; x < 2; ++x) {
          if (n >= (x ? T1 : T0)) continue;
          const int st = i % kStages;
          if (i >= kStages) ok = mbar_wait(&sm.bar[FB_K_FREE + st], (i / kStages - 1) & 1);
          if (!ok) break;
          const int row = (int)(entry[n] & 0x7fff) * 128 + x * BH;
          mbar_expect_tx(&sm.bar[FB_K_FULL + st], 3 * kBoxes * kHalfBox);
#pragma unroll
          for (int box = 0; box < kBoxes; ++box)
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) tma_load_4d(sm.k[st][box][pl], &map_k, &sm.bar[FB_K_FULL + st], box * 64, hk, row, b + pl * a.B);
          ++i;
        }
      if (!ok) report_device_error(p.status, 610);
    } else if (warp == 10 && lane == 0) {
      // ------------------------------------------------------------ Q and V planes
      if (T > 0) {
        mbar_expect_tx(&sm.bar[FB_Q], 3 * kBoxes * kRowBox);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
#pragma unroll
          for (int box = 0; box < kBoxes; ++box) tma_load_4d(sm.q[pl][box], &map_q, &sm.bar[FB_Q], box * 64, h, q0, b + pl * a.B);
      }
      bool ok = true;
      int i = 0;
      for (int n = 0; n < T && ok; ++n)
        for (int x = 0; x < 2; ++x) {
          if (n >= (x ? T1 : T0)) continue;
          const int st = i % kStages;
          if (i >= kStages) ok = mbar_wait(&sm.bar[FB_V_FREE + st], (i / kStages - 1) & 1);
          if (!ok) break;
          const int row = (int)(entry[n] & 0x7fff) * 128 + x * BH;
          mbar_expect_tx(&sm.bar[FB_V_FULL + st], 3 * kBoxes * kHalfBox);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl)
#pragma unroll
            for (int box = 0; box < kBoxes; ++box) tma_load_4d(sm.v[st][pl][box], &map_v, &sm.bar[FB_V_FULL + st], box * 64, hk, row, b + pl * a.B);
          ++i;
        }
      if (!ok) report_device_error(p.status, 612);
    } else if (warp == 9 && T > 0) {
      // ------------------------------------------------------------ MMA issue (whole warp, one elected lane issues)
      const bool leader = elect_one();
      const uint64_t dq = make_smem_desc(smem_u32(sm.q), 16, 1024);
      const uint64_t dk = make_smem_desc(smem_u32(sm.k), 16, 1024);
      const uint64_t dv = make_smem_desc(smem_u32(sm.v), kHalfBox, 1024);
      constexpr uint32_t kStageUnits = (3 * kBoxes * kHalfBox) >> 4;
      auto issue_s = [&](int x, int i) -> bool {
        const int st = i % kStages;
        if (!mbar_wait(&sm.bar[FB_K_FULL + st], (i / kStages) & 1)) return false;
        tc_fence_after();
        product_rows<kBoxes>(leader, tmem + x * 256, dq, dk + st * kStageUnits);
        if (leader) { mma_commit(&sm.bar[FB_S0 + x]); mma_commit(&sm.bar[FB_K_FREE + st]); }
        return true;
      };
      bool ok = mbar_wait(&sm.bar[FB_Q], 0) && issue_s(0, 0);
      if (ok && T1 > 0) ok = issue_s(1, 1);
      for (int n = 0; n < T && ok; ++n)
        for (int x = 0; x < 2 && ok; ++x) {
          if (n >= (x ? T1 : T0)) continue;
          const int i = 2 * n + x, st = i % kStages;
          ok = mbar_wait(&sm.bar[FB_V_FULL + st], (i / kStages) & 1) && mbar_wait(&sm.bar[FB_P0 + x], n & 1);
          if (ok && n > 0) ok = mbar_wait(&sm.bar[FB_OFREE0 + x], (n - 1) & 1);
          if (!ok) break;
          tc_fence_after();
          product_cols<kBoxes>(leader, tmem + x * 256 + 128, tmem + x * 256, dv + st * kStageUnits);
          if (leader) { mma_commit(&sm.bar[FB_O0 + x]); mma_commit(&sm.bar[FB_V_FREE + st]); }
          // the next S of this half overwrites the planes of P, behind the MMAs that read them
          if (n + 1 < (x ? T1 : T0)) ok = issue_s(x, i + 2);
        }
      if (!ok && leader) report_device_error(p.status, 620);
    }
  } else {
    // -------------------------------------------------------------- softmax warpgroups
    setmaxnreg_inc_208();
    const int x = wg, row = threadIdx.x & 127, q = q0 + row;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem + x * 256 + lane_base, tmem_o = tmem_s + 128;
    const float kb2 = a.key_bias ? __ldg(a.key_bias + h) * kLog2e : 0.f;
    const int Tx = x ? T1 : T0;
    float2 o[DP / 2];
#pragma unroll
    for (int j = 0; j < DP / 2; ++j) o[j] = both(0.f);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int n = 0; n < Tx; ++n) {
      const uint32_t e = entry[n];
      const int k0 = (int)(e & 0x7fff) * 128 + x * BH;
      uint32_t bits[2] = {0xffffffffu, 0xffffffffu};
      if (e & 0x8000u) row_bits64(p.spec, b, h, q, k0, bits);
      const bool cut = (e & 0x8000u) != 0;
      const float kbase = (float)(p.spec.k_offset + k0);
      // 16 scores from tensor memory (KB: in log2 units)
      auto scores16 = [&](int c, float2* v) {
        uint32_t r0[16], r1[16];
        tmem_ld16(tmem_s + c * 16, r0);
        tmem_ld16(tmem_s + 64 + c * 16, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = halves(r0, r1, j);
          if constexpr (KB)
            v[j] = __ffma2_rn(v[j], both(p.scale_log2), make_float2(kb2 * (kbase + (float)(c * 16 + 2 * j)), kb2 * (kbase + (float)(c * 16 + 2 * j + 1))));
        }
        if (cut) {
          const uint32_t w = (c < 2 ? bits[0] : bits[1]) >> ((c & 1) * 16);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (!((w >> (2 * j)) & 1u)) v[j].x = -INFINITY;
            if (!((w >> (2 * j + 1)) & 1u)) v[j].y = -INFINITY;
          }
        }
      };
      ok = mbar_wait(&sm.bar[FB_S0 + x], n & 1);
      if (!ok) break;
      tc_fence_after();
      // 128 head columns leave no registers for 64 scores beside O: those are read twice, once for the maximum
      constexpr bool kKeep = DP == 64;
      float2 s[kKeep ? 32 : 8];
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll (kKeep ? 4 : 1)
      for (int c = 0; c < 4; ++c) {
        float2* v = s + (kKeep ? c * 8 : 0);
        scores16(c, v);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          mx0 = max3(mx0, v[j].x, v[j].y);
          mx1 = max3(mx1, v[j + 1].x, v[j + 1].y);
        }
      }
      const float mx = fmaxf(mx0, mx1);
      const float m_new = fmaxf(m, KB || mx == -INFINITY ? mx : mx * p.scale_log2), m_safe = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = ex2(m - m_safe);
      m = m_new;
      const float2 sc = both(KB ? 1.f : p.scale_log2);
      float2 rs[2] = {both(0.f), both(0.f)};
#pragma unroll (kKeep ? 4 : 1)
      for (int c = 0; c < 4; ++c) {
        float2* v = s + (kKeep ? c * 8 : 0);
        if (!kKeep) scores16(c, v);
        uint32_t hm[16], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 t = __ffma2_rn(v[j], sc, both(-m_safe));
          const float2 pr = make_float2(ex2(t.x), ex2(t.y));
          rs[j & 1] = __fadd2_rn(rs[j & 1], pr);
          split3(pr, hm[j], hm[8 + j], lo[j]);
        }
        tmem_st16(tmem_s + c * 16, hm);        // over the 16 + 8 columns whose scores have just been used
        tmem_st8(tmem_s + 64 + c * 16, lo);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[FB_P0 + x]);
      l = l * alpha + ((rs[0].x + rs[0].y) + (rs[1].x + rs[1].y));
      ok = mbar_wait(&sm.bar[FB_O0 + x], n & 1);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < DP / 32; ++c) {
        uint32_t r0[32];
        tmem_ld32(tmem_o + c * 32, r0);
        if constexpr (DP == 64) {
          uint32_t r1[32];
          tmem_ld32(tmem_o + 64 + c * 32, r1);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) o[c * 16 + j] = __ffma2_rn(o[c * 16 + j], both(alpha), halves(r0, r1, j));
        } else {
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            o[c * 16 + j] = __ffma2_rn(o[c * 16 + j], both(alpha), make_float2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1])));
        }
      }
      tc_fence_before();
      mbar_arrive(&sm.bar[FB_OFREE0 + x]);
    }

    // ---- merge the two halves and write O and the log-sum-exp.  After the first rendezvous every MMA of the CTA has
    // completed (each warpgroup has seen its last P V), so the Q planes' buffer is free for staging.
    sm.ml[x][0][row] = m;
    sm.ml[x][1][row] = l;
    uint32_t syncs = 0;
    auto rendezvous = [&]() {
      mbar_arrive(&sm.bar[FB_SYNC]);
      ok = mbar_wait(&sm.bar[FB_SYNC], syncs & 1) && ok;
      ++syncs;
    };
    rendezvous();
    if constexpr (SHARED) {   // both partial results as they are; the cluster adds them up below
      float* stage = reinterpret_cast<float*>(sm.q) + (x * BM + row) * (DP + 4);
#pragma unroll
      for (int j = 0; j < DP; j += 4) *reinterpret_cast<float4*>(stage + j) = make_float4(o[j / 2].x, o[j / 2].y, o[j / 2 + 1].x, o[j / 2 + 1].y);
      if (!ok) report_device_error(p.status, 630 + warp);
    } else {
      const float mo = sm.ml[x ^ 1][0][row], lo = sm.ml[x ^ 1][1][row];
      const float mt = fmaxf(m, mo), ms = (mt == -INFINITY) ? 0.f : mt;
      const float fx = ex2(m - ms), fo = ex2(mo - ms);
      const float lt = l * fx + lo * fo;
      const float mine = lt > 0.f ? fx / lt : 0.f;
      constexpr int kPitch = DP + 4;
      float* stage = reinterpret_cast<float*>(sm.q) + row * kPitch;
      if (x == 0) {
#pragma unroll
        for (int j = 0; j < DP; j += 4) *reinterpret_cast<float4*>(stage + j) = make_float4(o[j / 2].x * mine, o[j / 2].y * mine, o[j / 2 + 1].x * mine, o[j / 2 + 1].y * mine);
      }
      rendezvous();
      if (x == 1) {
        float z = 0.f;
#pragma unroll
        for (int j = 0; j < DP; j += 4) {
          float4 v = *reinterpret_cast<float4*>(stage + j);
          v.x = fmaf(o[j / 2].x, mine, v.x); v.y = fmaf(o[j / 2].y, mine, v.y); v.z = fmaf(o[j / 2 + 1].x, mine, v.z); v.w = fmaf(o[j / 2 + 1].y, mine, v.w);
          *reinterpret_cast<float4*>(stage + j) = v;
          note_finite(z, (v.x + v.y) + (v.z + v.w));
        }
        if (z != 0.f) sm.not_finite = 1;
        if (q < a.N && a.lse) a.lse[((int64_t)b * a.Hq + h) * a.N + q] = lt > 0.f ? (mt + log2f(lt)) * kLn2 : -INFINITY;
      }
      rendezvous();
      if (ok) store_rows<256>(reinterpret_cast<const float*>(sm.q), kPitch, a.o, b, q0, a.N, h, a.d, threadIdx.x);
      else report_device_error(p.status, 630 + warp);
    }
  }
  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    if (warp < 8) sum_parts<DP>(reinterpret_cast<const float*>(sm.q), &sm.ml[0][0][0], &sm.not_finite, p, parts, part, q0, h, b);
    cluster_sync();   // shared memory stays until the others have read it
    if (part > 0) return;
  }
  if (warp < 8 && sm.not_finite) redo_row<REDO_FWD, DP / 16>(reinterpret_cast<float*>(smem_raw), p, qi, h, b);
}

// =================================================================================================================
// dK / dV: one CTA per (128-key tile, kv head, batch); K and V planes stay in shared memory, the q tiles of the q-side
// lists come in halves of 64 queries.  Both warpgroups work on every half tile, 32 query columns each (thread = key row):
//     St = K Q^T -> P, dPt = V dO^T -> dS,   dV += Pt dO (warpgroup 0 sums it in registers),  dK += dSt Q (warpgroup 1)
// MMA order  dV(n) St(n+1) dK(n) dPt(n+1): the next scores are computed while this tile's gradients accumulate.
//   warp 8: K, V, Q planes, warp 11: dO planes (TMA), warp 9: MMA issue, warp 10: lse and delta of the coming half tile.
// =================================================================================================================
enum {
  KB_KV = 0, KB_S, KB_DP, KB_P, KB_DS, KB_DV, KB_DK, KB_DVFREE, KB_DKFREE, KB_EPI0, KB_EPI1,
  KB_Q_FULL, KB_Q_FREE = KB_Q_FULL + 2, KB_DO_FULL = KB_Q_FREE + 2, KB_DO_FREE = KB_DO_FULL + 2, KB_STAT = KB_DO_FREE + 2,
  KB_NUM = KB_STAT + 2
};
struct WalkShare { int g, it, tiles; };   // the part of a walk that a CTA of a cluster takes: its first head and entry, its number of tiles
struct __align__(1024) DkdvSmem {
  uint8_t k[3][kRowBox];
  uint8_t v[3][kRowBox];
  uint8_t q[2][3][kHalfBox];
  uint8_t d_o[2][3][kHalfBox];
  alignas(16) float nlse2[2][BH], ndelta[2][BH];   // minus the log-sum-exp (log2 units) and delta
  uint64_t bar[KB_NUM];
  uint32_t tmem_base;
  WalkShare share;
  int not_finite;
};
static_assert(dkdv_smem<4>() <= sizeof(DkdvSmem), "a tile is done again in the same shared memory");
constexpr uint32_t COL_ST = 0, COL_DPT = 128, COL_DV = 256, COL_DK = 384;

// flattened walk over (group head, listed q tile, half tile); a half tile past the end of the queries is left out
template <bool SHARED>   // a part of the walk
struct HalfIter {
  QTileIter it;
  int N, h, qi, left;
  bool partial, second;
  __device__ HalfIter(const bma_block_lists& l, int b, int hk, int G, int kj, int N_, const WalkShare& w)
      : it(l, b, hk, G, kj), N(N_), h(0), qi(0), left(SHARED ? w.tiles : 0), partial(false), second(false) {
    if (SHARED && left > 0) it.start(w.g, w.it);
  }
  __device__ bool next(int& h_, int& q0_, bool& partial_) {
    if (second) {
      second = false;
      q0_ = qi * 128 + BH;
    } else {
      if ((SHARED && --left < 0) || !it.next(h, qi, partial)) return false;
      q0_ = qi * 128;
      second = q0_ + BH < N;
    }
    h_ = h;
    partial_ = partial;
    return true;
  }
};

// (one thread)
__device__ __noinline__ WalkShare walk_share(const F32Params& p, int b, int hk, int G, int kj) {
  WalkShare w{0, 0, 0};
  auto entries = [&](int g) {
    const int64_t row = ((int64_t)(p.l.B == 1 ? 0 : b) * p.l.H + (p.l.H == 1 ? 0 : hk * G + g)) * p.l.NKV + kj;
    return p.l.full_q_num[row] + p.l.q_num[row];
  };
  int all = 0;
  for (int g = 0; g < G; ++g) all += entries(g);
  const int part = (int)blockIdx.x % p.parts, skip = all * part / p.parts;
  w.tiles = all * (part + 1) / p.parts - skip;
  for (w.it = skip; w.g < G - 1; ++w.g) {
    const int n = entries(w.g);
    if (w.it < n) break;
    w.it -= n;
  }
  return w;
}

template <bool KB, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
f32_dkdv_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                const __grid_constant__ CUtensorMap map_qh, const __grid_constant__ CUtensorMap map_do, const __grid_constant__ F32Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  DkdvSmem& sm = *reinterpret_cast<DkdvSmem*>(smem_raw);
  const bma_attn_args& a = p.a;
  const int parts = SHARED ? p.parts : 1;
  int kj, hk;
  cta_of(p.order, (int)blockIdx.x / parts, kj, hk);
  const int b = hk / a.Hkv, G = a.Hq / a.Hkv;
  hk -= b * a.Hkv;
  const int k0 = kj * BM;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_device_error(p.status, 701);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < KB_NUM; ++i) {
      uint32_t count = 1;
      if (i == KB_P || i == KB_DS) count = 256;
      if (i == KB_DVFREE || i == KB_DKFREE || i == KB_EPI0 || i == KB_EPI1) count = 128;
      if (i == KB_STAT || i == KB_STAT + 1) count = 32;
      mbar_init(&sm.bar[i], count);
    }
    sm.not_finite = 0;
    fence_barrier_init();
    mbar_expect_tx(&sm.bar[KB_KV], 6 * kRowBox);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) {
      tma_load_4d(sm.k[pl], &map_k, &sm.bar[KB_KV], 0, hk, k0, b + pl * a.B);
      tma_load_4d(sm.v[pl], &map_v, &sm.bar[KB_KV], 0, hk, k0, b + pl * a.B);
    }
    if constexpr (SHARED) sm.share = walk_share(p, b, hk, G, kj);
  }
  if (warp == 8) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp >= 8) {
    setmaxnreg_dec_80();
    HalfIter<SHARED> walk(p.l, b, hk, G, kj, a.N, sm.share);
    int h, q0;
    bool partial, ok = true;
    if (warp == 8 || warp == 11) {
      // ------------------------------------------------------------ Q (warp 8) and dO (warp 11) planes
      if (lane == 0) {
        const bool is_q = warp == 8;
        for (int n = 0; ok && walk.next(h, q0, partial); ++n) {
          const int st = n & 1;
          uint64_t* full = &sm.bar[(is_q ? KB_Q_FULL : KB_DO_FULL) + st];
          if (n >= 2) ok = mbar_wait(&sm.bar[(is_q ? KB_Q_FREE : KB_DO_FREE) + st], ((n >> 1) - 1) & 1);
          if (!ok) break;
          mbar_expect_tx(full, 3 * kHalfBox);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) tma_load_4d(is_q ? sm.q[st][pl] : sm.d_o[st][pl], is_q ? &map_qh : &map_do, full, 0, h, q0, b + pl * a.B);
        }
        if (!ok) report_device_error(p.status, 710);
      }
    } else if (warp == 10) {
      // ------------------------------------------------------------ row statistics of the coming half tiles
      for (int n = 0; ok && walk.next(h, q0, partial); ++n) {
        const int st = n & 1;
        if (n >= 2) ok = mbar_wait(&sm.bar[KB_Q_FREE + st], ((n >> 1) - 1) & 1);   // dK(n-2) is behind every read of its statistics
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int idx = e * 32 + lane, q = q0 + idx;
          const int64_t off = ((int64_t)b * a.Hq + h) * a.N + q;
          const float lv = q < a.N ? __ldg(a.lse + off) : -INFINITY;
          sm.nlse2[st][idx] = (lv == -INFINITY) ? -INFINITY : -lv * kLog2e;   // -inf: the probabilities of the row become exactly 0
          sm.ndelta[st][idx] = q < a.N ? -__ldg(a.delta + off) : 0.f;
        }
        mbar_arrive(&sm.bar[KB_STAT + st]);
      }
      if (!ok && lane == 0) report_device_error(p.status, 715);
    } else {
      // ------------------------------------------------------------ MMA issue
      const bool leader = elect_one();
      const uint64_t dk = make_smem_desc(smem_u32(sm.k), 16, 1024), dv = make_smem_desc(smem_u32(sm.v), 16, 1024);
      const uint64_t dq = make_smem_desc(smem_u32(sm.q), 16, 1024), ddo = make_smem_desc(smem_u32(sm.d_o), 16, 1024);
      const uint64_t dqm = make_smem_desc(smem_u32(sm.q), kHalfBox, 1024), ddom = make_smem_desc(smem_u32(sm.d_o), kHalfBox, 1024);
      constexpr uint32_t kStageUnits = (3 * kHalfBox) >> 4;
      auto issue_st = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[KB_Q_FULL + (n & 1)], (n >> 1) & 1)) return false;
        tc_fence_after();
        product_rows<1>(leader, tmem + COL_ST, dk, dq + (n & 1) * kStageUnits);
        if (leader) mma_commit(&sm.bar[KB_S]);
        return true;
      };
      auto issue_dpt = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[KB_DO_FULL + (n & 1)], (n >> 1) & 1)) return false;
        tc_fence_after();
        product_rows<1>(leader, tmem + COL_DPT, dv, ddo + (n & 1) * kStageUnits);
        if (leader) mma_commit(&sm.bar[KB_DP]);
        return true;
      };
      bool have = walk.next(h, q0, partial);
      if (have) ok = mbar_wait(&sm.bar[KB_KV], 0) && issue_st(0) && issue_dpt(0);
      for (int n = 0; have && ok; ++n) {
        const int st = n & 1;
        const bool more = walk.next(h, q0, partial);
        ok = mbar_wait(&sm.bar[KB_P], n & 1);
        if (ok && n > 0) ok = mbar_wait(&sm.bar[KB_DVFREE], (n - 1) & 1);
        if (!ok) break;
        tc_fence_after();
        product_cols<1>(leader, tmem + COL_DV, tmem + COL_ST, ddom + st * kStageUnits);
        if (leader) { mma_commit(&sm.bar[KB_DV]); mma_commit(&sm.bar[KB_DO_FREE + st]); }
        if (more) ok = issue_st(n + 1);
        if (ok) ok = mbar_wait(&sm.bar[KB_DS], n & 1);
        if (ok && n > 0) ok = mbar_wait(&sm.bar[KB_DKFREE], (n - 1) & 1);
        if (!ok) break;
        tc_fence_after();
        product_cols<1>(leader, tmem + COL_DK, tmem + COL_DPT, dqm + st * kStageUnits);
        if (leader) { mma_commit(&sm.bar[KB_DK]); mma_commit(&sm.bar[KB_Q_FREE + st]); }
        if (more) ok = issue_dpt(n + 1);
        have = more;
      }
      if (!ok && leader) report_device_error(p.status, 720);
    }
  } else {
    // -------------------------------------------------------------- row threads
    setmaxnreg_inc_208();
    const int w = warp >> 2, row = threadIdx.x & 127, k = k0 + row;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tm = tmem + lane_base;
    float2 acc[32];   // warpgroup 0: dV, warpgroup 1: dK of this key row
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = both(0.f);
    bool ok = true;
    const uint32_t col_acc = w == 0 ? COL_DV : COL_DK;
    uint64_t* acc_full = &sm.bar[w == 0 ? KB_DV : KB_DK];
    uint64_t* acc_free = &sm.bar[w == 0 ? KB_DVFREE : KB_DKFREE];
    auto flush = [&](int n) -> bool {   // acc += the gradient contribution of half tile n
      if (!mbar_wait(acc_full, n & 1)) return false;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + col_acc + c * 32, r0);
        tmem_ld32(tm + col_acc + 64 + c * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c * 16 + j] = __fadd2_rn(acc[c * 16 + j], halves(r0, r1, j));
      }
      tc_fence_before();
      mbar_arrive(acc_free);
      return true;
    };
    HalfIter<SHARED> walk(p.l, b, hk, G, kj, a.N, sm.share);
    int h, q0, n = 0;
    bool partial;
    for (; ok && walk.next(h, q0, partial); ++n) {
      const int st = n & 1;
      const float kbk = KB ? __ldg(a.key_bias + h) * kLog2e * (float)(p.spec.k_offset + k) : 0.f;
      uint32_t bits = 0xffffffffu;
      if (partial) {
        const MaskView mv = make_mask_view(p.spec, b, h);
        int jlo, jhi;
        col_interval(mv, k, q0 + w * 32, 32, jlo, jhi);
        const int lo = max(jlo, 0), hi = min(jhi, 31);
        bits = (lo <= hi) ? ((0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) : 0u;
        if (mv.flags & kTableTerms) bits &= table_bits_col32(mv, k, q0 + w * 32);
      }
      ok = mbar_wait(&sm.bar[KB_STAT + st], (n >> 1) & 1) && mbar_wait(&sm.bar[KB_S], n & 1);
      if (!ok) break;
      tc_fence_after();
      float2 pr[16];
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_ST + w * 32, r0);
        tmem_ld32(tm + COL_ST + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 lv = *reinterpret_cast<const float4*>(&sm.nlse2[st][w * 32 + j4 * 4]);
          float2 l2[2] = {make_float2(lv.x, lv.y), make_float2(lv.z, lv.w)};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if constexpr (KB) l2[e] = __fadd2_rn(l2[e], both(kbk));
            const float2 t = __ffma2_rn(halves(r0, r1, j4 * 2 + e), both(p.scale_log2), l2[e]);
            pr[j4 * 2 + e] = make_float2(ex2(t.x), ex2(t.y));
          }
        }
        if (partial) keep_allowed(pr, bits);
      }
      store_planes32(tm + COL_ST, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[KB_P]);
      if (w == 1 && n > 0) ok = flush(n - 1);   // dK(n-1) was issued behind St(n): it completes under the exponentials
      if (ok) ok = mbar_wait(&sm.bar[KB_DP], n & 1);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_DPT + w * 32, r0);
        tmem_ld32(tm + COL_DPT + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 dl = *reinterpret_cast<const float4*>(&sm.ndelta[st][w * 32 + j4 * 4]);
          pr[j4 * 2] = __fmul2_rn(pr[j4 * 2], __fadd2_rn(halves(r0, r1, j4 * 2), make_float2(dl.x, dl.y)));
          pr[j4 * 2 + 1] = __fmul2_rn(pr[j4 * 2 + 1], __fadd2_rn(halves(r0, r1, j4 * 2 + 1), make_float2(dl.z, dl.w)));
        }
      }
      store_planes32(tm + COL_DPT, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[KB_DS]);
      if (w == 0) ok = flush(n);
    }
    if (ok && w == 1 && n > 0) ok = flush(n - 1);
    if (ok && n == 0) ok = mbar_wait(&sm.bar[KB_KV], 0);   // let the loads land before their buffers are reused
    // ---- epilogue: every score MMA that read K and V has completed, their buffers stage dV (0) and dK (1)
    constexpr int kPitch = 68;
    float* stage = reinterpret_cast<float*>(w == 0 ? &sm.v[0][0] : &sm.k[0][0]);
    const float sc = w == 0 ? 1.f : a.scale;
    float z = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      acc[j] = __fmul2_rn(acc[j], both(sc));
      note_finite(z, acc[j].x);
      note_finite(z, acc[j].y);
    }
    if (z != 0.f && parts == 1) sm.not_finite = 1;
#pragma unroll
    for (int j = 0; j < 64; j += 4)
      if (ok) *reinterpret_cast<float4*>(stage + row * kPitch + j) = make_float4(acc[j / 2].x, acc[j / 2].y, acc[j / 2 + 1].x, acc[j / 2 + 1].y);
    mbar_arrive(&sm.bar[KB_EPI0 + w]);
    ok = mbar_wait(&sm.bar[KB_EPI0 + w], 0) && ok;
    if (!ok) report_device_error(p.status, 730 + warp);
    else if (parts == 1) store_rows<128>(stage, kPitch, w == 0 ? a.dv : a.dk, b, k0, a.L, hk, a.d, row);
  }
  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    const int part = (int)blockIdx.x % parts;
    if (warp < 8) {
#pragma unroll 1
      for (int i = 0; i < 2; ++i)
        sum_rows<64>(reinterpret_cast<const float*>(i ? sm.k[0] : sm.v[0]), 68, i ? a.dk : a.dv, b, k0, a.L, hk, a.d, parts, part, &sm.not_finite);
    }
    cluster_sync();   // shared memory stays until the others have read it
    if (part > 0) return;
  }
  if (warp < 8 && sm.not_finite) redo_row<REDO_DKDV, 4>(reinterpret_cast<float*>(smem_raw), p, kj, hk, b);
}

// =================================================================================================================
// dQ: one CTA per (128-query tile, query head, batch); Q and dO planes stay in shared memory, the listed kv tiles come in
// halves of 64 keys through rings of three K and two V half tiles.  S is double buffered, so the next half's scores and
// exponentials run while  dQ(n) dP(n+1)  execute.  Both warpgroups work on every half tile (32 key columns each) and
// sum 32 columns of dQ each in registers.
// =================================================================================================================
enum {
  QB_Q = 0, QB_S, QB_DP = QB_S + 2, QB_DS, QB_DQ, QB_DQFREE, QB_EPI, QB_K_FULL, QB_K_FREE = QB_K_FULL + 3, QB_V_FULL = QB_K_FREE + 3,
  QB_V_FREE = QB_V_FULL + 2, QB_NUM = QB_V_FREE + 2
};
struct __align__(1024) DqSmem {
  uint8_t q[3][kRowBox];
  uint8_t d_o[3][kRowBox];
  uint8_t k[3][3][kHalfBox];
  uint8_t v[2][3][kHalfBox];
  KvList<kMaxKvBwd> list;
  uint64_t bar[QB_NUM];
  uint32_t tmem_base;
  int not_finite;
};
static_assert(dq_smem<4>() <= sizeof(DqSmem), "as above");
constexpr uint32_t COL_S2 = 0, COL_DP2 = 256, COL_DQ2 = 384;   // S: two buffers of 128 columns

template <bool KB, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
f32_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kh,
              const __grid_constant__ CUtensorMap map_vh, const __grid_constant__ CUtensorMap map_do, const __grid_constant__ F32Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  DqSmem& sm = *reinterpret_cast<DqSmem*>(smem_raw);
  const bma_attn_args& a = p.a;
  const int parts = SHARED ? p.parts : 1;
  int qi, h;
  cta_of(p.order, (int)blockIdx.x / parts, qi, h);
  qi = p.order.tiles - 1 - qi;
  const int b = h / a.Hq;
  h -= b * a.Hq;
  const int hk = h / (a.Hq / a.Hkv);
  const int q0 = qi * BM;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_device_error(p.status, 801);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < QB_NUM; ++i) mbar_init(&sm.bar[i], (i == QB_DS || i == QB_DQFREE || i == QB_EPI) ? 256 : 1);
    sm.not_finite = 0;
    fence_barrier_init();
    mbar_expect_tx(&sm.bar[QB_Q], 6 * kRowBox);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) {
      tma_load_4d(sm.q[pl], &map_q, &sm.bar[QB_Q], 0, h, q0, b + pl * a.B);
      tma_load_4d(sm.d_o[pl], &map_do, &sm.bar[QB_Q], 0, h, q0, b + pl * a.B);
    }
  }
  if (warp == 8) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  const int listed = build_kv_list(sm.list, p.l, p.spec, b, h, qi);
  const int part = (int)blockIdx.x % parts, t0 = listed * part / parts, T = listed * (part + 1) / parts - t0;   // this CTA's part of the list
  const uint16_t* entry = sm.list.entry + t0;
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  // half tiles in all; the second half of the last tile may lie past the end of the keys
  const int total = T == 0 ? 0 : 2 * T - ((int)(entry[T - 1] & 0x7fff) * 128 + BH >= a.L ? 1 : 0);

  if (warp >= 8) {
    setmaxnreg_dec_80();
    bool ok = true;
    if ((warp == 8 || warp == 10) && lane == 0) {
      // ------------------------------------------------------------ K (warp 8) and V (warp 10) planes
      const bool is_k = warp == 8;
      const int stages = is_k ? 3 : 2;
      for (int n = 0; n < total && ok; ++n) {
        const int st = n % stages;
        uint64_t* full = &sm.bar[(is_k ? QB_K_FULL : QB_V_FULL) + st];
        if (n >= stages) ok = mbar_wait(&sm.bar[(is_k ? QB_K_FREE : QB_V_FREE) + st], (n / stages - 1) & 1);
        if (!ok) break;
        const int row = (int)(entry[n >> 1] & 0x7fff) * 128 + (n & 1) * BH;
        mbar_expect_tx(full, 3 * kHalfBox);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) tma_load_4d(is_k ? sm.k[st][pl] : sm.v[st][pl], is_k ? &map_kh : &map_vh, full, 0, hk, row, b + pl * a.B);
      }
      if (!ok) report_device_error(p.status, 810);
    } else if (warp == 9 && total > 0) {
      // ------------------------------------------------------------ MMA issue
      const bool leader = elect_one();
      const uint64_t dq = make_smem_desc(smem_u32(sm.q), 16, 1024), ddo = make_smem_desc(smem_u32(sm.d_o), 16, 1024);
      const uint64_t dk = make_smem_desc(smem_u32(sm.k), 16, 1024), dv = make_smem_desc(smem_u32(sm.v), 16, 1024);
      const uint64_t dkm = make_smem_desc(smem_u32(sm.k), kHalfBox, 1024);
      constexpr uint32_t kStageUnits = (3 * kHalfBox) >> 4;
      auto issue_s = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[QB_K_FULL + n % 3], (n / 3) & 1)) return false;
        tc_fence_after();
        product_rows<1>(leader, tmem + COL_S2 + (n & 1) * 128, dq, dk + (n % 3) * kStageUnits);
        if (leader) mma_commit(&sm.bar[QB_S + (n & 1)]);
        return true;
      };
      auto issue_dp = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[QB_V_FULL + (n & 1)], (n >> 1) & 1)) return false;
        tc_fence_after();
        product_rows<1>(leader, tmem + COL_DP2, ddo, dv + (n & 1) * kStageUnits);
        if (leader) { mma_commit(&sm.bar[QB_DP]); mma_commit(&sm.bar[QB_V_FREE + (n & 1)]); }
        return true;
      };
      ok = mbar_wait(&sm.bar[QB_Q], 0) && issue_s(0) && issue_dp(0);
      if (ok && total > 1) ok = issue_s(1);
      for (int n = 0; n < total && ok; ++n) {
        ok = mbar_wait(&sm.bar[QB_DS], n & 1);
        if (ok && n > 0) ok = mbar_wait(&sm.bar[QB_DQFREE], (n - 1) & 1);
        if (!ok) break;
        tc_fence_after();
        product_cols<1>(leader, tmem + COL_DQ2, tmem + COL_DP2, dkm + (n % 3) * kStageUnits);
        if (leader) { mma_commit(&sm.bar[QB_DQ]); mma_commit(&sm.bar[QB_K_FREE + n % 3]); }
        if (n + 1 < total) ok = issue_dp(n + 1);
        if (ok && n + 2 < total) ok = issue_s(n + 2);   // its S buffer was read before the DS arrivals of half tile n
      }
      if (!ok && leader) report_device_error(p.status, 820);
    }
  } else {
    setmaxnreg_inc_208();
    const int w = warp >> 2, row = threadIdx.x & 127, q = q0 + row;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tm = tmem + lane_base;
    const float kb2 = a.key_bias ? __ldg(a.key_bias + h) * kLog2e : 0.f;
    float nlse2 = -INFINITY, ndelta = 0.f;   // minus the log-sum-exp (log2 units) and delta
    if (q < a.N) {
      const float lv = __ldg(a.lse + ((int64_t)b * a.Hq + h) * a.N + q);
      nlse2 = lv == -INFINITY ? -INFINITY : -lv * kLog2e;
      ndelta = -__ldg(a.delta + ((int64_t)b * a.Hq + h) * a.N + q);
    }
    float2 acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = both(0.f);
    bool ok = true;
    auto flush = [&](int n) -> bool {
      if (!mbar_wait(&sm.bar[QB_DQ], n & 1)) return false;
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld32(tm + COL_DQ2 + w * 32, r0);
      tmem_ld32(tm + COL_DQ2 + 64 + w * 32, r1);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] = __fadd2_rn(acc[j], halves(r0, r1, j));
      tc_fence_before();
      mbar_arrive(&sm.bar[QB_DQFREE]);
      return true;
    };
    for (int n = 0; n < total && ok; ++n) {
      const uint32_t e = entry[n >> 1];
      const int k0 = (int)(e & 0x7fff) * 128 + (n & 1) * BH;
      uint32_t bits = 0xffffffffu;
      if (e & 0x8000u) {
        uint32_t both[2];
        row_bits64(p.spec, b, h, q, k0, both);
        bits = w == 0 ? both[0] : both[1];
      }
      const float kbase = (float)(p.spec.k_offset + k0 + w * 32);
      ok = mbar_wait(&sm.bar[QB_S + (n & 1)], (n >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      float2 pr[16];
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_S2 + (n & 1) * 128 + w * 32, r0);
        tmem_ld32(tm + COL_S2 + (n & 1) * 128 + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float2 l2 = both(nlse2);
          if constexpr (KB) l2 = __fadd2_rn(l2, make_float2(kb2 * (kbase + (float)(2 * j)), kb2 * (kbase + (float)(2 * j + 1))));
          const float2 t = __ffma2_rn(halves(r0, r1, j), both(p.scale_log2), l2);
          pr[j] = make_float2(ex2(t.x), ex2(t.y));
        }
        if (e & 0x8000u) keep_allowed(pr, bits);
      }
      if (n > 0) ok = flush(n - 1);
      if (ok) ok = mbar_wait(&sm.bar[QB_DP], n & 1);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_DP2 + w * 32, r0);
        tmem_ld32(tm + COL_DP2 + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) pr[j] = __fmul2_rn(pr[j], __fadd2_rn(halves(r0, r1, j), both(ndelta)));
      }
      store_planes32(tm + COL_DP2, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[QB_DS]);
    }
    if (ok && total > 0) ok = flush(total - 1);
    if (ok && total == 0) ok = mbar_wait(&sm.bar[QB_Q], 0);
    float z = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      acc[j] = __fmul2_rn(acc[j], both(a.scale));
      note_finite(z, acc[j].x);
      note_finite(z, acc[j].y);
    }
    if (z != 0.f && parts == 1) sm.not_finite = 1;
    constexpr int kPitch = 68;
    float* stage = reinterpret_cast<float*>(&sm.q[0][0]);   // every MMA that read the Q planes has completed
    if (ok) {
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4*>(stage + row * kPitch + w * 32 + j) = make_float4(acc[j / 2].x, acc[j / 2].y, acc[j / 2 + 1].x, acc[j / 2 + 1].y);
    }
    mbar_arrive(&sm.bar[QB_EPI]);
    ok = mbar_wait(&sm.bar[QB_EPI], 0) && ok;
    if (!ok) report_device_error(p.status, 830 + warp);
    else if (parts == 1) store_rows<256>(stage, kPitch, a.dq, b, q0, a.N, h, a.d, threadIdx.x);
  }
  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    if (warp < 8) sum_rows<64>(reinterpret_cast<const float*>(&sm.q[0][0]), 68, a.dq, b, q0, a.N, h, a.d, parts, part, &sm.not_finite);
    cluster_sync();   // shared memory stays until the others have read it
    if (part > 0) return;
  }
  if (warp < 8 && sm.not_finite) redo_row<REDO_DQ, 4>(reinterpret_cast<float*>(smem_raw), p, qi, h, b);
}

// =================================================================================================================
// Head dimensions 65 - 128, backward.  The planes of two [128 x 128] operands (192 KB) leave no room for the streamed side, so
// of the two resident operands one keeps its planes in shared memory (96 KB) and the other in tensor memory as the A operand
// (192 columns).  Gradients leave through one 64-column accumulator, a chunk of 64 head columns at a time, which the row
// threads add up in registers (warpgroup w: columns [32w, 32w + 32) of every chunk).  The streamed side comes as 64-column
// boxes (three planes, 24 KB).  Bound by the tensor core (24 plane products per block) and the gaps around the single
// accumulator.  Forward and backward, causal, against the FP32 tile kernels: B=2 L=2048 H=16 d=128 9811 -> 1247 us, B=1 L=4096
// 8/2 heads 11504 -> 2279 us, B=2 L=1111 12/3 heads 3327 -> 715 us; 2-norm errors of the gradients against float64
// 2.5e-7 - 4.1e-7 (tile kernels 4.0e-7 - 1.2e-6).
// =================================================================================================================
constexpr uint32_t kBoxPlanes = 3 * kHalfBox;    // one streamed box: hi, mid, lo of [64 rows x 64 columns]
constexpr uint32_t COL_W_S = 0, COL_W_DP = 128, COL_W_ACC = 256, COL_W_A = 320;

// The sums of product_rows<2> with the two streamed boxes wherever they are, and A in shared memory or (A_TMEM) at `a`.
// Descriptors are passed as their low words (address, leading offset); the high word is the same for all of them, and an MMA
// warp that keeps whole descriptors alive over the four products spills registers.
__device__ __forceinline__ uint64_t desc_of(uint32_t low) { return make_smem_desc(0, 0, 1024) + low; }
__device__ __forceinline__ uint32_t desc_low(const void* smem, uint32_t lbo) { return (uint32_t)make_smem_desc(smem_u32(smem), lbo, 1024); }
template <bool A_TMEM>
__device__ __forceinline__ void product_rows_wide(bool leader, uint32_t region, uint32_t a, uint32_t box0, uint32_t box1) {
  asm volatile("" : "+r"(a), "+r"(box0), "+r"(box1));   // keeps the compiler from hoisting 60 sums out of the caller's loop
  if (!leader) return;
  constexpr uint32_t kBPlane = kHalfBox >> 4;
  auto term = [&](int pa, int pb, uint32_t col, uint32_t idesc, bool start) {
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const uint64_t b = desc_of((ks < 4 ? box0 : box1) + pb * kBPlane + (uint32_t)(((ks & 3) * 32) >> 4));
      const uint32_t acc = !(start && ks == 0);
      if constexpr (A_TMEM) mma_ts(region + col, a + pa * 64 + ks * 8, b, idesc, acc);
      else mma_ss(region + col, desc_of(a + (uint32_t)((pa * 2 * kRowBox + (ks >> 2) * kRowBox + (ks & 3) * 32) >> 4)), b, idesc, acc);
    }
  };
  term(2, 0, 0, kIdescN64, true);
  term(0, 2, 64, kIdescN64, true);
  term(1, 0, 0, kIdescN128, false);
  term(0, 0, 0, kIdescN128, false);
}
// region[0, 64) <- P B with the planes of P [128 x 64] in tensor memory at `p` and B one box read MN-major.
__device__ __forceinline__ void product_chunk(bool leader, uint32_t region, uint32_t p, uint32_t box) {
  asm volatile("" : "+r"(p), "+r"(box));
  if (!leader) return;
  constexpr int kTerms[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};   // (plane of P, plane of B)
#pragma unroll
  for (int t = 0; t < 6; ++t)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      mma_ts(region, p + plane_col(kTerms[t][0], ks), desc_of(box + (uint32_t)((kTerms[t][1] * kHalfBox + ks * 2048) >> 4)), kIdescN64T, (t > 0) || (ks > 0));
}
// Planes of this thread's row of an A operand (128 columns) from the workspace into tensor memory, half of the columns per
// warpgroup; rows outside the tensor are zero.
__device__ __forceinline__ void load_planes_tmem(uint32_t tm, int w, const uint8_t* planes, int B, int L, int H, int b, int l, int h) {
#pragma unroll
  for (int pl = 0; pl < 3; ++pl) {
    uint32_t r[32];
    const uint4* src = reinterpret_cast<const uint4*>(planes + ((((int64_t)pl * B + b) * L + l) * H + h) * 256 + w * 128);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint4 v = l < L ? __ldg(src + u) : make_uint4(0u, 0u, 0u, 0u);
      r[4 * u] = v.x; r[4 * u + 1] = v.y; r[4 * u + 2] = v.z; r[4 * u + 3] = v.w;
    }
    tmem_st32(tm + COL_W_A + pl * 64 + w * 32, r);
  }
  tmem_wait_st();
}

struct F32WideParams {
  F32Params f;
  const uint8_t* a_planes;   // planes of V (dK/dV) or dO (dQ) in the workspace
};

// dK / dV, query half tiles of 64.  MMA order per half tile  dV0 dK0 dV1 St(n+1) dK1 dPt(n+1): the box of Q that dK0 frees is
// refilled under dV1, and the exponentials of the next half tile run under its dPt.
enum {
  XB_K = 0, XB_A, XB_S, XB_DP, XB_P, XB_DS, XB_ACC, XB_ACCFREE, XB_EPI, XB_Q_FULL, XB_Q_FREE = XB_Q_FULL + 3, XB_DO_FULL = XB_Q_FREE + 3,
  XB_DO_FREE = XB_DO_FULL + 2, XB_STAT = XB_DO_FREE + 2, XB_STATFREE = XB_STAT + 2, XB_NUM = XB_STATFREE + 2
};
struct __align__(1024) DkdvWideSmem {
  uint8_t k[3][2][kRowBox];
  uint8_t q[3][kBoxPlanes];
  uint8_t d_o[2][kBoxPlanes];
  alignas(16) float nlse2[2][BH], ndelta[2][BH];   // minus the log-sum-exp (log2 units) and delta
  uint64_t bar[XB_NUM];
  uint32_t tmem_base;
  WalkShare share;
  int not_finite;
};
static_assert(dkdv_smem<8>() <= sizeof(DkdvWideSmem), "as above");
constexpr int kWidePitch = 132;
static_assert(2 * BM * kWidePitch * sizeof(float) <= sizeof(uint8_t[3][2][kRowBox]) + 3 * kBoxPlanes, "dV and dK are staged over K and Q");

template <bool KB, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
f32_dkdv_wide_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_qh,
                     const __grid_constant__ CUtensorMap map_do, const __grid_constant__ F32WideParams wp) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  DkdvWideSmem& sm = *reinterpret_cast<DkdvWideSmem*>(smem_raw);
  const F32Params& p = wp.f;
  const bma_attn_args& a = p.a;
  const int parts = SHARED ? p.parts : 1;
  int kj, hk;
  cta_of(p.order, (int)blockIdx.x / parts, kj, hk);
  const int b = hk / a.Hkv, G = a.Hq / a.Hkv;
  hk -= b * a.Hkv;
  const int k0 = kj * BM;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_device_error(p.status, 751);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < XB_NUM; ++i) {
      uint32_t count = 1;
      if (i == XB_A || i == XB_P || i == XB_DS || i == XB_ACCFREE || i == XB_EPI) count = 256;
      if (i == XB_STAT || i == XB_STAT + 1) count = 32;
      mbar_init(&sm.bar[i], count);
    }
    sm.not_finite = 0;
    fence_barrier_init();
    mbar_expect_tx(&sm.bar[XB_K], 6 * kRowBox);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
#pragma unroll
      for (int box = 0; box < 2; ++box) tma_load_4d(sm.k[pl][box], &map_k, &sm.bar[XB_K], box * 64, hk, k0, b + pl * a.B);
    if constexpr (SHARED) sm.share = walk_share(p, b, hk, G, kj);
  }
  if (warp == 8) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp >= 8) {
    setmaxnreg_dec_80();
    HalfIter<SHARED> walk(p.l, b, hk, G, kj, a.N, sm.share);
    int h, q0;
    bool partial, ok = true;
    if (warp == 8 || warp == 11) {
      // ------------------------------------------------------------ Q (warp 8, ring of three boxes) and dO (warp 11, two)
      if (lane == 0) {
        const bool is_q = warp == 8;
        const int slots = is_q ? 3 : 2;
        for (int i = 0; ok && walk.next(h, q0, partial);)
          for (int box = 0; box < 2 && ok; ++box, ++i) {
            const int slot = i % slots;
            uint64_t* full = &sm.bar[(is_q ? XB_Q_FULL : XB_DO_FULL) + slot];
            if (i >= slots) ok = mbar_wait(&sm.bar[(is_q ? XB_Q_FREE : XB_DO_FREE) + slot], (i / slots - 1) & 1);
            if (!ok) break;
            mbar_expect_tx(full, kBoxPlanes);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl)
              tma_load_4d((is_q ? sm.q[slot] : sm.d_o[slot]) + pl * kHalfBox, is_q ? &map_qh : &map_do, full, box * 64, h, q0, b + pl * a.B);
          }
        if (!ok) report_device_error(p.status, 760);
      }
    } else if (warp == 10) {
      // ------------------------------------------------------------ row statistics of the coming half tiles
      for (int n = 0; ok && walk.next(h, q0, partial); ++n) {
        const int st = n & 1;
        if (n >= 2) ok = mbar_wait(&sm.bar[XB_STATFREE + st], ((n >> 1) - 1) & 1);
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int idx = e * 32 + lane, q = q0 + idx;
          const int64_t off = ((int64_t)b * a.Hq + h) * a.N + q;
          const float lv = q < a.N ? __ldg(a.lse + off) : -INFINITY;
          sm.nlse2[st][idx] = (lv == -INFINITY) ? -INFINITY : -lv * kLog2e;   // -inf: the probabilities of the row become exactly 0
          sm.ndelta[st][idx] = q < a.N ? -__ldg(a.delta + off) : 0.f;
        }
        mbar_arrive(&sm.bar[XB_STAT + st]);
      }
      if (!ok && lane == 0) report_device_error(p.status, 765);
    } else {
      // ------------------------------------------------------------ MMA issue
      const bool leader = elect_one();
      const uint32_t dk = desc_low(sm.k, 16);
      const uint32_t dq = desc_low(sm.q, 16), ddo = desc_low(sm.d_o, 16);
      const uint32_t dqm = desc_low(sm.q, kHalfBox), ddom = desc_low(sm.d_o, kHalfBox);
      constexpr uint32_t kBoxUnits = kBoxPlanes >> 4;
      auto issue_st = [&](int n) -> bool {
        const int i0 = 2 * n, i1 = 2 * n + 1;
        if (!mbar_wait(&sm.bar[XB_Q_FULL + i0 % 3], (i0 / 3) & 1) || !mbar_wait(&sm.bar[XB_Q_FULL + i1 % 3], (i1 / 3) & 1)) return false;
        tc_fence_after();
        product_rows_wide<false>(leader, tmem + COL_W_S, dk, dq + (i0 % 3) * kBoxUnits, dq + (i1 % 3) * kBoxUnits);
        if (leader) mma_commit(&sm.bar[XB_S]);
        return true;
      };
      auto issue_dpt = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[XB_DO_FULL], n & 1) || !mbar_wait(&sm.bar[XB_DO_FULL + 1], n & 1)) return false;
        tc_fence_after();
        product_rows_wide<true>(leader, tmem + COL_W_DP, tmem + COL_W_A, ddo, ddo + kBoxUnits);
        if (leader) mma_commit(&sm.bar[XB_DP]);
        return true;
      };
      int chunk = 0;   // chunks issued so far
      auto acc_ready = [&]() -> bool {
        const bool r = chunk == 0 || mbar_wait(&sm.bar[XB_ACCFREE], (chunk - 1) & 1);
        ++chunk;
        tc_fence_after();
        return r;
      };
      bool have = walk.next(h, q0, partial);
      if (have) ok = mbar_wait(&sm.bar[XB_K], 0) && issue_st(0) && mbar_wait(&sm.bar[XB_A], 0) && issue_dpt(0);
      for (int n = 0; have && ok; ++n) {
        const bool more = walk.next(h, q0, partial);
        const int s0 = (2 * n) % 3, s1 = (2 * n + 1) % 3;
        ok = mbar_wait(&sm.bar[XB_P], n & 1) && acc_ready();
        if (!ok) break;
        product_chunk(leader, tmem + COL_W_ACC, tmem + COL_W_S, ddom);
        if (leader) { mma_commit(&sm.bar[XB_ACC]); mma_commit(&sm.bar[XB_DO_FREE]); }
        ok = mbar_wait(&sm.bar[XB_DS], n & 1) && acc_ready();
        if (!ok) break;
        product_chunk(leader, tmem + COL_W_ACC, tmem + COL_W_DP, dqm + s0 * kBoxUnits);
        if (leader) { mma_commit(&sm.bar[XB_ACC]); mma_commit(&sm.bar[XB_Q_FREE + s0]); mma_commit(&sm.bar[XB_STATFREE + (n & 1)]); }
        ok = acc_ready();
        if (!ok) break;
        product_chunk(leader, tmem + COL_W_ACC, tmem + COL_W_S, ddom + kBoxUnits);
        if (leader) { mma_commit(&sm.bar[XB_ACC]); mma_commit(&sm.bar[XB_DO_FREE + 1]); }
        if (more) ok = issue_st(n + 1);
        ok = ok && acc_ready();
        if (!ok) break;
        product_chunk(leader, tmem + COL_W_ACC, tmem + COL_W_DP, dqm + s1 * kBoxUnits);
        if (leader) { mma_commit(&sm.bar[XB_ACC]); mma_commit(&sm.bar[XB_Q_FREE + s1]); }
        if (more) ok = issue_dpt(n + 1);
        have = more;
      }
      if (!ok && leader) report_device_error(p.status, 770);
    }
  } else {
    // -------------------------------------------------------------- row threads
    setmaxnreg_inc_208();
    const int w = warp >> 2, row = threadIdx.x & 127, k = k0 + row;
    const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    load_planes_tmem(tm, w, wp.a_planes, a.B, a.L, a.Hkv, b, k, hk);
    tc_fence_before();
    mbar_arrive(&sm.bar[XB_A]);
    float2 acc[4][16];   // columns [32w, 32w + 32) of dV0, dK0, dV1, dK1 of this key row
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[c][j] = both(0.f);
    bool ok = true;
    HalfIter<SHARED> walk(p.l, b, hk, G, kj, a.N, sm.share);
    int h, q0, n = 0;
    bool partial;
    for (; ok && walk.next(h, q0, partial); ++n) {
      const int st = n & 1;
      const float kbk = KB ? __ldg(a.key_bias + h) * kLog2e * (float)(p.spec.k_offset + k) : 0.f;
      uint32_t bits = 0xffffffffu;
      if (partial) {
        const MaskView mv = make_mask_view(p.spec, b, h);
        int jlo, jhi;
        col_interval(mv, k, q0 + w * 32, 32, jlo, jhi);
        const int lo = max(jlo, 0), hi = min(jhi, 31);
        bits = (lo <= hi) ? ((0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) : 0u;
        if (mv.flags & kTableTerms) bits &= table_bits_col32(mv, k, q0 + w * 32);
      }
      ok = mbar_wait(&sm.bar[XB_STAT + st], (n >> 1) & 1) && mbar_wait(&sm.bar[XB_S], n & 1);
      if (!ok) break;
      tc_fence_after();
      float2 pr[16];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r0[16], r1[16];
        tmem_ld16(tm + COL_W_S + w * 32 + c * 16, r0);
        tmem_ld16(tm + COL_W_S + 64 + w * 32 + c * 16, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float2 l2 = *reinterpret_cast<const float2*>(&sm.nlse2[st][w * 32 + c * 16 + 2 * j]);
          if constexpr (KB) l2 = __fadd2_rn(l2, both(kbk));
          const float2 t = __ffma2_rn(halves(r0, r1, j), both(p.scale_log2), l2);
          pr[c * 8 + j] = make_float2(ex2(t.x), ex2(t.y));
        }
      }
      if (partial) keep_allowed(pr, bits);
      store_planes32(tm + COL_W_S, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[XB_P]);
      ok = mbar_wait(&sm.bar[XB_DP], n & 1);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r0[16], r1[16];
        tmem_ld16(tm + COL_W_DP + w * 32 + c * 16, r0);
        tmem_ld16(tm + COL_W_DP + 64 + w * 32 + c * 16, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          pr[c * 8 + j] = __fmul2_rn(pr[c * 8 + j], __fadd2_rn(halves(r0, r1, j), *reinterpret_cast<const float2*>(&sm.ndelta[st][w * 32 + c * 16 + 2 * j])));
      }
      store_planes32(tm + COL_W_DP, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[XB_DS]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {   // 4 n + c has the parity of c
        if (ok) ok = mbar_wait(&sm.bar[XB_ACC], c & 1);
        if (!ok) break;
        tc_fence_after();
        uint32_t r[32];
        tmem_ld32(tm + COL_W_ACC + w * 32, r);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(&sm.bar[XB_ACCFREE]);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c][j] = __fadd2_rn(acc[c][j], make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])));
      }
    }
    if (ok && n == 0) ok = mbar_wait(&sm.bar[XB_K], 0);   // let the loads land before their buffers are reused
    float z = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (c & 1) acc[c][j] = __fmul2_rn(acc[c][j], both(a.scale));
        note_finite(z, acc[c][j].x);
        note_finite(z, acc[c][j].y);
      }
    if (z != 0.f && parts == 1) sm.not_finite = 1;
    // ---- epilogue: every MMA has completed; dV and dK are staged over the K planes and the Q ring
    mbar_arrive(&sm.bar[XB_EPI]);
    ok = mbar_wait(&sm.bar[XB_EPI], 0) && ok;
    float* stage = reinterpret_cast<float*>(smem_raw);
    if (ok) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float* dst = stage + (c & 1) * BM * kWidePitch + row * kWidePitch + (c >> 1) * 64 + w * 32;
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(dst + j) = make_float4(acc[c][j / 2].x, acc[c][j / 2].y, acc[c][j / 2 + 1].x, acc[c][j / 2 + 1].y);
      }
    }
    mbar_arrive(&sm.bar[XB_EPI]);
    ok = mbar_wait(&sm.bar[XB_EPI], 1) && ok;
    if (!ok) {
      report_device_error(p.status, 780 + warp);
    } else if (parts == 1) {
      store_rows<256>(stage, kWidePitch, a.dv, b, k0, a.L, hk, a.d, threadIdx.x);
      store_rows<256>(stage + BM * kWidePitch, kWidePitch, a.dk, b, k0, a.L, hk, a.d, threadIdx.x);
    }
  }
  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    const int part = (int)blockIdx.x % parts;
    if (warp < 8) {
      const float* stage = reinterpret_cast<const float*>(smem_raw);
#pragma unroll 1
      for (int i = 0; i < 2; ++i)
        sum_rows<128>(stage + i * BM * kWidePitch, kWidePitch, i ? a.dk : a.dv, b, k0, a.L, hk, a.d, parts, part, &sm.not_finite);
    }
    cluster_sync();   // shared memory stays until the others have read it
    if (part > 0) return;
  }
  if (warp < 8 && sm.not_finite) redo_row<REDO_DKDV, 8>(reinterpret_cast<float*>(smem_raw), p, kj, hk, b);
}

// dQ, key half tiles of 64: Q planes in shared memory, dO planes in tensor memory.  MMA order  dQ0 dQ1 S(n+1) dP(n+1).
enum {
  YB_Q = 0, YB_A, YB_S, YB_DP, YB_DS, YB_ACC, YB_ACCFREE, YB_EPI, YB_V_FULL, YB_V_FREE, YB_K_FULL, YB_K_FREE = YB_K_FULL + 3, YB_NUM = YB_K_FREE + 3
};
struct __align__(1024) DqWideSmem {
  uint8_t q[3][2][kRowBox];
  uint8_t k[3][kBoxPlanes];
  uint8_t v[2][kBoxPlanes];
  KvList<kMaxKvBwd> list;
  uint64_t bar[YB_NUM];
  uint32_t tmem_base;
  int not_finite;
};

static_assert(dq_smem<8>() <= sizeof(DqWideSmem), "as above");

template <bool KB, bool SHARED>
__global__ void __launch_bounds__(kThreads, 1)
f32_dq_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kh,
                   const __grid_constant__ CUtensorMap map_vh, const __grid_constant__ F32WideParams wp) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  DqWideSmem& sm = *reinterpret_cast<DqWideSmem*>(smem_raw);
  const F32Params& p = wp.f;
  const bma_attn_args& a = p.a;
  const int parts = SHARED ? p.parts : 1;
  int qi, h;
  cta_of(p.order, (int)blockIdx.x / parts, qi, h);
  qi = p.order.tiles - 1 - qi;
  const int b = h / a.Hq;
  h -= b * a.Hq;
  const int hk = h / (a.Hq / a.Hkv);
  const int q0 = qi * BM;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_device_error(p.status, 851);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < YB_NUM; ++i) mbar_init(&sm.bar[i], (i == YB_A || i == YB_DS || i == YB_ACCFREE || i == YB_EPI) ? 256 : 1);
    sm.not_finite = 0;
    fence_barrier_init();
    mbar_expect_tx(&sm.bar[YB_Q], 6 * kRowBox);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
#pragma unroll
      for (int box = 0; box < 2; ++box) tma_load_4d(sm.q[pl][box], &map_q, &sm.bar[YB_Q], box * 64, h, q0, b + pl * a.B);
  }
  if (warp == 8) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  const int listed = build_kv_list(sm.list, p.l, p.spec, b, h, qi);
  const int part = (int)blockIdx.x % parts, t0 = listed * part / parts, T = listed * (part + 1) / parts - t0;   // this CTA's part of the list
  const uint16_t* entry = sm.list.entry + t0;
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  // half tiles in all; the second half of the last tile may lie past the end of the keys
  const int total = T == 0 ? 0 : 2 * T - ((int)(entry[T - 1] & 0x7fff) * 128 + BH >= a.L ? 1 : 0);

  if (warp >= 8) {
    setmaxnreg_dec_80();
    bool ok = true;
    if (warp == 8 && lane == 0) {
      // ------------------------------------------------------------ K: ring of three boxes
      for (int i = 0; i < 2 * total && ok; ++i) {
        const int slot = i % 3, n = i >> 1;
        if (i >= 3) ok = mbar_wait(&sm.bar[YB_K_FREE + slot], (i / 3 - 1) & 1);
        if (!ok) break;
        const int r0 = (int)(entry[n >> 1] & 0x7fff) * 128 + (n & 1) * BH;
        mbar_expect_tx(&sm.bar[YB_K_FULL + slot], kBoxPlanes);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
          tma_load_4d(sm.k[slot] + pl * kHalfBox, &map_kh, &sm.bar[YB_K_FULL + slot], (i & 1) * 64, hk, r0, b + pl * a.B);
      }
      if (!ok) report_device_error(p.status, 860);
    } else if (warp == 10 && lane == 0) {
      // ------------------------------------------------------------ V: both boxes, one stage
      for (int n = 0; n < total && ok; ++n) {
        if (n >= 1) ok = mbar_wait(&sm.bar[YB_V_FREE], (n - 1) & 1);
        if (!ok) break;
        const int r0 = (int)(entry[n >> 1] & 0x7fff) * 128 + (n & 1) * BH;
        mbar_expect_tx(&sm.bar[YB_V_FULL], 2 * kBoxPlanes);
#pragma unroll
        for (int box = 0; box < 2; ++box)
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) tma_load_4d(sm.v[box] + pl * kHalfBox, &map_vh, &sm.bar[YB_V_FULL], box * 64, hk, r0, b + pl * a.B);
      }
      if (!ok) report_device_error(p.status, 862);
    } else if (warp == 9 && total > 0) {
      // ------------------------------------------------------------ MMA issue
      const bool leader = elect_one();
      const uint32_t dq = desc_low(sm.q, 16);
      const uint32_t dk = desc_low(sm.k, 16), dv = desc_low(sm.v, 16);
      const uint32_t dkm = desc_low(sm.k, kHalfBox);
      constexpr uint32_t kBoxUnits = kBoxPlanes >> 4;
      auto issue_s = [&](int n) -> bool {
        const int i0 = 2 * n, i1 = 2 * n + 1;
        if (!mbar_wait(&sm.bar[YB_K_FULL + i0 % 3], (i0 / 3) & 1) || !mbar_wait(&sm.bar[YB_K_FULL + i1 % 3], (i1 / 3) & 1)) return false;
        tc_fence_after();
        product_rows_wide<false>(leader, tmem + COL_W_S, dq, dk + (i0 % 3) * kBoxUnits, dk + (i1 % 3) * kBoxUnits);
        if (leader) mma_commit(&sm.bar[YB_S]);
        return true;
      };
      auto issue_dp = [&](int n) -> bool {
        if (!mbar_wait(&sm.bar[YB_V_FULL], n & 1)) return false;
        tc_fence_after();
        product_rows_wide<true>(leader, tmem + COL_W_DP, tmem + COL_W_A, dv, dv + kBoxUnits);
        if (leader) { mma_commit(&sm.bar[YB_DP]); mma_commit(&sm.bar[YB_V_FREE]); }
        return true;
      };
      ok = mbar_wait(&sm.bar[YB_Q], 0) && issue_s(0) && mbar_wait(&sm.bar[YB_A], 0) && issue_dp(0);
      for (int n = 0; n < total && ok; ++n) {
        ok = mbar_wait(&sm.bar[YB_DS], n & 1);
#pragma unroll
        for (int c = 0; c < 2 && ok; ++c) {
          if (2 * n + c > 0) ok = mbar_wait(&sm.bar[YB_ACCFREE], (2 * n + c - 1) & 1);
          if (!ok) break;
          tc_fence_after();
          const int slot = (2 * n + c) % 3;
          product_chunk(leader, tmem + COL_W_ACC, tmem + COL_W_DP, dkm + slot * kBoxUnits);
          if (leader) { mma_commit(&sm.bar[YB_ACC]); mma_commit(&sm.bar[YB_K_FREE + slot]); }
        }
        if (ok && n + 1 < total) ok = issue_s(n + 1) && issue_dp(n + 1);   // S(n) was read before the DS arrivals of half tile n
      }
      if (!ok && leader) report_device_error(p.status, 870);
    }
  } else {
    setmaxnreg_inc_208();
    const int w = warp >> 2, row = threadIdx.x & 127, q = q0 + row;
    const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    load_planes_tmem(tm, w, wp.a_planes, a.B, a.N, a.Hq, b, q, h);
    tc_fence_before();
    mbar_arrive(&sm.bar[YB_A]);
    const float kb2 = a.key_bias ? __ldg(a.key_bias + h) * kLog2e : 0.f;
    float nlse2 = -INFINITY, ndelta = 0.f;   // minus the log-sum-exp (log2 units) and delta
    if (q < a.N) {
      const float lv = __ldg(a.lse + ((int64_t)b * a.Hq + h) * a.N + q);
      nlse2 = lv == -INFINITY ? -INFINITY : -lv * kLog2e;
      ndelta = -__ldg(a.delta + ((int64_t)b * a.Hq + h) * a.N + q);
    }
    float2 acc[2][16];   // columns [32w, 32w + 32) of the two chunks of dQ of this row
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[c][j] = both(0.f);
    bool ok = true;
    for (int n = 0; n < total && ok; ++n) {
      const uint32_t e = entry[n >> 1];
      const int k0 = (int)(e & 0x7fff) * 128 + (n & 1) * BH;
      uint32_t bits = 0xffffffffu;
      if (e & 0x8000u) {
        uint32_t both[2];
        row_bits64(p.spec, b, h, q, k0, both);
        bits = w == 0 ? both[0] : both[1];
      }
      const float kbase = (float)(p.spec.k_offset + k0 + w * 32);
      ok = mbar_wait(&sm.bar[YB_S], n & 1);
      if (!ok) break;
      tc_fence_after();
      float2 pr[16];
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_W_S + w * 32, r0);
        tmem_ld32(tm + COL_W_S + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float2 l2 = both(nlse2);
          if constexpr (KB) l2 = __fadd2_rn(l2, make_float2(kb2 * (kbase + (float)(2 * j)), kb2 * (kbase + (float)(2 * j + 1))));
          const float2 t = __ffma2_rn(halves(r0, r1, j), both(p.scale_log2), l2);
          pr[j] = make_float2(ex2(t.x), ex2(t.y));
        }
        if (e & 0x8000u) keep_allowed(pr, bits);
      }
      ok = mbar_wait(&sm.bar[YB_DP], n & 1);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tm + COL_W_DP + w * 32, r0);
        tmem_ld32(tm + COL_W_DP + 64 + w * 32, r1);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) pr[j] = __fmul2_rn(pr[j], __fadd2_rn(halves(r0, r1, j), both(ndelta)));
      }
      store_planes32(tm + COL_W_DP, w * 2, pr);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[YB_DS]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (ok) ok = mbar_wait(&sm.bar[YB_ACC], c);   // chunk 2 n + c
        if (!ok) break;
        tc_fence_after();
        uint32_t r[32];
        tmem_ld32(tm + COL_W_ACC + w * 32, r);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(&sm.bar[YB_ACCFREE]);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c][j] = __fadd2_rn(acc[c][j], make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])));
      }
    }
    if (ok && total == 0) ok = mbar_wait(&sm.bar[YB_Q], 0);
    float z = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        acc[c][j] = __fmul2_rn(acc[c][j], both(a.scale));
        note_finite(z, acc[c][j].x);
        note_finite(z, acc[c][j].y);
      }
    if (z != 0.f && parts == 1) sm.not_finite = 1;
    // every thread has seen the last chunk, so every MMA that read the Q planes has completed
    mbar_arrive(&sm.bar[YB_EPI]);
    ok = mbar_wait(&sm.bar[YB_EPI], 0) && ok;
    float* stage = reinterpret_cast<float*>(&sm.q[0][0][0]);
    if (ok) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(stage + row * kWidePitch + c * 64 + w * 32 + j) =
              make_float4(acc[c][j / 2].x, acc[c][j / 2].y, acc[c][j / 2 + 1].x, acc[c][j / 2 + 1].y);
    }
    mbar_arrive(&sm.bar[YB_EPI]);
    ok = mbar_wait(&sm.bar[YB_EPI], 1) && ok;
    if (!ok) report_device_error(p.status, 880 + warp);
    else if (parts == 1) store_rows<256>(stage, kWidePitch, a.dq, b, q0, a.N, h, a.d, threadIdx.x);
  }
  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    if (warp < 8) sum_rows<128>(reinterpret_cast<const float*>(&sm.q[0][0][0]), kWidePitch, a.dq, b, q0, a.N, h, a.d, parts, part, &sm.not_finite);
    cluster_sync();   // shared memory stays until the others have read it
    if (part > 0) return;
  }
  if (warp < 8 && sm.not_finite) redo_row<REDO_DQ, 8>(reinterpret_cast<float*>(smem_raw), p, qi, h, b);
}

// ---- host ------------------------------------------------------------------------------------------------------
int padded_d(const bma_attn_args& a) { return a.d <= 64 ? 64 : 128; }
size_t plane_bytes(int B, int L, int H, int dp) { return (size_t)3 * B * L * H * dp * 2; }
size_t align_up(size_t x) { return (x + 1023) / 1024 * 1024; }

struct Planes {
  size_t q, k, v, d_o, used, lists, total;   // offsets in the workspace: planes, marks of listed blocks, block lists (backward)
};
// Few queries against many keys may see a small part of them: then only the planes of listed kv blocks are made.  (What the
// other blocks' planes hold is read by the dK / dV kernel alone, as the resident operand of a CTA that has no query tile.)
// Marking takes a launch (2 us), the planes of 4M values of K and V as much; with more query tiles than a quarter of the kv
// blocks, the other kernels take far longer than the planes.  (16 queries that see 512 of 65536 keys, B = 4, 16/4 heads of 64,
// the whole call: 247 us with all planes, 64 with the listed ones.)
bool used_blocks(const bma_attn_args& a) {
  return 4 * ceil_div(a.N, BM) <= ceil_div(a.L, BM) && (int64_t)a.B * a.L * a.Hkv * a.d >= (1 << 22);
}
Planes planes_layout(const bma_attn_args& a, bool backward) {
  const int dp = padded_d(a);
  Planes p;
  p.q = 0;
  p.k = align_up(plane_bytes(a.B, a.N, a.Hq, dp));
  p.v = p.k + align_up(plane_bytes(a.B, a.L, a.Hkv, dp));
  p.d_o = p.v + align_up(plane_bytes(a.B, a.L, a.Hkv, dp));
  p.used = p.d_o + (backward ? align_up(plane_bytes(a.B, a.N, a.Hq, dp)) : 0);
  p.lists = p.used + (used_blocks(a) ? align_up((size_t)a.B * ceil_div(a.L, BM)) : 0);
  const size_t NQ = ceil_div(a.N, BM), NKV = ceil_div(a.L, BM);
  p.total = p.lists + (backward ? align_up(sizeof(int32_t) * (2 * (NQ + NKV) + 4 * NQ * NKV)) : 0);
  return p;
}
// The arrays of lists that the pass writes itself
bma_block_lists own_lists(const bma_block_lists& sizes, uint8_t* at) {
  bma_block_lists l = sizes;
  int32_t* p = reinterpret_cast<int32_t*>(at);
  auto take = [&](int64_t n) { int32_t* r = p; p += n; return r; };
  const int64_t cells = (int64_t)l.NQ * l.NKV;
  l.kv_num = take(l.NQ); l.full_kv_num = take(l.NQ); l.q_num = take(l.NKV); l.full_q_num = take(l.NKV);
  l.kv_idx = take(cells); l.full_kv_idx = take(cells); l.q_idx = take(cells); l.full_q_idx = take(cells);
  return l;
}

int launch_split(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& l, const Planes& pl, uint8_t* ws, bool backward, bool own_delta,
                 cudaStream_t st) {
  SplitParams sp;
  const bool lists_wanted = backward && !l.kv_num;
  sp.o = a.o;
  sp.delta = own_delta ? a.delta : nullptr;
  sp.jobs = backward ? 4 : 3;
  sp.lists = lists_wanted ? own_lists(l, ws + pl.lists) : l;
  sp.spec = spec;
  sp.B = a.B; sp.d = a.d;
  sp.used = nullptr; sp.used_B = l.B; sp.NKV = l.NKV;
  if (used_blocks(a)) {
    used_blocks_kernel<<<(unsigned)l.B, 256, 0, st>>>(l, spec, backward, ws + pl.used);
    count_launches(1);
    sp.used = ws + pl.used;
  }
  sp.job[0] = {a.q, ws + pl.q, a.N, a.Hq};
  sp.job[1] = {a.k, ws + pl.k, a.L, a.Hkv};
  sp.job[2] = {a.v, ws + pl.v, a.L, a.Hkv};
  sp.job[3] = {a.d_o, ws + pl.d_o, a.N, a.Hq};
  const int dp = padded_d(a);
  const int64_t most = std::max((int64_t)a.B * a.N * a.Hq, (int64_t)a.B * a.L * a.Hkv) * (dp / 8);
  const dim3 grid((unsigned)std::min<int64_t>((most + 255) / 256, 148 * 8), sp.jobs + (lists_wanted ? 1 : 0));
  if (dp == 64) split_kernel<64><<<grid, 256, 0, st>>>(sp);
  else split_kernel<128><<<grid, 256, 0, st>>>(sp);
  count_launches(1);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

int plane_map(CUtensorMap* m, const uint8_t* base, int B, int L, int H, int dp, int rows) {
  return make_tile_map_bf16(m, base, 3 * B, L, H, dp, (int64_t)L * H * dp, (int64_t)H * dp, dp, rows);
}

// CTAs by query tile (streaming the planes of K and V), by key tile (those of Q and dO of a head group)
LaunchOrder q_order(const bma_attn_args& a, int dp) { return launch_order(ceil_div(a.N, BM), (int64_t)a.B * a.Hq, (int64_t)12 * a.L * dp * a.Hkv / a.Hq); }
LaunchOrder k_order(const bma_attn_args& a, int dp) { return launch_order(ceil_div(a.L, BM), (int64_t)a.B * a.Hkv, (int64_t)12 * a.N * dp * (a.Hq / a.Hkv)); }

int make_params(F32Params& p, const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists) {
  p.a = a; p.spec = spec; p.l = lists;
  p.parts = 1; p.first = 0;
  p.scale_log2 = a.scale * kLog2e;
  p.status = device_status_ptr();
  BMA_REQUIRE(p.status != nullptr, BMA_ERR_CUDA);
  return BMA_OK;
}

cudaLaunchConfig_t f32_fwd_config(int tiles, int parts, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * parts));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  return cfg;
}
// Clusters of `parts` CTAs of the forward kernel that the device runs at the same time.
bool f32_fwd_kb(const bma_attn_args& a) { return a.key_bias || !(a.scale > 0.f); }
int f32_fwd_clusters(const bma_attn_args& a, int dp, int parts) {
  static ClusterCounts known[2][2];
  const bool kb = f32_fwd_kb(a);
  ClusterCounts& k = known[dp == 128][kb];
  if (dp == 128) return clusters_at_once(k, kb ? f32_fwd_kernel<128, true, true> : f32_fwd_kernel<128, false, true>, kThreads, sizeof(FwdSmem<128>), parts);
  return clusters_at_once(k, kb ? f32_fwd_kernel<64, true, true> : f32_fwd_kernel<64, false, true>, kThreads, sizeof(FwdSmem<64>), parts);
}

// How many CTAs share a tile's key list: `parts` in one launch of all tiles, or, where every tile takes as long, 1 for whole waves of
// tiles and `last_parts` for the `last` ones, in a launch of their own (which costs short walks more than it gives).  Launches of up to four waves leave SMs without work: too
// few tiles, a last wave of a few, or a causal mask whose longest walk takes longer than the average SM's share.  The model counts key tiles:
// a walk of w tiles takes w / parts + 3, the three for set-up, merge and the partials' way through shared memory (a CTA takes 8 - 14 us
// besides its tiles of 3.1 us at 64 head columns, 4.8 at 128).  Calls: 1 x 1500 tokens, 16/4 heads of 128, no mask, 148 + 44 tiles in 3
// parts 147 -> 116 us; causal 1 x 1000, 8 heads of 64 76 -> 44, 1 x 4096,
// 4 heads of 128 169 -> 116 (of which about 30 and 15 are the lists' launch and the host path).
struct FwdShare {
  int parts, last, last_parts;
};
// CTAs that share a walk of a backward pass, likewise, with float32 accumulators to add up.  (Calls, forward and backward, causal: 1 x 1423, 4/1
// heads of 128 750 -> 195 us, 1 x 4096, 8/2 heads of 128 2220 -> 805, 1 x 4096, 4 heads of 64 404 -> 280, 1 x 3000, 16/4 heads of 64 823 -> 538;
// forward, host path and launch order included.  The shared kernels are instances of their own: the part of a walk costs the plain dK / dV
// kernel 7 % in registers, 173 -> 186 us on 2 x 2048 tokens of 16 heads of 64.)
template <typename K>
int f32_bwd_parts(const Walks& w, int64_t ctas, ClusterCounts& known, K kernel, size_t smem) {
  if (ctas > 4 * kSms) return 1;
  return share_walks(w, 3.0, (int)std::max(1.0, w.longest), [&](int parts) { return clusters_at_once(known, kernel, kThreads, smem, parts); });
}

FwdShare f32_fwd_share(const bma_attn_args& a, const bma_mask_spec& spec, int dp, int NQ, int NKV) {
  FwdShare best{1, 0, 1};
  if ((int64_t)NQ * a.B * a.Hq > 4 * kSms || NKV < 2) return best;
  const Walks w = q_walks(a, spec);
  const int tiles = w.ctas;
  const double o = 3., longest = w.longest;
  auto even = [&](int count, int parts, int clusters) { return (double)ceil_div(count, clusters) * (longest / parts + o); };
  best.parts = share_walks(w, o, NKV, [&](int parts) { return f32_fwd_clusters(a, dp, parts); });
  double cost = even(tiles, best.parts, f32_fwd_clusters(a, dp, best.parts));
  const int sms = device_sms(current_device()), last = tiles % sms;
  if (w.even && w.known && tiles > sms && last > 0)
    for (int parts = 2; parts <= std::min(kMaxParts, NKV); ++parts) {
      const int clusters = f32_fwd_clusters(a, dp, parts);
      if (clusters < last) continue;
      const double c = even(tiles - last, 1, sms) + even(last, parts, clusters);
      if (c < 0.95 * cost) { cost = c; best = {1, last, parts}; }
    }
  return best;
}

}  // namespace

size_t f32_workspace_bytes(const bma_attn_args& a, bool backward) {
  if (a.q.dtype != BMA_DTYPE_F32 || !sm100_device()) return 0;
  if (a.d > 128 || ceil_div(a.L, BM) > (backward ? kMaxKvBwd : kMaxKvFwd)) return 0;
  return planes_layout(a, backward).total;
}

int f32_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws, cudaStream_t st) {
  const Planes pl = planes_layout(a, false);
  uint8_t* w = static_cast<uint8_t*>(ws);
  const int dp = padded_d(a);
  F32Params p;
  int rc;
  if ((rc = make_params(p, a, spec, lists)) || (rc = launch_split(a, spec, lists, pl, w, false, false, st))) return rc;
  CUtensorMap mq, mk, mv;
  if ((rc = plane_map(&mq, w + pl.q, a.B, a.N, a.Hq, dp, BM)) || (rc = plane_map(&mk, w + pl.k, a.B, a.L, a.Hkv, dp, BH)) ||
      (rc = plane_map(&mv, w + pl.v, a.B, a.L, a.Hkv, dp, BH)))
    return rc;
  p.order = q_order(a, dp);
  auto launch = [&](auto plain, auto shared, size_t smem) -> int {
    const int items = (int)launch_ctas(p.order);
    auto run = [&](int first, int count, int parts) -> int {
      const auto kernel = parts > 1 ? shared : plain;
      BMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      p.parts = parts; p.first = first;
      cudaLaunchConfig_t cfg = f32_fwd_config(count, parts, smem, st);
      cudaLaunchAttribute attr = cluster_attribute(parts);
      if (parts > 1) { cfg.attrs = &attr; cfg.numAttrs = 1; }
      BMA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, mq, mk, mv, p));
      count_launches(1, parts);
      return BMA_OK;
    };
    const FwdShare share = f32_fwd_share(a, spec, dp, lists.NQ, lists.NKV);
    const int r = run(0, items - share.last, share.parts);
    return r || !share.last ? r : run(items - share.last, share.last, share.last_parts);
  };
  if (f32_fwd_kb(a)) rc = dp == 64 ? launch(f32_fwd_kernel<64, true, false>, f32_fwd_kernel<64, true, true>, sizeof(FwdSmem<64>))
                                                   : launch(f32_fwd_kernel<128, true, false>, f32_fwd_kernel<128, true, true>, sizeof(FwdSmem<128>));
  else rc = dp == 64 ? launch(f32_fwd_kernel<64, false, false>, f32_fwd_kernel<64, false, true>, sizeof(FwdSmem<64>))
                     : launch(f32_fwd_kernel<128, false, false>, f32_fwd_kernel<128, false, true>, sizeof(FwdSmem<128>));
  if (rc) return rc;
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

int f32_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& given, void* ws, bool own_delta, cudaStream_t st) {
  const Planes pl = planes_layout(a, true);
  uint8_t* w = static_cast<uint8_t*>(ws);
  const bma_block_lists lists = given.kv_num ? given : own_lists(given, w + pl.lists);
  F32Params p;
  int rc;
  if ((rc = make_params(p, a, spec, lists)) || (rc = launch_split(a, spec, given, pl, w, true, own_delta, st))) return rc;
  CUtensorMap mq, mk, mv, mdo, mqh, mkh, mvh, mdoh;
  static ClusterCounts known[4][2];
  const int kb = a.key_bias != nullptr;
  const int64_t k_ctas = (int64_t)lists.NKV * a.B * a.Hkv, q_ctas = (int64_t)lists.NQ * a.B * a.Hq;
  const bool few = std::min(k_ctas, q_ctas) <= 4 * kSms;
  const Walks kw = few ? k_walks(a, spec) : Walks{}, qw = few ? q_walks(a, spec) : Walks{};
  auto launch = [&](auto kernel, const LaunchOrder& order, int parts, size_t smem, auto... args) -> int {
    BMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(launch_ctas(order) * parts);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = cluster_attribute(parts);
    if (parts > 1) { cfg.attrs = &attr; cfg.numAttrs = 1; }
    BMA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    count_launches(1, parts);
    return BMA_OK;
  };
  if (a.d > 64) {
    if ((rc = plane_map(&mq, w + pl.q, a.B, a.N, a.Hq, 128, BM)) || (rc = plane_map(&mk, w + pl.k, a.B, a.L, a.Hkv, 128, BM)) ||
        (rc = plane_map(&mqh, w + pl.q, a.B, a.N, a.Hq, 128, BH)) || (rc = plane_map(&mkh, w + pl.k, a.B, a.L, a.Hkv, 128, BH)) ||
        (rc = plane_map(&mvh, w + pl.v, a.B, a.L, a.Hkv, 128, BH)) || (rc = plane_map(&mdoh, w + pl.d_o, a.B, a.N, a.Hq, 128, BH)))
      return rc;
    auto dkdv = a.key_bias ? f32_dkdv_wide_kernel<true, false> : f32_dkdv_wide_kernel<false, false>;
    auto dkdv_shared = a.key_bias ? f32_dkdv_wide_kernel<true, true> : f32_dkdv_wide_kernel<false, true>;
    auto dq = a.key_bias ? f32_dq_wide_kernel<true, false> : f32_dq_wide_kernel<false, false>;
    auto dq_shared = a.key_bias ? f32_dq_wide_kernel<true, true> : f32_dq_wide_kernel<false, true>;
    F32WideParams wp{p, w + pl.v};
    wp.f.order = k_order(a, 128);
    wp.f.parts = f32_bwd_parts(kw, k_ctas, known[0][kb], dkdv_shared, sizeof(DkdvWideSmem));
    if ((rc = launch(wp.f.parts > 1 ? dkdv_shared : dkdv, wp.f.order, wp.f.parts, sizeof(DkdvWideSmem), mk, mqh, mdoh, wp))) return rc;
    wp.a_planes = w + pl.d_o;
    wp.f.order = q_order(a, 128);
    wp.f.parts = f32_bwd_parts(qw, q_ctas, known[1][kb], dq_shared, sizeof(DqWideSmem));
    return launch(wp.f.parts > 1 ? dq_shared : dq, wp.f.order, wp.f.parts, sizeof(DqWideSmem), mq, mkh, mvh, wp);
  }
  if ((rc = plane_map(&mq, w + pl.q, a.B, a.N, a.Hq, 64, BM)) || (rc = plane_map(&mk, w + pl.k, a.B, a.L, a.Hkv, 64, BM)) ||
      (rc = plane_map(&mv, w + pl.v, a.B, a.L, a.Hkv, 64, BM)) || (rc = plane_map(&mdo, w + pl.d_o, a.B, a.N, a.Hq, 64, BM)) ||
      (rc = plane_map(&mqh, w + pl.q, a.B, a.N, a.Hq, 64, BH)) || (rc = plane_map(&mkh, w + pl.k, a.B, a.L, a.Hkv, 64, BH)) ||
      (rc = plane_map(&mvh, w + pl.v, a.B, a.L, a.Hkv, 64, BH)) || (rc = plane_map(&mdoh, w + pl.d_o, a.B, a.N, a.Hq, 64, BH)))
    return rc;
  auto dkdv = a.key_bias ? f32_dkdv_kernel<true, false> : f32_dkdv_kernel<false, false>;
  auto dkdv_shared = a.key_bias ? f32_dkdv_kernel<true, true> : f32_dkdv_kernel<false, true>;
  auto dq = a.key_bias ? f32_dq_kernel<true, false> : f32_dq_kernel<false, false>;
  auto dq_shared = a.key_bias ? f32_dq_kernel<true, true> : f32_dq_kernel<false, true>;
  p.order = k_order(a, 64);
  p.parts = f32_bwd_parts(kw, k_ctas, known[2][kb], dkdv_shared, sizeof(DkdvSmem));
  if ((rc = launch(p.parts > 1 ? dkdv_shared : dkdv, p.order, p.parts, sizeof(DkdvSmem), mk, mv, mqh, mdoh, p))) return rc;
  p.order = q_order(a, 64);
  p.parts = f32_bwd_parts(qw, q_ctas, known[3][kb], dq_shared, sizeof(DqSmem));
  return launch(p.parts > 1 ? dq_shared : dq, p.order, p.parts, sizeof(DqSmem), mq, mkh, mvh, mdo, p);
}

}  // namespace bma
