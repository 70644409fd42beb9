// FP32 SIMT attention kernels (forward, dK/dV, dQ) driven by the block lists.
//
// These cover what the tensor-core kernels do not: bfloat16 head dims other than 64 and 128, float32
// sequences beyond the lengths of attn_f32_sm100.cu, tiles of those kernels whose result is not finite (the
// bf16 planes of an infinity are not numbers), and a forced backend -- as the exact-arithmetic
// cross-check of the tensor-core paths.  All arithmetic is FP32 FMA; inputs may be float32 or bfloat16
// and are widened when a tile is staged.
//
// Semantics follow jaxmodules/attention.py:52-105 (scores exp(q.k/sqrt(d)) times mask, rows
// without an allowed key give 0) with a max-subtracted online softmax, which is the same
// function.  Empty blocks are never visited, full blocks skip the element predicate.
//
// Tile: 64 queries x 64 keys per CTA of 256 threads; thread (ty, tx) = (tid/16, tid%16) owns
// score rows 4*ty..4*ty+3, score columns 4*tx..4*tx+3, and output columns tx + 16*c.
#include <algorithm>

#include "simt_tiles.cuh"

namespace bma {
namespace {

template <typename T, int DC, bool WIDE>
__global__ void __launch_bounds__(NT) simt_fwd_kernel(const SimtParams p) {
  extern __shared__ __align__(16) float sm[];
  fwd_tile<T, DC, WIDE, CtaSync>(sm, p, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <typename T, typename TDO, int DC, bool WIDE>
__global__ void __launch_bounds__(NT) simt_bwd_dkdv_kernel(const SimtParams p) {
  extern __shared__ __align__(16) float sm[];
  dkdv_tile<T, TDO, DC, WIDE, CtaSync>(sm, p, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <typename T, typename TDO, int DC, bool WIDE>
__global__ void __launch_bounds__(NT) simt_bwd_dq_kernel(const SimtParams p) {
  extern __shared__ __align__(16) float sm[];
  dq_tile<T, TDO, DC, WIDE, CtaSync>(sm, p, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <typename K>
int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) BMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return BMA_OK;
}

template <typename T, int DC, bool WIDE>
int launch_fwd(const SimtParams& p, cudaStream_t st) {
  int rc = set_smem(simt_fwd_kernel<T, DC, WIDE>, fwd_smem<DC>());
  if (rc) return rc;
  dim3 grid(ceil_div(p.a.N, TQ), p.a.Hq, p.a.B);
  simt_fwd_kernel<T, DC, WIDE><<<grid, NT, fwd_smem<DC>(), st>>>(p);
  count_launches(1);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

template <typename T, typename TDO, int DC, bool WIDE>
int launch_bwd(const SimtParams& p, cudaStream_t st) {
  int rc = set_smem(simt_bwd_dkdv_kernel<T, TDO, DC, WIDE>, dkdv_smem<DC>());
  if (rc) return rc;
  rc = set_smem(simt_bwd_dq_kernel<T, TDO, DC, WIDE>, dq_smem<DC>());
  if (rc) return rc;
  dim3 gkv(ceil_div(p.a.L, TK), p.a.Hkv, p.a.B);
  simt_bwd_dkdv_kernel<T, TDO, DC, WIDE><<<gkv, NT, dkdv_smem<DC>(), st>>>(p);
  dim3 gq(ceil_div(p.a.N, TQ), p.a.Hq, p.a.B);
  simt_bwd_dq_kernel<T, TDO, DC, WIDE><<<gq, NT, dq_smem<DC>(), st>>>(p);
  count_launches(2);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

template <typename T, bool WIDE>
int dispatch_fwd(const SimtParams& p, cudaStream_t st) {
  const int d = p.a.d;
  if (d <= 16) return launch_fwd<T, 1, WIDE>(p, st);
  if (d <= 32) return launch_fwd<T, 2, WIDE>(p, st);
  if (d <= 64) return launch_fwd<T, 4, WIDE>(p, st);
  if (d <= 128) return launch_fwd<T, 8, WIDE>(p, st);
  return BMA_ERR_UNSUPPORTED;
}
template <typename T, typename TDO, bool WIDE>
int dispatch_bwd(const SimtParams& p, cudaStream_t st) {
  const int d = p.a.d;
  if (d <= 16) return launch_bwd<T, TDO, 1, WIDE>(p, st);
  if (d <= 32) return launch_bwd<T, TDO, 2, WIDE>(p, st);
  if (d <= 64) return launch_bwd<T, TDO, 4, WIDE>(p, st);
  if (d <= 128) return launch_bwd<T, TDO, 8, WIDE>(p, st);
  return BMA_ERR_UNSUPPORTED;
}

}  // namespace

int simt_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st) {
  BMA_REQUIRE(lists.q_block == TQ && lists.kv_block == TK, BMA_ERR_ARG);
  const SimtParams p = simt_params(a, spec, lists);
  if (a.q.dtype == BMA_DTYPE_F32) return dispatch_fwd<float, false>(p, st);
  return dispatch_fwd<__nv_bfloat16, false>(p, st);
}

int simt_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st) {
  BMA_REQUIRE(lists.q_block == TQ && lists.kv_block == TK && lists.q_num, BMA_ERR_ARG);
  const SimtParams p = simt_params(a, spec, lists);
  const bool f32 = a.q.dtype == BMA_DTYPE_F32, do_f32 = a.d_o.dtype == BMA_DTYPE_F32;
  if (f32 && do_f32) return dispatch_bwd<float, float, false>(p, st);
  if (f32) return dispatch_bwd<float, __nv_bfloat16, false>(p, st);
  if (do_f32) return dispatch_bwd<__nv_bfloat16, float, false>(p, st);
  return dispatch_bwd<__nv_bfloat16, __nv_bfloat16, false>(p, st);
}

int simt_wide_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st) {
  return dispatch_fwd<float, true>(simt_params(a, spec, lists), st);
}

int simt_wide_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st) {
  const SimtParams p = simt_params(a, spec, lists);
  return a.d_o.dtype == BMA_DTYPE_F32 ? dispatch_bwd<float, float, true>(p, st) : dispatch_bwd<float, __nv_bfloat16, true>(p, st);
}

}  // namespace bma
