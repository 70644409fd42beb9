// Compact addressing of the backward scratch (the bf16 dS tiles that the dK/dV kernel hands to the dQ replay
// kernel): one 32 KB slot per VISITED block instead of one per block of the dense [B, Hq, NQ, NKV] grid.
//
//   slot(b, h, qi, kj) = head_base[b * Hq + h] + row_base[b', h', qi] + rank[b', h', qi, kj]
//
// with (b', h') the list head that (b, h) reads (the lists broadcast over B and / or H), rank = the number of
// visited kv tiles of row qi below kj (the order in which the query-major replay kernel walks the row, so it
// needs no table: its running count IS the rank), row_base = exclusive prefix of the row counts inside a list
// head, head_base = exclusive prefix over (b, h) in row-major order of the list heads' totals.  A launch over a
// range of (batch, head) units subtracts the head_base of its first head.
//
// One small launch per backward call (two with many list heads) builds the tables from the kv-side lists into the front of the caller's workspace.
#include <algorithm>

#include "bwd_preprocess.cuh"
#include "common.cuh"

namespace bma {

namespace {

constexpr int kMaxKvTilesBwd = 1024;  // the tensor-core backward takes L <= 131072
// List heads up to which one launch builds all tables: eight warps take four heads each then, about as long as a second
// launch.  (2048 heads of two rows, B = 32, H = 64, N = 256, forward and backward: 775 us with one launch, 689 with two.)
constexpr int kHeadsInOneLaunch = 32;

__device__ __forceinline__ int row_visits(const bma_block_lists& l, int64_t row) {
  return min(max(__ldg(l.full_kv_num + row), 0), l.NKV) + min(max(__ldg(l.kv_num + row), 0), l.NKV);
}
__device__ __forceinline__ long long block_sum256(long long v, long long* part) {   // the sum over 256 threads, to all of them
  for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  long long t = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += part[i];
  return t;
}

// All tables in one launch; every CTA adds up from the row counts what it needs itself, so that none waits for another
// (three dependent launches before took 8 us; this one 3 - 5).  The last CTA alone reads the rows of all list heads: with
// many heads that would be a chain of dependent reads on one SM, so there (kHeadsInOneLaunch) the CTAs of a head's last rows
// write its total and a second launch (HEADS) adds the totals up.
//   CTA head * ceil(NQ / 8) + g: rank[row][kj] = number of visited kv tiles below kj, or -1 when (row, kj) is not
//     visited, for eight rows (one warp each), and row_base of these rows = visits of the head's rows before them;
//   the last CTA: head_base[i], i in [0, B * Hq] = exclusive prefix over (b, h) of the list heads' totals.
// (A row base counts list entries; a block listed twice leaves an unused slot behind.)
enum SlotPhase { ALL, ROWS, HEADS };
__device__ __forceinline__ void slot_tables(SlotPhase phase, const bma_block_lists& l, int B, int Hq, int32_t* __restrict__ rank,
                                            int32_t* __restrict__ row_base, int64_t* __restrict__ head_total,
                                            int64_t* __restrict__ head_base, int cta, int ctas) {
  __shared__ uint32_t bits[8][kMaxKvTilesBwd / 32];
  __shared__ long long part[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int groups = (l.NQ + 7) / 8;
  if (phase == HEADS || (phase == ALL && cta == ctas - 1)) {
    const int LHEADS = phase == HEADS ? 0 : l.B * l.H;
    for (int i = w; i < LHEADS; i += 8) {   // one warp per list head
      long long s = 0;
      for (int r = lane; r < l.NQ; r += 32) s += row_visits(l, (int64_t)i * l.NQ + r);
      for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) head_total[i] = s;
    }
    __syncthreads();
    const int64_t n = (int64_t)B * Hq;
    long long carry = 0;
    for (int64_t base = 0; base < n; base += 256) {
      const int64_t i = base + threadIdx.x;
      long long v = 0;
      if (i < n) {
        const int b = (int)(i / Hq), h = (int)(i % Hq);
        v = head_total[(int64_t)(l.B == 1 ? 0 : b) * l.H + (l.H == 1 ? 0 : h)];
      }
      long long incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
      }
      __syncthreads();
      if (lane == 31) part[w] = incl;
      __syncthreads();
      long long before = carry, all = 0;
      for (int j = 0; j < 8; ++j) {
        if (j < w) before += part[j];
        all += part[j];
      }
      if (i < n) head_base[i] = before + incl - v;
      carry += all;
    }
    if (threadIdx.x == 0) head_base[n] = carry;
    return;
  }
  const int64_t head_row = (int64_t)(cta / groups) * l.NQ;
  const int first = (cta % groups) * 8;
  long long s = 0;
  for (int r = threadIdx.x; r < first; r += 256) s += row_visits(l, head_row + r);
  const int before = (int)block_sum256(s, part);
  const int r = first + w;
  if (r >= l.NQ) return;
  const int64_t row = head_row + r;
  if (lane == 0) {
    int mine = before;
    for (int i = first; i < r; ++i) mine += row_visits(l, head_row + i);
    row_base[row] = mine;
    if (phase == ROWS && r == l.NQ - 1) head_total[cta / groups] = mine + row_visits(l, row);
  }
  const int words = (l.NKV + 31) / 32;
  bits[w][lane] = 0u;
  __syncwarp();
  const int nfull = min(max(l.full_kv_num[row], 0), l.NKV), npart = min(max(l.kv_num[row], 0), l.NKV);
  const int32_t* full_idx = l.full_kv_idx + row * l.NKV;
  const int32_t* part_idx = l.kv_idx + row * l.NKV;
  for (int i = lane; i < nfull; i += 32) {
    const int j = full_idx[i];
    if (j >= 0 && j < l.NKV) atomicOr(&bits[w][j >> 5], 1u << (j & 31));
  }
  for (int i = lane; i < npart; i += 32) {
    const int j = part_idx[i];
    if (j >= 0 && j < l.NKV) atomicOr(&bits[w][j >> 5], 1u << (j & 31));
  }
  __syncwarp();
  const uint32_t mine = lane < words ? bits[w][lane] : 0u;
  int prefix = __popc(mine);   // inclusive scan over the lanes' word counts
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, prefix, off);
    if (lane >= off) prefix += v;
  }
  const int below = prefix - __popc(mine);
  int32_t* out = rank + row * l.NKV;
  for (int word = 0; word < words; ++word) {   // whole words at a time, so that the stores are coalesced
    const uint32_t bw = __shfl_sync(0xffffffffu, mine, word);
    const int start = __shfl_sync(0xffffffffu, below, word);
    const int j = word * 32 + lane;
    if (j < l.NKV) out[j] = (bw >> lane) & 1u ? start + __popc(bw & ((1u << lane) - 1u)) : -1;
  }
}

__global__ void __launch_bounds__(256) slot_tables_kernel(SlotPhase phase, const bma_block_lists l, int B, int Hq, const SlotTables t) {
  slot_tables(phase, l, B, Hq, t.rank, t.row_base, t.head_total, t.head_base, blockIdx.x, gridDim.x);
}
// The tables by the first `ctas` CTAs, delta and the bf16 copy of the cotangent by the others: both come before the dK/dV kernel and neither
// needs the other.  A launch less: 4.6 us of the host and 4 of the device (2 x 1000 tokens, lambda window, 16/4 heads: the call 161 -> 154 us).
template <typename TO, typename TDO>
__global__ void __launch_bounds__(256) slots_and_preprocess_kernel(const bma_block_lists l, int B, int Hq, const SlotTables t, int ctas,
                                                                   const bma_attn_args a, __nv_bfloat16* __restrict__ do_bf16) {
  if ((int)blockIdx.x < ctas) slot_tables(ALL, l, B, Hq, t.rank, t.row_base, t.head_total, t.head_base, blockIdx.x, ctas);
  else preprocess_rows4<TO, TDO>(a, do_bf16, (int)blockIdx.x - ctas, (int)gridDim.x - ctas);
}

// visited[b', h'] = sum over the rows of a list head of (kv_num + full_kv_num)
__global__ void __launch_bounds__(256) visited_kernel(bma_block_lists l, int64_t* __restrict__ visited) {
  __shared__ long long part[8];
  const int64_t row0 = (int64_t)blockIdx.x * l.NQ;
  long long s = 0;
  for (int i = threadIdx.x; i < l.NQ; i += blockDim.x) s += (long long)l.kv_num[row0 + i] + l.full_kv_num[row0 + i];
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long t = 0;
    for (int i = 0; i < 8; ++i) t += part[i];
    visited[blockIdx.x] = t;
  }
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

// Layout of the tables at the front of the backward workspace.
SlotTables slot_tables_layout(const bma_attn_args& a, const bma_block_lists& l, void* ws) {
  SlotTables t;
  uint8_t* p = static_cast<uint8_t*>(ws);
  size_t off = 0;
  t.head_base = reinterpret_cast<int64_t*>(p + off);
  off = align_up(off + sizeof(int64_t) * ((size_t)a.B * a.Hq + 1), 256);
  t.head_total = reinterpret_cast<int64_t*>(p + off);
  off = align_up(off + sizeof(int64_t) * (size_t)l.B * l.H, 256);
  t.row_base = reinterpret_cast<int32_t*>(p + off);
  off = align_up(off + sizeof(int32_t) * (size_t)l.B * l.H * l.NQ, 256);
  t.rank = reinterpret_cast<int32_t*>(p + off);
  off = align_up(off + sizeof(int32_t) * (size_t)l.B * l.H * l.NQ * l.NKV, 1024);
  t.bytes = off;
  return t;
}

int slot_tables_build(const bma_attn_args& a, const bma_block_lists& l, const SlotTables& t, const BwdPreprocess* pre, cudaStream_t st) {
  BMA_REQUIRE(l.NKV <= kMaxKvTilesBwd, BMA_ERR_LIMIT);
  const int64_t ctas = (int64_t)l.B * l.H * ((l.NQ + 7) / 8) + 1;
  BMA_REQUIRE(ctas <= INT32_MAX, BMA_ERR_LIMIT);
  const bool one = (int64_t)l.B * l.H <= kHeadsInOneLaunch;
  if (pre && one && a.d <= 128 && preprocess_vectors(pre->a, pre->out)) {
    const unsigned grid = (unsigned)(ctas + preprocess_rows4_ctas(pre->a));
    const bool of = pre->a.o.dtype == BMA_DTYPE_F32, gf = pre->a.d_o.dtype == BMA_DTYPE_F32;
    auto launch = [&](auto kernel) { kernel<<<grid, 256, 0, st>>>(l, a.B, a.Hq, t, (int)ctas, pre->a, pre->out); };
    if (of && gf) launch(slots_and_preprocess_kernel<float, float>);
    else if (of) launch(slots_and_preprocess_kernel<float, __nv_bfloat16>);
    else if (gf) launch(slots_and_preprocess_kernel<__nv_bfloat16, float>);
    else launch(slots_and_preprocess_kernel<__nv_bfloat16, __nv_bfloat16>);
    count_launches(1);
    BMA_CUDA_TRY(cudaGetLastError());
    return BMA_OK;
  }
  if (pre) {
    const int rc = bma_attn_bwd_preprocess(&pre->a, pre->out, st);
    if (rc) return rc;
  }
  slot_tables_kernel<<<(unsigned)(one ? ctas : ctas - 1), 256, 0, st>>>(one ? ALL : ROWS, l, a.B, a.Hq, t);
  if (!one) slot_tables_kernel<<<1, 256, 0, st>>>(HEADS, l, a.B, a.Hq, t);
  count_launches(one ? 1 : 2);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

int block_lists_visited(const bma_block_lists& l, int64_t* visited, cudaStream_t st) {
  visited_kernel<<<(unsigned)(l.B * l.H), 256, 0, st>>>(l, visited);
  count_launches(1);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

}  // namespace bma
