// Block-mask compilation (integer work, HBM-write bound).
//
// Produces the arrays of the reference's BlockMask (jaxmodules/block_mask.py:17-42) for a
// device-evaluable mask description, bit-exact with what create_block_mask
// (jaxmodules/block_mask.py:454-498) followed by BlockMask.from_blocks (:227-275) and
// get_sparse_{kv,q}_data_from_blocks (:411-451) returns:
//   pass 0 (only for segment masks)  per-block min/max of the segment ids
//   pass 1 classify                  one flag per block: 0 empty, 1 partial (any ^ all), 2 full (all); inside pass 2 unless
//                                    wide rows have blocks that must be scanned
//   pass 2 compact                   per row: count + [set indices ascending, unset indices ascending]
//                                    (== stable argsort(-blocks)), once along kv and once along q.
// The reference evaluates the dense B*H*Q*KV mask twice; here structured masks are classified
// from interval arithmetic on the block corners, and only blocks that a segment boundary or a
// bitmap touches are scanned element by element.  Masks that do not depend on b or h are
// classified once and the rows are replicated on the way out, so the cost is writing the
// int32 lists.
#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace bma {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxRowWidth = 16384;  // widest index row kept in shared memory (2 rows * 4 B * width)

__host__ __device__ inline bool depends_on_b(const bma_mask_spec& s) {
  return (s.flags & BMA_MASK_SEGMENT) || ((s.flags & BMA_MASK_BITMAP) && s.bitmap_B > 1) ||
         ((s.flags & BMA_MASK_TILES) && s.tiles_B > 1);
}
__host__ __device__ inline bool depends_on_h(const bma_mask_spec& s) {
  return ((s.flags & BMA_MASK_BITMAP) && s.bitmap_H > 1) || ((s.flags & BMA_MASK_TILES) && s.tiles_H > 1);
}

struct SegSummary {  // workspace views, each [B, nblocks]
  int32_t* qmin; int32_t* qmax; int32_t* kmin; int32_t* kmax;
};

// pass 0: min / max segment id of every q block and every kv block (valid part only).
__global__ void seg_summary_kernel(bma_mask_spec spec, int B, int NQ, int NKV, int QB, int KVB, SegSummary out) {
  const int lane = threadIdx.x & 31;
  const int warps_per_cta = blockDim.x >> 5;
  const int64_t total = (int64_t)B * (NQ + NKV);
  for (int64_t w = (int64_t)blockIdx.x * warps_per_cta + (threadIdx.x >> 5); w < total;
       w += (int64_t)gridDim.x * warps_per_cta) {
    const int b = (int)(w / (NQ + NKV));
    const int r = (int)(w % (NQ + NKV));
    const bool is_q = r < NQ;
    const int blk = is_q ? r : r - NQ;
    const int bs = is_q ? QB : KVB;
    const int valid = is_q ? spec.q_valid : spec.k_valid;
    const int off = is_q ? spec.q_offset : spec.k_offset;
    const int32_t* row = is_q ? spec.seg_q + (int64_t)b * spec.seg_q_stride : spec.seg_k + (int64_t)b * spec.seg_k_stride;
    const int lo = blk * bs, hi = min(lo + bs, valid);
    int mn = INT32_MAX, mx = INT32_MIN;
    for (int i = lo + lane; i < hi; i += 32) {
      int v = __ldg(row + off + i);
      mn = min(mn, v);
      mx = max(mx, v);
    }
    for (int o = 16; o; o >>= 1) {
      mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
      if (is_q) { out.qmin[(int64_t)b * NQ + blk] = mn; out.qmax[(int64_t)b * NQ + blk] = mx; }
      else      { out.kmin[(int64_t)b * NKV + blk] = mn; out.kmax[(int64_t)b * NKV + blk] = mx; }
    }
  }
}

// Flag of one block in closed form (interval terms on the block corners, segment-id ranges, stored tile classes): 0 empty,
// 1 partial, 2 full, or 3 where only the elements can tell (a segment boundary, a bit table or a change of the block
// window inside the block).
constexpr int kUndecided = 3;
__device__ __forceinline__ int block_flag(const bma_mask_spec& spec, const SegSummary& seg, int cb, int ch, int qi, int kj,
                                          int NQ, int NKV, int QB, int KVB) {
  bool any = false, all = false;
  if (!interval_classify(spec, qi * QB, kj * KVB, QB, KVB, any, all)) return kUndecided;
  if (!any) return 0;
  bool scan = false;
  if (spec.flags & BMA_MASK_SEGMENT) {
    const int qmn = seg.qmin[(int64_t)cb * NQ + qi], qmx = seg.qmax[(int64_t)cb * NQ + qi];
    const int kmn = seg.kmin[(int64_t)cb * NKV + kj], kmx = seg.kmax[(int64_t)cb * NKV + kj];
    if (qmx < kmn || qmn > kmx) return 0;                                  // ids never meet
    if (!(qmn == qmx && kmn == kmx && qmn == kmn)) {                       // a boundary crosses the block
      if (spec.flags & BMA_MASK_COMPILE_CONSERVATIVE) all = false;         // "partial" without looking closer
      else scan = true;
    }
  }
  if (spec.flags & BMA_MASK_BITMAP) scan = true;
  if (spec.flags & BMA_MASK_TILES) {
    // a block that IS a stored tile takes the tile's class (exactly, when no other term cuts the block); any other
    // block geometry is scanned element by element
    const bool is_tile = QB == 128 && KVB == 128 && (spec.q_offset & 127) == 0 && (spec.k_offset & 127) == 0;
    if (!is_tile) scan = true;
    else {
      const int64_t t = (((int64_t)(cb % spec.tiles_B) * spec.tiles_H + (ch % spec.tiles_H)) * spec.tiles_q +
                         ((qi * QB + spec.q_offset) >> 7)) * spec.tiles_k + ((kj * KVB + spec.k_offset) >> 7);
      const int tc = spec.tile_class[t];
      if (tc == 0) return 0;
      if (tc == 1) {
        if (all || (spec.flags & BMA_MASK_COMPILE_CONSERVATIVE)) all = false;   // cut by the tile alone: partial
        else scan = true;                                                        // cut by two terms: may be empty
      }
    }
  }
  return scan ? kUndecided : all ? 2 : 1;
}

// Flag of one block by its elements, by one whole warp: a lane takes a query row at a time and four words of 32 keys, so
// that a 128 x 128 block is four batches of independent loads (stops as soon as the block is known to be partial).
// Element by element with a row at a time, the 8 x 8 blocks of 128 x 128 of a bit table took 122 us in a launch of their own;
// the whole build of their lists, scan included, now takes 12.
// The first 32 x 32 elements come first by themselves: most blocks that a segment edge crosses are known to be partial then, and
// a batch of 32 x 128 segment ids costs four times as many comparisons (documents of 77 tokens, 16 x 4096, whole build
// with blocks of 64: element by element 63 us, batches alone 76, now 66; blocks of 128: 75, 68, 61).
__device__ __forceinline__ int scan_block(const bma_mask_spec& spec, int cb, int ch, int qi, int kj, int QB, int KVB) {
  const int lane = threadIdx.x & 31;
  const MaskView m = make_mask_view(spec, cb, ch);
  const int q0 = qi * QB, k0 = kj * KVB;
  const int q_end = min(q0 + QB, spec.q_valid), k_end = min(k0 + KVB, spec.k_valid);
  bool any = false;
  bool all = (q0 + QB <= spec.q_valid) && (k0 + KVB <= spec.k_valid);
  for (int step = 0; !(any && !all); ++step) {
    const int r = q0 + max(step - 1, 0) * 32, k_to = step == 0 ? min(k0 + 32, k_end) : k_end;
    if (r >= q_end) break;
    const int q = r + lane;
    bool row_any = false, row_all = true;
    if (q < q_end) {
      int jlo, jhi;
      row_interval(m, q, k0, jlo, jhi);
      for (int kb = k0; kb < k_to; kb += 128) {
        uint32_t bits[4], want[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int j0 = kb - k0 + c * 32, n = min(32, k_to - kb - c * 32);
          want[c] = n <= 0 ? 0u : 0xffffffffu >> (32 - n);
          const int lo = max(jlo - j0, 0), hi = min(jhi - j0, 31);
          bits[c] = (lo <= hi) ? ((0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) & want[c] : 0u;
          if (bits[c] && (m.flags & kTableTerms)) bits[c] &= table_bits_row32(m, q, kb + c * 32);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          row_any |= bits[c] != 0u;
          row_all &= bits[c] == want[c];
        }
      }
    }
    any |= __any_sync(0xffffffffu, row_any) != 0;
    all &= __all_sync(0xffffffffu, row_all) != 0;
    if (r + 32 >= q_end && k_to == k_end) break;   // (a block of 32 x 32 is done after the first look)
  }
  return all ? 2 : (any ? 1 : 0);
}

// pass 1a: one THREAD per block.  Closed forms decide almost every block; flags leave as coalesced bytes.  The blocks that
// stay open are appended to a work list for pass 1b.
// The list and its counter live in output arrays that pass 2 overwrites afterwards (`todo` = kv_idx, one
// int32 per block at least; `todo_count` = kv_num[0]), so the scratch stays at one byte per block.
struct BlockCoord { int cb, ch, qi, kj; };
__device__ __forceinline__ BlockCoord block_coord(int64_t w, int CH, int NQ, int NKV) {
  BlockCoord c;
  const int64_t row = w / NKV;
  c.kj = (int)(w - row * NKV);
  uint32_t r = (uint32_t)row;
  c.qi = (int)(r % (uint32_t)NQ);
  r /= (uint32_t)NQ;
  c.ch = (int)(r % (uint32_t)CH);
  c.cb = (int)(r / (uint32_t)CH);
  return c;
}

__global__ void classify_kernel(bma_mask_spec spec, int CB, int CH, int NQ, int NKV, int QB, int KVB,
                                SegSummary seg, uint8_t* __restrict__ flags, int32_t* __restrict__ todo,
                                int32_t* __restrict__ todo_count) {
  const int lane = threadIdx.x & 31;
  const int64_t total = (int64_t)CB * CH * NQ * NKV;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // `base` is the warp's first block: uniform across the warp, so the ballot below sees all 32 lanes
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < total; base += stride) {
    const int64_t w = base + lane;
    bool scan = false;
    if (w < total) {
      const BlockCoord c = block_coord(w, CH, NQ, NKV);
      const int f = block_flag(spec, seg, c.cb, c.ch, c.qi, c.kj, NQ, NKV, QB, KVB);
      scan = f == kUndecided;
      flags[w] = (uint8_t)f;   // rewritten by pass 1b when `scan`
    }
    const unsigned m = __ballot_sync(0xffffffffu, scan);
    if (m != 0u) {  // one atomic per warp
      const int leader = __ffs(m) - 1;
      int pos = 0;
      if (lane == leader) pos = atomicAdd(todo_count, __popc(m));
      pos = __shfl_sync(0xffffffffu, pos, leader);
      if (scan) todo[pos + __popc(m & ((1u << lane) - 1u))] = (int32_t)w;
    }
  }
}

// pass 1b: one WARP per listed block.
__global__ void scan_kernel(bma_mask_spec spec, int CH, int NQ, int NKV, int QB, int KVB, uint8_t* __restrict__ flags,
                            const int32_t* __restrict__ todo, const int32_t* __restrict__ todo_count) {
  const int lane = threadIdx.x & 31;
  const int warps_per_cta = blockDim.x >> 5;
  const int count = *todo_count;
  for (int i = blockIdx.x * warps_per_cta + (threadIdx.x >> 5); i < count; i += gridDim.x * warps_per_cta) {
    const int64_t w = todo[i];
    const BlockCoord c = block_coord(w, CH, NQ, NKV);
    const int f = scan_block(spec, c.cb, c.ch, c.qi, c.kj, QB, KVB);
    if (lane == 0) flags[w] = (uint8_t)f;
  }
}

// pass 2: one CTA per (classification row, replica chunk).  TRANSPOSED = q-side lists.
// Shared memory: 2 index rows of `NC` int32, the row's `NC` flag bytes, + scan scratch.
// With `flags` null the CTA classifies its row itself, so that passes 1a and 1b, their launches and the flag bytes fall
// away.  Each block is then classified once per list side; that is cheap in closed form, and elements are scanned here
// only where a row is short (kInlineScanWidth).
struct RowSource {
  const uint8_t* flags;
  bma_mask_spec spec;
  SegSummary seg;
  int QB, KVB;
};
template <bool TRANSPOSED, bool SCAN>
__device__ __forceinline__ void compact_row(const RowSource& src, int CB, int CH, int NQ, int NKV, int out_B,
                                            int out_H, int32_t* __restrict__ part_num, int32_t* __restrict__ part_idx,
                                            int32_t* __restrict__ full_num, int32_t* __restrict__ full_idx) {
  extern __shared__ int32_t smem[];
  const int NR = TRANSPOSED ? NKV : NQ;   // rows of the output
  const int NC = TRANSPOSED ? NQ : NKV;   // row width
  int32_t* row_p = smem;
  int32_t* row_f = smem + NC;
  __shared__ int warp_p[kThreads / 32], warp_f[kThreads / 32];
  __shared__ int tot_p, tot_f;

  const int r = blockIdx.x % NR;
  const int ch = (blockIdx.x / NR) % CH;
  const int cb = blockIdx.x / (NR * CH);
  // the row's flags go to shared memory first: all loads of a thread are in flight together (a column of the
  // flag grid, for the q-side lists, is one byte per 32-byte sector), and both passes below read them twice
  uint8_t* fl = reinterpret_cast<uint8_t*>(smem + 2 * NC);
  if (src.flags) {
    const uint8_t* fbase = src.flags + (int64_t)(cb * CH + ch) * NQ * NKV;
    for (int c = threadIdx.x; c < NC; c += kThreads) fl[c] = TRANSPOSED ? fbase[(int64_t)c * NKV + r] : fbase[(int64_t)r * NKV + c];
    __syncthreads();
  } else {
    int open = 0;
    for (int c = threadIdx.x; c < NC; c += kThreads) {
      const int f = block_flag(src.spec, src.seg, cb, ch, TRANSPOSED ? c : r, TRANSPOSED ? r : c, NQ, NKV, src.QB, src.KVB);
      open |= f == kUndecided;
      fl[c] = (uint8_t)f;
    }
    if (!SCAN) {
      __syncthreads();
    } else if (__syncthreads_or(open)) {
      for (int c = threadIdx.x >> 5; c < NC; c += kThreads / 32) {   // one warp per open block
        const int f = fl[c];
        __syncwarp();
        if (f != kUndecided) continue;
        const int g = scan_block(src.spec, cb, ch, TRANSPOSED ? c : r, TRANSPOSED ? r : c, src.QB, src.KVB);
        if ((threadIdx.x & 31) == 0) fl[c] = (uint8_t)g;
      }
      __syncthreads();
    }
  }
  auto flag_at = [&](int c) -> int { return fl[c]; };

  const int per = (NC + kThreads - 1) / kThreads;
  const int c0 = min(NC, (int)threadIdx.x * per), c1 = min(NC, c0 + per);
  int np = 0, nf = 0;
  for (int c = c0; c < c1; ++c) {
    const int f = flag_at(c);
    np += (f == 1);
    nf += (f == 2);
  }
  // exclusive block scan of (np, nf)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int sp = np, sf = nf;
  for (int o = 1; o < 32; o <<= 1) {
    int tp = __shfl_up_sync(0xffffffffu, sp, o), tf = __shfl_up_sync(0xffffffffu, sf, o);
    if (lane >= o) { sp += tp; sf += tf; }
  }
  if (lane == 31) { warp_p[wid] = sp; warp_f[wid] = sf; }
  __syncthreads();
  if (threadIdx.x == 0) {
    int ap = 0, af = 0;
    for (int i = 0; i < kThreads / 32; ++i) {
      int tp = warp_p[i], tf = warp_f[i];
      warp_p[i] = ap; warp_f[i] = af;
      ap += tp; af += tf;
    }
    tot_p = ap; tot_f = af;
  }
  __syncthreads();
  int before_p = warp_p[wid] + sp - np, before_f = warp_f[wid] + sf - nf;
  const int total_p = tot_p, total_f = tot_f;
  for (int c = c0; c < c1; ++c) {
    const int f = flag_at(c);
    if (f == 1) row_p[before_p++] = c; else row_p[total_p + (c - before_p)] = c;
    if (f == 2) row_f[before_f++] = c; else row_f[total_f + (c - before_f)] = c;
  }
  __syncthreads();

  // replicate to every (b, h) of the output that this classification row stands for
  const int rep_b = (CB == out_B) ? 1 : out_B, rep_h = (CH == out_H) ? 1 : out_H;
  const int reps = rep_b * rep_h;
  for (int rep = blockIdx.y; rep < reps; rep += gridDim.y) {
    const int b = (CB == out_B) ? cb : rep / rep_h;
    const int h = (CH == out_H) ? ch : rep % rep_h;
    const int64_t row = ((int64_t)b * out_H + h) * NR + r;
    if (threadIdx.x == 0) { part_num[row] = total_p; full_num[row] = total_f; }
    int32_t* dp = part_idx + row * NC;
    int32_t* df = full_idx + row * NC;
    if ((NC & 3) == 0 && (((uintptr_t)part_idx | (uintptr_t)full_idx) & 15) == 0) {
      const int4* sp4 = reinterpret_cast<const int4*>(row_p);
      const int4* sf4 = reinterpret_cast<const int4*>(row_f);
      for (int i = threadIdx.x; i < NC / 4; i += kThreads) {
        reinterpret_cast<int4*>(dp)[i] = sp4[i];
        reinterpret_cast<int4*>(df)[i] = sf4[i];
      }
    } else {
      for (int i = threadIdx.x; i < NC; i += kThreads) { dp[i] = row_p[i]; df[i] = row_f[i]; }
    }
  }
}

// The kv side (blockIdx.z = 0) and, where wanted, the q side (1) in ONE launch: no launch gap between them, and the tail of
// one side fills with the other's rows.  The builder is bound by the HBM writes of the index arrays.
template <bool SCAN>
__global__ void __launch_bounds__(kThreads) compact_kernel(const __grid_constant__ RowSource src, int CB, int CH, int NQ, int NKV,
                                                           int out_B, int out_H, const __grid_constant__ bma_block_lists l) {
  if (blockIdx.z == 0) {
    if ((int)blockIdx.x < CB * CH * NQ)
      compact_row<false, SCAN>(src, CB, CH, NQ, NKV, out_B, out_H, l.kv_num, l.kv_idx, l.full_kv_num, l.full_kv_idx);
  } else {
    if ((int)blockIdx.x < CB * CH * NKV)
      compact_row<true, SCAN>(src, CB, CH, NQ, NKV, out_B, out_H, l.q_num, l.q_idx, l.full_q_num, l.full_q_idx);
  }
}

// Widest row whose open blocks are scanned by the CTA that compacts it: its eight warps take four blocks each then, a few
// microseconds more than the launches of the separate passes cost; a wider row is better spread over the whole chip.
// (In closed form the row is always classified here: 1024 x 1024 blocks, both sides, 32 heads: 93 us against 101 with the
// flags written and read back, of which 82 us are the index arrays at the copy rate.)
constexpr int kInlineScanWidth = 32;
// ... and most blocks of such rows: each is scanned once per list side there, which costs more than two launches once the chip is
// full.  (32 x 32 blocks of 128 of a bit table per head, whole build: 32 heads 64 us in separate passes, 62 here; 512 heads 125
// and 133.)
constexpr int64_t kInlineScanBlocks = 1 << 15;

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct WorkspacePlan {
  size_t flags_off, seg_off, total;
  int CB, CH;
};

WorkspacePlan plan_workspace(const bma_mask_spec& s, int B, int H, int NQ, int NKV) {
  WorkspacePlan p;
  p.CB = depends_on_b(s) ? B : 1;
  p.CH = depends_on_h(s) ? H : 1;
  p.flags_off = 0;
  size_t flags_bytes = (size_t)p.CB * p.CH * NQ * NKV;
  p.seg_off = align_up(flags_bytes, 256);
  size_t seg_bytes = (s.flags & BMA_MASK_SEGMENT) ? sizeof(int32_t) * 2 * (size_t)B * (NQ + NKV) : 0;
  p.total = p.seg_off + align_up(seg_bytes, 256);
  return p;
}

}  // namespace

size_t mask_compile_workspace_bytes(const bma_mask_spec& spec, int B, int H, int NQ, int NKV) {
  return plan_workspace(spec, B, H, NQ, NKV).total;
}

int mask_compile_validate(const bma_mask_spec& s, int B, int H, const bma_block_lists& l) {
  BMA_REQUIRE(B > 0 && H > 0 && l.NQ > 0 && l.NKV > 0 && l.q_block > 0 && l.kv_block > 0, BMA_ERR_ARG);
  BMA_REQUIRE(l.kv_num && l.kv_idx && l.full_kv_num && l.full_kv_idx, BMA_ERR_ARG);
  const bool any_q = l.q_num || l.q_idx || l.full_q_num || l.full_q_idx;
  const bool all_q = l.q_num && l.q_idx && l.full_q_num && l.full_q_idx;
  BMA_REQUIRE(!any_q || all_q, BMA_ERR_ARG);
  BMA_REQUIRE((l.B == B || (l.B == 1 && !depends_on_b(s))) && (l.H == H || (l.H == 1 && !depends_on_h(s))), BMA_ERR_ARG);
  BMA_REQUIRE(interval_terms_valid(s), BMA_ERR_ARG);
  BMA_REQUIRE((int64_t)l.NQ * l.q_block >= s.q_valid && (int64_t)l.NKV * l.kv_block >= s.k_valid, BMA_ERR_ARG);
  if (s.flags & BMA_MASK_SEGMENT) BMA_REQUIRE(s.seg_q && s.seg_k, BMA_ERR_ARG);
  if (s.flags & BMA_MASK_BITMAP)
    BMA_REQUIRE(s.bitmap && s.bitmap_B > 0 && s.bitmap_H > 0 && s.bitmap_words > 0 && s.bitmap_q > 0, BMA_ERR_ARG);
  if (s.flags & BMA_MASK_TILES) {
    BMA_REQUIRE(s.tile_class && s.tile_slot && s.tiles_B > 0 && s.tiles_H > 0 && s.tiles_q > 0 && s.tiles_k > 0, BMA_ERR_ARG);
    BMA_REQUIRE((int64_t)s.tiles_q * 128 >= (int64_t)s.q_valid + s.q_offset && (int64_t)s.tiles_k * 128 >= (int64_t)s.k_valid + s.k_offset,
                BMA_ERR_ARG);
  }
  BMA_REQUIRE(l.NQ <= kMaxRowWidth && l.NKV <= kMaxRowWidth, BMA_ERR_LIMIT);
  return BMA_OK;
}

// Launches the three passes with `workspace` as scratch (flags, then segment summaries).
int mask_compile_launch(const bma_mask_spec& spec, int B, int H, const bma_block_lists& l, void* workspace,
                        cudaStream_t st) {
  const WorkspacePlan p = plan_workspace(spec, B, H, l.NQ, l.NKV);
  uint8_t* flags = static_cast<uint8_t*>(workspace) + p.flags_off;
  SegSummary seg{nullptr, nullptr, nullptr, nullptr};
  int sm_count = 148;
  {
    int dev = 0;
    BMA_CUDA_TRY(cudaGetDevice(&dev));
    BMA_CUDA_TRY(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  if (spec.flags & BMA_MASK_SEGMENT) {
    int32_t* base = reinterpret_cast<int32_t*>(static_cast<uint8_t*>(workspace) + p.seg_off);
    seg.qmin = base;
    seg.qmax = seg.qmin + (size_t)B * l.NQ;
    seg.kmin = seg.qmax + (size_t)B * l.NQ;
    seg.kmax = seg.kmin + (size_t)B * l.NKV;
    const int64_t warps = (int64_t)B * (l.NQ + l.NKV);
    const int grid = (int)std::min<int64_t>((warps + 7) / 8, (int64_t)sm_count * 8);
    seg_summary_kernel<<<grid, kThreads, 0, st>>>(spec, B, l.NQ, l.NKV, l.q_block, l.kv_block, seg);
    count_launches(1);
  }
  // Blocks that closed forms cannot decide exist only with these terms (a block window whose blocks are whole multiples of
  // the list's query blocks never changes inside one).
  const bool window_cuts = (spec.flags & BMA_MASK_BLOCK_WINDOW) && (spec.win_block % l.q_block != 0 || spec.q_offset % l.q_block != 0);
  const bool may_scan = (spec.flags & (BMA_MASK_BITMAP | BMA_MASK_TILES)) || window_cuts ||
                        ((spec.flags & BMA_MASK_SEGMENT) && !(spec.flags & BMA_MASK_COMPILE_CONSERVATIVE));
  const int width = std::max(l.NQ, l.NKV);
  RowSource src{nullptr, spec, seg, l.q_block, l.kv_block};
  const int64_t blocks = (int64_t)p.CB * p.CH * l.NQ * l.NKV;
  if (may_scan && (width > kInlineScanWidth || blocks > kInlineScanBlocks)) {
    const int grid = (int)std::min<int64_t>((blocks + kThreads - 1) / kThreads, (int64_t)sm_count * 16);
    BMA_CUDA_TRY(cudaMemsetAsync(l.kv_num, 0, sizeof(int32_t), st));
    classify_kernel<<<grid, kThreads, 0, st>>>(spec, p.CB, p.CH, l.NQ, l.NKV, l.q_block, l.kv_block, seg, flags, l.kv_idx, l.kv_num);
    scan_kernel<<<sm_count * 8, kThreads, 0, st>>>(spec, p.CH, l.NQ, l.NKV, l.q_block, l.kv_block, flags, l.kv_idx, l.kv_num);
    count_launches(2);
    src.flags = flags;
  }
  const int rows = p.CB * p.CH * (l.q_num ? width : l.NQ);
  const int NC = l.q_num ? width : l.NKV;
  const int reps = ((p.CB == l.B) ? 1 : l.B) * ((p.CH == l.H) ? 1 : l.H);
  const int gy = std::min(std::max(1, std::min(reps, (sm_count * 4 + rows - 1) / rows)), 65535);
  const size_t smem = sizeof(int32_t) * 2 * (size_t)NC + align_up((size_t)NC, 16);
  const dim3 grid(rows, gy, l.q_num ? 2 : 1);
  auto launch = [&](auto kernel) -> int {
    if (smem > 48 * 1024) BMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, kThreads, smem, st>>>(src, p.CB, p.CH, l.NQ, l.NKV, l.B, l.H, l);
    return BMA_OK;
  };
  const int rc = (may_scan && !src.flags) ? launch(compact_kernel<true>) : launch(compact_kernel<false>);
  if (rc) return rc;
  count_launches(1);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

// ---------------------------------------------------------------------------------------------
// Variant for callers that must not allocate: the scratch lives in the module image.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr size_t kStaticScratchBytes = size_t(4) << 20;  // 4 MiB per GPU that loads the library

// Block flags and segment summaries of bma_mask_compile_static.  Every call on a device uses this
// one array, so two calls whose kernels overlap on the GPU race on it.  Nothing in it has to start
// at zero: the classify pass writes every flag and the summary pass every summary before they are
// read, so no clearing is needed between calls.
static __device__ __align__(256) uint8_t g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevicesStatic = 64;
void* g_static_scratch_ptr[kMaxDevicesStatic] = {};
std::mutex g_static_scratch_mutex;

// Device address of g_static_scratch on the current device.  In host code the symbol name is only
// a handle, not an address a kernel may dereference; the address comes from the runtime, once per
// device, with that device current.
int static_scratch_address(void** out) {
  int dev = 0;
  BMA_CUDA_TRY(cudaGetDevice(&dev));
  BMA_REQUIRE(dev >= 0 && dev < kMaxDevicesStatic, BMA_ERR_LIMIT);
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (!g_static_scratch_ptr[dev]) {
    void* ptr = nullptr;
    BMA_CUDA_TRY(cudaGetSymbolAddress((void**)&ptr, g_static_scratch));
    BMA_REQUIRE(ptr != nullptr, BMA_ERR_CUDA);
    g_static_scratch_ptr[dev] = ptr;
  }
  *out = g_static_scratch_ptr[dev];
  return BMA_OK;
}

}  // namespace

size_t mask_compile_static_limit() { return kStaticScratchBytes; }

int mask_compile_static(const bma_mask_spec& spec, int B, int H, const bma_block_lists& l, cudaStream_t st) {
  int rc = mask_compile_validate(spec, B, H, l);
  if (rc != BMA_OK) return rc;
  if (mask_compile_workspace_bytes(spec, B, H, l.NQ, l.NKV) > kStaticScratchBytes) return BMA_ERR_LIMIT;
  void* scratch = nullptr;
  rc = static_scratch_address(&scratch);
  if (rc != BMA_OK) return rc;
  return mask_compile_launch(spec, B, H, l, scratch, st);
}

}  // namespace bma
