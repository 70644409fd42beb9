// Shared helpers for the blockwise masked attention kernels: status handling, the device
// form of the mask predicate, and small numeric utilities.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "../../include/bma.h"

namespace bma {

// ---- host-side error plumbing ----------------------------------------------------------
void set_last_cuda_error(cudaError_t e, const char* where);

#define BMA_CUDA_TRY(expr)                                   \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) {                                 \
      ::bma::set_last_cuda_error(_e, #expr);                 \
      return BMA_ERR_CUDA;                                   \
    }                                                        \
  } while (0)

#define BMA_REQUIRE(cond, code) \
  do {                          \
    if (!(cond)) return (code); \
  } while (0)

// Device-side status word (one per device, lives for the lifetime of the module).  Kernels
// get its address as an argument and record a non-zero code with atomicCAS when a bounded
// wait or a bounds check gives up.  Returns nullptr (and records the CUDA error) on failure.
int* device_status_ptr();

// Host-side count of kernels launched by this library in this process (diagnostics).
constexpr int kMaxParts = 8;   // CTAs of a cluster
void count_launches(int n, int cluster = 1);

__device__ __forceinline__ void report_device_error(int* status, int code) { atomicCAS(status, 0, code); }

// Terms of the mask that are looked up (segment ids, bit table, tile bits) rather than computed from the indices.
constexpr int kTableTerms = BMA_MASK_SEGMENT | BMA_MASK_BITMAP | BMA_MASK_TILES;

// ---- order of a launch's CTAs -------------------------------------------------------------
// One CTA per (tile, head, batch).  CTAs start in the order of their linear index: one head after another, the longest walk of each
// (under a causal mask) first, or the longest walks of all heads first.  In the first order a launch ends with the longest walks of its last
// heads on an idle chip: 512 CTAs of 16 causal tiles take 1.29 of the even span, 1.05 in the second (float32, 2 x 2048 tokens, 16
// heads of 64: kernels 570 -> 480 us, the call 600 -> 545; bf16, forward and backward: 1 x 4096, 16 heads of 128 366 -> 304 us, 4 x 1024, 32/8
// heads of 128 281 -> 250, 1 x 8192, 16/8 heads of 64 912 -> 791, packed documents 2 x 4096, 16 heads 562 -> 470).  The second is for
// launches whose end counts, at most 4 waves, and whose heads together stream (K and V forward) no more than L2 holds: in a
// longer launch the end is a few per cent, less than what heads side by side cost there (dQ replay of 7 waves, 8 x 2048, 16 heads: the
// call 690 -> 713 us; causal B=8 L=4096 H=32 d=128, 28 and 55 waves: 4800 -> 4950).
constexpr int kSms = 148;
constexpr int64_t kStreamInL2 = 64 << 20;   // of 126 MB, of which a line may take two (one per die)
inline bool longest_first(int64_t tiles, int64_t heads, int64_t batches, int64_t stream_bytes_per_head) {
  return tiles * heads * batches <= 4 * kSms && heads <= 65535 && heads * batches * stream_bytes_per_head <= kStreamInL2;
}
// With `parts` CTAs to a (tile, head, batch), which are a cluster.
inline dim3 cta_grid(bool by_rank, int tiles, int heads, int batches, int parts = 1) {
  return by_rank ? dim3(heads * parts, batches, tiles) : dim3(tiles * parts, heads, batches);
}
inline cudaLaunchAttribute cluster_attribute(int x, int y = 1) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = x; attr.val.clusterDim.y = y; attr.val.clusterDim.z = 1;
  return attr;
}
// The current device, and its number of SMs (asked once per device).
constexpr int kMaxDevices = 64;
inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices ? dev : 0;
}
inline int device_sms(int dev) {
  static std::atomic<int> known[kMaxDevices];
  int n = known[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    return kSms;
  }
  known[dev].store(n, std::memory_order_relaxed);
  return n;
}
// How many clusters of `parts` CTAs of a kernel the current device runs at the same time (0 where it runs none).  `known` keeps the answers for one
// instance of a kernel, by device; a question that fails is asked again by the next call.
struct ClusterCounts {
  std::atomic<int> plus_one[kMaxDevices][kMaxParts + 1];
};
template <typename K>
int clusters_at_once(ClusterCounts& known, K kernel, int threads, size_t smem, int parts) {
  const int dev = current_device();
  if (parts == 1) return device_sms(dev);
  std::atomic<int>& k = known.plus_one[dev][parts];
  const int n = k.load(std::memory_order_relaxed);
  if (n) return n - 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kSms * parts);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr = cluster_attribute(parts);
  cfg.attrs = &attr; cfg.numAttrs = 1;
  int most = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  k.store(1 + most, std::memory_order_relaxed);
  return most;
}
// Walks of a launch: its CTAs, the longest and all of them together, in tiles.
struct Walks {
  int ctas;
  double longest, sum;
  bool even;      // all about as long as the longest
  bool known;     // false: as if terms of the mask that are looked up allowed everything
};
// Bands and block windows bound a walk by the 128-tiles that they are wide, and the two that they cut; `heads` such walks make one.
inline void bound_walks(Walks& w, const bma_mask_spec& s, int heads) {
  double width = 1e30;
  if (s.flags & BMA_MASK_BAND) width = (double)s.band_left + s.band_right;
  if (s.flags & BMA_MASK_BLOCK_WINDOW) width = std::min(width, ((double)s.win_left + s.win_right) * s.win_block);
  w.longest = std::min(w.longest, heads * (width / 128 + 2.));
  w.sum = std::min(w.sum, w.longest * w.ctas);
}
// Walks of the 128-query tiles over key tiles, of the key tiles over a head group's query tiles, as the arguments and the mask say and nothing else:
// the order of a sum does not depend on the workspace of a call or on the ranges it is run in.  (Of terms that are looked up nothing is known here.)
inline Walks q_walks(const bma_attn_args& a, const bma_mask_spec& spec) {
  const int heads = a.B * a.Hq, NQ = (a.N + 127) / 128, NKV = (a.L + 127) / 128;
  const bool known = !(spec.flags & kTableTerms);
  Walks w{NQ * heads, (double)NKV, (double)NQ * heads * NKV, true, known};
  if (spec.flags & BMA_MASK_CAUSAL) {
    w = {NQ * heads, 0., 0., false, known};
    for (int qi = 0; qi < NQ; ++qi) {
      const int64_t keys = std::min<int64_t>((int64_t)(qi + 1) * 128, a.N) + spec.q_offset - spec.k_offset;
      const double t = (double)std::min<int64_t>(std::max<int64_t>((keys + 127) / 128, 0), NKV);
      w.longest = std::max(w.longest, t);
      w.sum += t * heads;
    }
  }
  bound_walks(w, spec, 1);
  return w;
}
inline Walks k_walks(const bma_attn_args& a, const bma_mask_spec& spec) {
  const int G = a.Hq / a.Hkv, NQ = (a.N + 127) / 128, NKV = (a.L + 127) / 128;
  const Walks q = q_walks(a, spec);
  Walks w{NKV * a.B * a.Hkv, (double)G * NQ, q.sum, q.even, q.known};
  bound_walks(w, spec, G);
  return w;
}
// The number of CTAs that share a walk, for the shortest time of the launch.  With n clusters at once a launch takes the longest of: waves of
// walks of one length, or else the longest walk, or the even share of all; each CTA `extra` tiles besides its own.  Where the walks may be much
// shorter than they are taken to be, more CTAs than run at once cost more than they give, and have to promise a quarter less time (float32,
// documents of 300 of 4096 tokens, one head of 64, forward: 4 CTAs to a walk, all of them at once, 40 us, as unshared; 8 in two waves 54).
template <typename N>
int share_walks(const Walks& w, double extra, int most_parts, N clusters) {
  int best = 1;
  double cost = 1e30;
  for (int parts = 1; parts <= most_parts && parts <= kMaxParts; ++parts) {
    const int n = clusters(parts);
    if (n < 1) continue;
    const double c = w.even ? (double)((w.ctas + n - 1) / n) * (w.longest / parts + extra)
                            : std::max(w.longest / parts + extra, (w.sum / parts + w.ctas * extra) / n * 1.05);
    if (c < (w.known || n >= w.ctas ? 0.95 : 0.75) * cost) { cost = c; best = parts; }
  }
  return best;
}
// rank: 0 for the first tile to start of its head
__device__ __forceinline__ void cta_of(bool by_rank, int& rank, int& head, int& batch) {
  rank = by_rank ? blockIdx.z : blockIdx.x;
  head = by_rank ? blockIdx.x : blockIdx.y;
  batch = by_rank ? blockIdx.y : blockIdx.z;
}
// With the order known to the compiler: the selects above cost the loops of the d = 64 kernels registers, 1.5 and 3.5 % (B=4 L=4096 H=32/8
// causal, dK/dV 825 -> 838 us, forward 433 -> 448).
template <bool BY_RANK>
__device__ __forceinline__ void cta_of(int& rank, int& head, int& batch) {
  rank = BY_RANK ? blockIdx.z : blockIdx.x;
  head = BY_RANK ? blockIdx.x : blockIdx.y;
  batch = BY_RANK ? blockIdx.y : blockIdx.z;
}
__device__ __forceinline__ void cta_of_cluster(bool by_rank, int& rank, int& head, int& batch) {   // the same for a launch in clusters (or not)
  const dim3 id = __clusterIdx();
  rank = by_rank ? id.z : id.x;
  head = by_rank ? id.x : id.y;
  batch = by_rank ? id.y : id.z;
}
// The same in groups, for the float32 kernels, which run 6 - 12 times as long on a byte, so that no launch is too long for it:
// one-dimensional grid, rank 0 of every head of a group, then rank 1, and so on; `head` counts the (batch, head) pairs.
struct LaunchOrder {
  int tiles, heads, group;
};
__device__ __forceinline__ void cta_of(const LaunchOrder& o, int index, int& rank, int& head) {
  const int per = o.group * o.tiles, g = index / per, r = index - g * per;
  const int in_group = min(o.group, o.heads - g * o.group);   // (the last group may be smaller)
  rank = __shfl_sync(0xffffffffu, r / in_group, 0);           // (warp-uniform, which the compiler does not see through divisions)
  head = __shfl_sync(0xffffffffu, g * o.group + r % in_group, 0);
}
inline LaunchOrder launch_order(int tiles, int64_t heads, int64_t stream_bytes_per_head) {
  int64_t group = kStreamInL2 / (stream_bytes_per_head > 0 ? stream_bytes_per_head : 1);
  if (group < 1) group = 1;
  const int64_t groups = heads > group ? (heads + group - 1) / group : 1;
  return {tiles, (int)heads, (int)((heads + groups - 1) / groups)};   // groups of one size: a small last one would end the launch alone
}
inline unsigned launch_ctas(const LaunchOrder& o) { return (unsigned)(o.tiles * o.heads); }

// What the interval terms of a mask have to satisfy, for lists to be compiled from them or for a pass to know its blocks without lists.
inline bool interval_terms_valid(const bma_mask_spec& s) {
  if (s.q_valid < 0 || s.k_valid < 0) return false;
  if ((s.flags & BMA_MASK_BLOCK_WINDOW) && !(s.win_block > 0 && s.win_left >= 0 && s.win_right >= 0 && (int64_t)s.win_left + s.win_right <= s.win_nblk)) return false;
  return !(s.flags & BMA_MASK_BAND) || (s.band_left >= 0 && s.band_right >= 0);
}

// ---- mask predicate --------------------------------------------------------------------
// Device copy of bma_mask_spec with the per-(b,h) row pointers resolved once per CTA.
struct MaskView {
  int flags;
  int q_valid, k_valid;
  int q_offset, k_offset;
  int band_left, band_right;
  int win_block, win_left, win_right, win_nblk;
  const int32_t* seg_q_row;     // &seg_q[b*stride]
  const int32_t* seg_k_row;
  const uint32_t* bitmap_bh;    // &bitmap[((b%BB)*BH + h%BH) * bitmap_q * words]
  int bitmap_words;
  const uint8_t* tile_class_bh; // TILES: &tile_class[((b%TB)*TH + h%TH) * tiles_q * tiles_k], likewise tile_slot_bh
  const int32_t* tile_slot_bh;
  const uint32_t* tile_bits;
  int tiles_k;
};

__device__ __forceinline__ MaskView make_mask_view(const bma_mask_spec& s, int b, int h) {
  MaskView m;
  m.flags = s.flags;
  m.q_valid = s.q_valid; m.k_valid = s.k_valid;
  m.q_offset = s.q_offset; m.k_offset = s.k_offset;
  m.band_left = s.band_left; m.band_right = s.band_right;
  m.win_block = s.win_block; m.win_left = s.win_left; m.win_right = s.win_right; m.win_nblk = s.win_nblk;
  m.seg_q_row = (s.flags & BMA_MASK_SEGMENT) ? s.seg_q + (int64_t)b * s.seg_q_stride : nullptr;
  m.seg_k_row = (s.flags & BMA_MASK_SEGMENT) ? s.seg_k + (int64_t)b * s.seg_k_stride : nullptr;
  m.bitmap_words = s.bitmap_words;
  m.bitmap_bh = nullptr;
  if (s.flags & BMA_MASK_BITMAP) {
    int64_t bh = (int64_t)(b % s.bitmap_B) * s.bitmap_H + (h % s.bitmap_H);
    m.bitmap_bh = s.bitmap + bh * (int64_t)s.bitmap_q * s.bitmap_words;
  }
  m.tile_class_bh = nullptr; m.tile_slot_bh = nullptr; m.tile_bits = nullptr; m.tiles_k = 0;
  if (s.flags & BMA_MASK_TILES) {
    const int64_t bh = ((int64_t)(b % s.tiles_B) * s.tiles_H + (h % s.tiles_H)) * s.tiles_q * s.tiles_k;
    m.tile_class_bh = s.tile_class + bh;
    m.tile_slot_bh = s.tile_slot + bh;
    m.tile_bits = s.tile_bits;
    m.tiles_k = s.tiles_k;
  }
  return m;
}

// TILES term: the 32 keys [gk32, gk32 + 32) (gk32 a multiple of 32) of global query gq as a bit word.
__device__ __forceinline__ uint32_t tiles_word(const MaskView& m, int gq, int gk32) {
  const int64_t t = (int64_t)(gq >> 7) * m.tiles_k + (gk32 >> 7);
  const int c = __ldg(m.tile_class_bh + t);
  if (c != 1) return c == 2 ? 0xffffffffu : 0u;
  const int slot = __ldg(m.tile_slot_bh + t);
  if (slot < 0) return 0u;   // a cut tile that was not stored (the builder ran out of room): nothing is read
  return __ldg(m.tile_bits + ((int64_t)slot * 256 + (gq & 127)) * 4 + ((gk32 & 127) >> 5));
}
// The transposed copy: the 32 queries [gq32, gq32 + 32) (gq32 a multiple of 32) of global key gk.
__device__ __forceinline__ uint32_t tiles_word_t(const MaskView& m, int gk, int gq32) {
  const int64_t t = (int64_t)(gq32 >> 7) * m.tiles_k + (gk >> 7);
  const int c = __ldg(m.tile_class_bh + t);
  if (c != 1) return c == 2 ? 0xffffffffu : 0u;
  const int slot = __ldg(m.tile_slot_bh + t);
  if (slot < 0) return 0u;
  return __ldg(m.tile_bits + ((int64_t)slot * 256 + 128 + (gk & 127)) * 4 + ((gq32 & 127) >> 5));
}

// First key index and one-past-last key index of the reference's block window for the
// query at global index gq (start clamped like XLA's dynamic_slice).
__device__ __forceinline__ void block_window_range(const MaskView& m, int gq, int& k_lo, int& k_hi) {
  int i = gq / m.win_block;
  int total = m.win_left + m.win_right;
  int s = max(0, i - m.win_left);
  s = min(s, m.win_nblk - total);
  k_lo = s * m.win_block;
  k_hi = (s + total) * m.win_block;
}

// mask_fn(b, h, q, k) for local indices q, k (tile offset + lane offset).
__device__ __forceinline__ bool mask_allowed(const MaskView& m, int q, int k) {
  bool ok = (q < m.q_valid) & (k < m.k_valid);
  const int gq = q + m.q_offset, gk = k + m.k_offset;
  if (m.flags & BMA_MASK_CAUSAL) ok &= (gk <= gq);
  if (m.flags & BMA_MASK_BAND) ok &= (gk >= gq - m.band_left) & (gk <= gq + m.band_right);
  if (m.flags & BMA_MASK_BLOCK_WINDOW) {
    int lo, hi;
    block_window_range(m, gq, lo, hi);
    ok &= (gk >= lo) & (gk < hi);
  }
  if ((m.flags & BMA_MASK_SEGMENT) && ok) ok = (__ldg(m.seg_q_row + gq) == __ldg(m.seg_k_row + gk));
  if ((m.flags & BMA_MASK_BITMAP) && ok)
    ok = (__ldg(m.bitmap_bh + (int64_t)gq * m.bitmap_words + (gk >> 5)) >> (gk & 31)) & 1u;
  if ((m.flags & BMA_MASK_TILES) && ok) ok = (tiles_word(m, gq, gk & ~31) >> (gk & 31)) & 1u;
  return ok;
}

// Bit j of the result: ids[j] == ref for j in [0, n) (n <= 32), 0 for j >= n.  `ids` is a run of
// segment ids in global memory; the common aligned full run is read with four-wide loads.
__device__ __forceinline__ uint32_t seg_equal_bits32(const int32_t* ids, int n, int ref) {
  uint32_t w = 0;
  if (n >= 32 && (reinterpret_cast<uintptr_t>(ids) & 15) == 0) {
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
      const int4 v = __ldg(reinterpret_cast<const int4*>(ids) + j4);
      w |= (uint32_t)(v.x == ref) << (j4 * 4);
      w |= (uint32_t)(v.y == ref) << (j4 * 4 + 1);
      w |= (uint32_t)(v.z == ref) << (j4 * 4 + 2);
      w |= (uint32_t)(v.w == ref) << (j4 * 4 + 3);
    }
  } else {
    for (int j = 0; j < 32; ++j)
      if (j < n && __ldg(ids + j) == ref) w |= 1u << j;
  }
  return w;
}

// Bits of the segment and bit-table terms of query row q (local) for the 32 keys starting at local
// key k_start: bit j set = key k_start + j passes both terms.  The interval terms (valid box,
// causal, band, block window) are NOT included; callers AND this with their interval bits.
__device__ __forceinline__ uint32_t table_bits_row32(const MaskView& m, int q, int k_start) {
  uint32_t w = 0xffffffffu;
  if (q >= m.q_valid) return 0u;
  const int gq = q + m.q_offset, gk = k_start + m.k_offset;
  const int n = min(32, m.k_valid - k_start);
  if (n <= 0) return 0u;
  if (m.flags & BMA_MASK_SEGMENT) w &= seg_equal_bits32(m.seg_k_row + gk, n, __ldg(m.seg_q_row + gq));
  if (m.flags & BMA_MASK_BITMAP) {
    const uint32_t* rowp = m.bitmap_bh + (int64_t)gq * m.bitmap_words;
    const int word = gk >> 5, sh = gk & 31;
    uint32_t v = __ldg(rowp + word) >> sh;
    if (sh && word + 1 < m.bitmap_words) v |= __ldg(rowp + word + 1) << (32 - sh);
    w &= v;
  }
  if (m.flags & BMA_MASK_TILES) {   // keys past k_valid fall outside the interval bits the caller ANDs with
    const int sh = gk & 31;
    uint32_t v = tiles_word(m, gq, gk - sh) >> sh;
    if (sh && ((gk - sh + 32) >> 7) < m.tiles_k) v |= tiles_word(m, gq, gk - sh + 32) << (32 - sh);
    w &= v;
  }
  return w;
}

// The same for the 32 queries starting at local query q_start (bit j = query q_start + j) and key row k (local), called by a
// whole warp whose lanes hold 32 consecutive keys.  The bit table is stored by query row: lane j fetches the word of query
// q_start + j that covers the warp's keys, and 32 ballots turn the 32 x 32 bits over (one load a lane; gathering the bits
// of its own key took each lane 32 loads, and the dK/dV kernel 62 us on 2 x 1000 tokens with 16 heads over 4, now 48).
__device__ __forceinline__ uint32_t table_bits_col32(const MaskView& m, int k, int q_start) {
  uint32_t w = 0xffffffffu;
  const int gk = k + m.k_offset, gq = q_start + m.q_offset;
  const int n = min(32, m.q_valid - q_start);
  if (m.flags & BMA_MASK_BITMAP) {
    const int lane = threadIdx.x & 31;
    const int gk0 = gk - lane, word = gk0 >> 5, sh = gk0 & 31;
    uint32_t v = 0;
    if (lane < n && word < m.bitmap_words) {
      const uint32_t* rowp = m.bitmap_bh + (int64_t)(gq + lane) * m.bitmap_words + word;
      v = __ldg(rowp) >> sh;
      if (sh && word + 1 < m.bitmap_words) v |= __ldg(rowp + 1) << (32 - sh);
    }
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const uint32_t col = __ballot_sync(0xffffffffu, (v >> j) & 1u);
      if (lane == j) mine = col;
    }
    w &= mine;
  }
  if (k >= m.k_valid || n <= 0) return 0u;
  if (m.flags & BMA_MASK_SEGMENT) w &= seg_equal_bits32(m.seg_q_row + gq, n, __ldg(m.seg_k_row + gk));
  if (m.flags & BMA_MASK_TILES) {   // every cut tile is stored by key row as well: one word per 32 queries
    const int sh = gq & 31;
    uint32_t v = tiles_word_t(m, gk, gq - sh) >> sh;
    if (sh && n > 32 - sh) v |= tiles_word_t(m, gk, gq - sh + 32) << (32 - sh);
    w &= v;             // queries past q_valid fall outside the interval bits the caller ANDs with
  }
  return w;
}

// Allowed key interval [jlo, jhi] (tile-local, inclusive) of query row q for interval-only masks.
__device__ __forceinline__ void row_interval(const MaskView& m, int q, int k0, int& jlo, int& jhi) {
  if (q >= m.q_valid) { jlo = 1; jhi = 0; return; }
  const int gq = q + m.q_offset;
  int lo = 0, hi = INT32_MAX;
  if (m.flags & BMA_MASK_CAUSAL) hi = min(hi, gq);
  if (m.flags & BMA_MASK_BAND) { lo = max(lo, gq - m.band_left); hi = min(hi, gq + m.band_right); }
  if (m.flags & BMA_MASK_BLOCK_WINDOW) {
    int wlo, whi;
    block_window_range(m, gq, wlo, whi);
    lo = max(lo, wlo);
    hi = min(hi, whi - 1);
  }
  jlo = lo - m.k_offset - k0;
  jhi = min(hi - m.k_offset, m.k_valid - 1) - k0;
}

// Allowed query interval [jlo, jhi] (local to the `width` columns from q0, inclusive) of key row k for masks made of
// interval terms.  The block window of query block i starts at s(i) = clamp(i - left, 0, nblk - total): both ends are
// non-decreasing in i, so the query blocks whose window contains the key form one range, whatever the window's
// block size is relative to the tile.
__device__ __forceinline__ void col_interval(const MaskView& m, int k, int q0, int width, int& jlo, int& jhi) {
  jlo = 0;
  jhi = min(width, m.q_valid - q0) - 1;
  if (k >= m.k_valid) { jlo = 1; jhi = 0; return; }
  const int gk = k + m.k_offset;
  const int base = m.q_offset + q0;  // global index of column 0
  if (m.flags & BMA_MASK_CAUSAL) jlo = max(jlo, gk - base);
  if (m.flags & BMA_MASK_BAND) {  // gq - left <= gk <= gq + right  <=>  gk - right <= gq <= gk + left
    jlo = max(jlo, gk - m.band_right - base);
    jhi = min(jhi, gk + m.band_left - base);
  }
  if (m.flags & BMA_MASK_BLOCK_WINDOW) {
    const int wb = m.win_block, total = m.win_left + m.win_right, last_start = m.win_nblk - total;
    const int kb = gk / wb;            // key block of this key
    const int t = kb - total + 1;      // the window reaches the key iff s(i) >= t ...
    if (t > last_start) { jlo = 1; jhi = 0; return; }
    if (t > 0) jlo = max(jlo, (t + m.win_left) * wb - base);
    if (kb < last_start) jhi = min(jhi, (kb + m.win_left + 1) * wb - 1 - base);   // ... and s(i) <= kb
  }
}

// One block as the interval terms see it: its valid queries and keys by their global indices, and the range of k - q that causal and band
// terms allow.
struct IntervalBox {
  int64_t qa, qb, ka, kb, lo, hi;
  bool empty, whole;    // nothing valid; everything valid
};
__host__ __device__ __forceinline__ IntervalBox interval_box(const bma_mask_spec& s, int q0, int k0, int QB, int KVB) {
  IntervalBox x;
  const int64_t q_end = q0 + (int64_t)QB, k_end = k0 + (int64_t)KVB;
  x.whole = q_end <= s.q_valid && k_end <= s.k_valid;
  x.qa = (int64_t)q0 + s.q_offset; x.qb = (q_end < s.q_valid ? q_end : s.q_valid) - 1 + s.q_offset;
  x.ka = (int64_t)k0 + s.k_offset; x.kb = (k_end < s.k_valid ? k_end : s.k_valid) - 1 + s.k_offset;
  x.empty = x.qb < x.qa || x.kb < x.ka;
  x.lo = INT64_MIN / 4; x.hi = INT64_MAX / 4;
  if (s.flags & BMA_MASK_CAUSAL) x.hi = 0;
  if (s.flags & BMA_MASK_BAND) {
    x.lo = -(int64_t)s.band_left;
    if (s.band_right < x.hi) x.hi = s.band_right;
  }
  return x;
}
// Whether some key of [ka, kb] lies in the allowed range of a query of [qa, qb]: k - q takes every integer value in [ka - qb, kb - qa].
__host__ __device__ __forceinline__ bool interval_any(const IntervalBox& x, int64_t qa, int64_t qb, int64_t ka, int64_t kb) {
  return ka <= kb && (x.lo > ka - qb ? x.lo : ka - qb) <= (x.hi < kb - qa ? x.hi : kb - qa);
}
__host__ __device__ __forceinline__ bool interval_all(const IntervalBox& x) { return x.whole && x.ka - x.qb >= x.lo && x.kb - x.qa <= x.hi; }
// First key of the block window of a query, and the window's width (by global indices).
__host__ __device__ __forceinline__ int64_t window_start(int block, int left, int right, int nblk, int64_t gq) {
  const int64_t st = gq / block - left, last = (int64_t)nblk - left - right;
  return ((st > 0 ? st : 0) < last ? (st > 0 ? st : 0) : last) * block;
}

// Exact any/all of the interval terms (valid box, causal, band, block window) on one block.
// Returns false when the block window changes inside the q block, in which case the caller
// has to scan.  any/all are only meaningful when true is returned.
__device__ __forceinline__ bool interval_classify(const bma_mask_spec& s, int q0, int k0, int QB, int KVB,
                                                  bool& any, bool& all) {
  const IntervalBox x = interval_box(s, q0, k0, QB, KVB);
  any = false; all = false;
  if (x.empty) return true;
  int64_t ka = x.ka, kb = x.kb;  // key range after intersecting with the window (for "any")
  if (s.flags & BMA_MASK_BLOCK_WINDOW) {
    if (x.qa / s.win_block != x.qb / s.win_block) return false;
    const int64_t st = window_start(s.win_block, s.win_left, s.win_right, s.win_nblk, x.qa);
    ka = max(ka, st);
    kb = min(kb, st + ((int64_t)s.win_left + s.win_right) * s.win_block - 1);
  }
  any = interval_any(x, x.qa, x.qb, ka, kb);
  all = ka == x.ka && kb == x.kb && interval_all(x);
  return true;
}

// Class of one block of a mask of interval terms alone, as its elements say: 0 empty, 1 partial, 2 full.  Both ends of the block window
// are non-decreasing in the query.  So the keys of the block's queries lie between the start of the first one's window and the end of the
// last one's, which leaves most blocks empty, and every query sees what lies between the start of the last one's and the end of the first one's.
// The few blocks between the two are decided by runs of queries of one window each.  (A window of 4 blocks of 64 to either side, 4096
// tokens: 160 of 1024 blocks of 128; float32, 8 heads of 64, forward and backward 222 us, 790 with every block of such a row walked as partial.)
// (A function of its own, with values for arguments: inlined or with references it costs the kernels that call it registers or a stack.)
inline __host__ __device__ __noinline__ int window_class(int block, int left, int right, int nblk, IntervalBox x) {
  const int64_t width = ((int64_t)left + right) * block, first = window_start(block, left, right, nblk, x.qa), last = window_start(block, left, right, nblk, x.qb);
  auto any = [&](int64_t qa, int64_t qb, int64_t lo, int64_t hi) { return interval_any(x, qa, qb, x.ka > lo ? x.ka : lo, x.kb < hi ? x.kb : hi); };
  if (!any(x.qa, x.qb, first, last + width - 1)) return 0;
  if (x.ka >= last && x.kb < first + width && interval_all(x)) return 2;
  for (int64_t qa = x.qa; qa <= x.qb;) {
    const int64_t end = (qa / block + 1) * block - 1, qb = end < x.qb ? end : x.qb, st = window_start(block, left, right, nblk, qa);
    if (any(qa, qb, st, st + width - 1)) return 1;
    qa = qb + 1;
  }
  return 0;
}
__host__ __device__ __forceinline__ int interval_class(const bma_mask_spec& s, int qi, int kj, int QB, int KVB) {
  const IntervalBox x = interval_box(s, qi * QB, kj * KVB, QB, KVB);
  if (x.empty) return 0;
  if (s.flags & BMA_MASK_BLOCK_WINDOW) return window_class(s.win_block, s.win_left, s.win_right, s.win_nblk, x);
  return interval_all(x) ? 2 : interval_any(x, x.qa, x.qb, x.ka, x.kb) ? 1 : 0;
}

struct QTileIter {  // flattened walk over (group head, listed q tile), from its entry `skip` on
  const bma_block_lists& l;
  int b, hk, G, kj;
  int g, it, nfull, npart;
  const int32_t* full_idx;
  const int32_t* part_idx;
  __device__ QTileIter(const bma_block_lists& l_, int b_, int hk_, int G_, int kj_, int skip = 0)
      : l(l_), b(b_), hk(hk_), G(G_), kj(kj_), g(-1), it(0), nfull(0), npart(0), full_idx(nullptr), part_idx(nullptr) {
    while (skip > 0) {   // (fewer entries than that is a caller's error: the walk then ends at once)
      if (++g >= G) { it = nfull + npart; return; }
      load_head();
      it = min(skip, nfull + npart);
      skip -= it;
    }
  }
  __device__ void load_head() {
    const int h = hk * G + g;
    const int lb = l.B == 1 ? 0 : b, lh = l.H == 1 ? 0 : h;
    const int64_t row = ((int64_t)lb * l.H + lh) * l.NKV + kj;
    nfull = l.full_q_num[row];
    npart = l.q_num[row];
    full_idx = l.full_q_idx + row * l.NQ;
    part_idx = l.q_idx + row * l.NQ;
    it = 0;
  }
  __device__ void start(int g_, int it_) {   // from entry it_ of head g_ on
    g = g_;
    load_head();
    it = it_;
  }
  __device__ bool next(int& h, int& qi, bool& partial) {
    if (g < 0) { g = 0; load_head(); }
    if (g >= G) return false;
    while (it >= nfull + npart) {
      if (++g >= G) return false;
      load_head();
    }
    h = hk * G + g;
    partial = it >= nfull;
    qi = partial ? part_idx[it - nfull] : full_idx[it];
    ++it;
    return true;
  }
};

// ---- numeric helpers -------------------------------------------------------------------
__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Host-side dispatchers implemented in the individual .cu files.
int simt_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st);
int simt_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st);
// float32 over lists of BMA_F32_TILE blocks
int simt_wide_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st);
int simt_wide_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st);
int sm100_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws, size_t ws_bytes,
              cudaStream_t st);
size_t sm100_fwd_workspace_bytes(const bma_attn_args& a, const bma_block_lists& lists);
bool sm100_fwd_uses_workspace(const bma_attn_args& a, const bma_block_lists& lists);
bool sm100_fwd_wants_lists(const bma_attn_args& a, const bma_mask_spec& spec);
struct BwdPreprocess;
int sm100_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws,
              size_t ws_bytes, const int64_t* visited_host, cudaEvent_t mark, const BwdPreprocess* pre, cudaStream_t st);
size_t sm100_bwd_workspace_bytes(const bma_attn_args& a);
size_t sm100_bwd_scratch_bytes(const bma_attn_args& a, const bma_block_lists& lists, const int64_t* visited_host);
size_t sm100_bwd_scratch_min_bytes(const bma_attn_args& a, const bma_block_lists& lists, const int64_t* visited_host);
// float32 on the tensor core (attn_f32_sm100.cu): 0 where the path does not take the request
size_t f32_workspace_bytes(const bma_attn_args& a, bool backward);
int f32_fwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws, cudaStream_t st);
// own_delta: a.delta is written, from a.o and a.d_o.  Lists without arrays: the mask has interval terms only, and the pass writes them itself.
int f32_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws, bool own_delta, cudaStream_t st);
bool sm100_device();
bool sm100_supported(const bma_attn_args& a);
bool sm100_bwd_supported(const bma_attn_args& a);

// Compact slot addressing of the backward scratch (bwd_slots.cu): tables at the front of the workspace.
// The preprocess that a backward pass has still to run: the arguments with the cotangent as it came, and the bf16 copy to write (or null)
struct BwdPreprocess {
  bma_attn_args a;
  __nv_bfloat16* out;
};
struct SlotTables {
  int64_t* head_base;   // [B*Hq + 1] exclusive prefix of visited blocks over (b, h), row-major
  int64_t* head_total;  // [lists.B * lists.H]
  int32_t* row_base;    // [lists.B, lists.H, NQ] exclusive prefix inside a list head
  int32_t* rank;        // [lists.B, lists.H, NQ, NKV] position of kj among the row's visited tiles, -1 = not visited
  size_t bytes;         // size of the tables (a multiple of 1024); the slots follow
};
SlotTables slot_tables_layout(const bma_attn_args& a, const bma_block_lists& l, void* ws);
// With `pre`: the preprocess too, in the same launch where that can be.
int slot_tables_build(const bma_attn_args& a, const bma_block_lists& l, const SlotTables& t, const BwdPreprocess* pre, cudaStream_t st);
int block_lists_visited(const bma_block_lists& l, int64_t* visited, cudaStream_t st);

constexpr int kSimtTile = 64;
constexpr int kSm100Tile = 128;

}  // namespace bma
