// Backward dK / dV for bf16, head dims 64 and 128, on the sm_100a tensor core (tcgen05 + TMEM + TMA).
// (dQ is produced by a query-major kernel — attn_bwd_dq_replay_sm100.cu from the dS tiles this
// kernel stores, or attn_bwd_dq_sm100.cu by recomputation; splitting the backward in two keeps every
// accumulator in tensor memory: no global reductions, no float32 workspace, and a fixed summation order.)
//
// One CTA per (kv tile of 128 keys, kv head, batch), one CTA per SM (all 512 TMEM columns).  K and
// V of the tile stay in shared memory; the CTA walks the q tiles named by the q-side block lists of
// every query head of the group (full tiles first, then partial ones) and per q tile runs four
// 128x128x128 MMAs:
//     St  = K Q^T            A = K (K-major),  B = Q  (K-major)      -> TMEM [256,384)
//     dPt = V dO^T           A = V (K-major),  B = dO (K-major)      -> TMEM [384,512)
//     dV += Pt dO            A = Pt (bf16 in TMEM, over St),   B = dO (MN-major) -> TMEM [0,128)
//     dK += dSt Q            A = dSt (bf16 in TMEM, over dPt), B = Q  (MN-major) -> TMEM [128,256)
// with Pt = exp2(St*scale*log2e - lse*log2e) and dSt = Pt * (dPt - delta) computed by sixteen warps
// (thread = key row; the four warpgroups split the 128 query columns, 32 each).
//
// Pipelining: MMA order  dV(n) St(n+1) dK(n) dPt(n+1).  Pt and dSt are handed over separately, so dV and the next St run while
// the consumers work on dSt, and dK and the next dPt while they stage dSt and take the exponentials of tile n+1.  Each thread
// writes its Pt and dSt (bf16) over St / dPt columns that it has itself just read, so the consumers never wait for one
// another, nor for a buffer, inside a tile; what overwrites an operand is issued behind the MMAs that read it (MMAs of one
// issuing thread execute in order).  One warp stages lse*log2e and delta of the coming q tiles in shared memory.
// Sixteen warps (four per scheduler, 104 registers each) hide the latencies of tensor memory loads, exponentials and barriers
// that eight warps of 208 registers left open.  Eight warps with one hand-over of Pt and dSt together -> eight with two ->
// sixteen with two: packed documents (B=4 L=16384 H=16 d=128) 1960 -> 1865 -> 1730 us, lambda window 2 x 1000 48 -> 44 ->
// 38 us, sliding window L=8192 464 -> 453 -> 437 us, causal d=64 (B=4 L=4096 H=32) 898 -> 840 -> 848 us; causal B=8 L=4096
// H=32 d=128 stays at 2160 us (3200 cycles per tile, at about 1.5 GHz).
//
// With a scratch buffer (BwdParams::ds_out) the kernel also hands every dSt tile to the dQ kernel:
// each consumer thread stages its 32 dSt values as half of a 128-byte line of a 32 KB tile image laid out
// like a 128-byte-swizzled MMA operand in shared memory, one warp sends the image to its slot with one
// bulk store, and dQ += dS K then needs no recomputation of S and dP (5 instead of 7 MMAs per block
// for the whole backward, paid with 32 KB of HBM traffic each way).
// Every mbarrier wait is bounded; on a timeout the thread records an error code and unwinds.
#include <algorithm>

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace bma {

int sm100_bwd_dq(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, cudaStream_t st);
int sm100_bwd_dq_from_ds(const bma_attn_args& a, const bma_block_lists& lists, const void* ds, const SlotTables& tables,
                         int64_t capacity, int b0, int nb, int hk0, int nhk,
                         cudaStream_t st);

namespace {

using namespace ptx;

constexpr int BT = kSm100Tile;  // the head dimension HD (64 or 128) is a template parameter
constexpr int kCols = 32;                     // query columns of a tile per consumer thread
constexpr int kParts = BT / kCols;
constexpr int kConsumers = 128 * kParts;
constexpr int kThreads = kConsumers + 128;   // + one warpgroup of single-warp roles:
constexpr int kWarpTma = kConsumers / 32, kWarpMma = kWarpTma + 1, kWarpStat = kWarpTma + 2, kWarpHand = kWarpTma + 3;
// Tensor memory column (of St or dPt) of the packed Pt / dSt values of 16-query step ks: a thread packs its 32 columns into
// the first 16 of them.
__device__ constexpr uint32_t packed_col(int ks) { return (uint32_t)((ks >> 1) * kCols + (ks & 1) * 8); }
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kHalfTile = BT * 64 * 2;
template <int HD> constexpr uint32_t kTileBytesOf = (HD / 64) * kHalfTile;  // a [128 x HD] operand tile
constexpr uint32_t kDsBytes = 2 * kHalfTile;  // dSt: [128 keys x 128 queries]
constexpr uint32_t COL_DV = 0, COL_DK = 128, COL_ST = 256, COL_DPT = 384;

enum {
  BAR_KV = 0, BAR_FULLQ0, BAR_FULLQ1, BAR_FULLDO0, BAR_FULLDO1, BAR_STAT0, BAR_STAT1,
  BAR_S1, BAR_S2, BAR_P, BAR_DS, BAR_DK0, BAR_DK1, BAR_DV0, BAR_DV1, BAR_SYNC2, BAR_STG, BAR_DSR,
  NUM_BARS
};

template <int HD>
struct __align__(1024) BwdSmem {
  uint8_t k[kTileBytesOf<HD>];
  uint8_t v[kTileBytesOf<HD>];
  uint8_t ds[kDsBytes];  // staging of the dSt image for the hand-over (not an MMA operand)
  uint8_t q[2][kTileBytesOf<HD>];
  uint8_t d_o[2][kTileBytesOf<HD>];
  float lse2[2][BT];
  float delta[2][BT];
  uint64_t bar[NUM_BARS];
  uint32_t tmem_base;
};

struct BwdParams {
  bma_attn_args a;
  bma_mask_spec spec;
  bma_block_lists l;
  float scale_log2;
  int* status;
  uint8_t* ds_out;  // null, or the slots of kDsBytes: the dSt image of every visited block, addressed compactly:
                    // slot = head_base[b, h] - head_base[first head of the launch] + row_base[qi] + rank[qi][kj]
  const int64_t* head_base;
  const int32_t* row_base;
  const int32_t* rank;
  int64_t capacity; // slots the buffer holds (a slot index beyond it is reported, never written)
  int b0, hk0;      // first batch / kv head of this launch (the grid covers a range when the scratch is smaller
  int nhk;          // than the whole problem), and the number of kv heads in the range
  bool by_rank;     // order of the CTAs, see cta_of
  int parts;        // CTAs of a cluster that share a kv tile's walk
};

// Rendezvous of the kConsumers (512) consumer threads on an mbarrier: arrive, then a bounded wait (a plain
// bar.sync would wait forever for a thread that gave up on an earlier wait).
__device__ __forceinline__ bool consumer_sync(uint64_t* bar, uint32_t parity) {
  mbar_arrive(bar);
  return mbar_wait(bar, parity);
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 640 threads start with 96 registers each: 512 x 104 + 128 x 64 is the same sum
__device__ __forceinline__ void setmaxnreg_inc_consumers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 104;"); }
__device__ __forceinline__ void setmaxnreg_dec_roles() { asm volatile("setmaxnreg.dec.sync.aligned.u32 64;"); }

// dK and dV of a kv tile from the accumulators of a cluster's CTAs, each [128] rows of dK | dV in float32 at `stage`: the rows are dealt out
// over the CTAs, four columns to a thread.
template <int HD> constexpr int kStagePitch = 2 * HD + 4;
template <int HD>
__device__ __noinline__ void sum_parts(const float* stage, const BwdParams& p, int k0, int hk, int b) {
  const bma_attn_args& a = p.a;
  const int part = (int)__clusterRelativeBlockRank();
  constexpr int kPer = 2 * HD / 4;   // groups of four columns of a row
#pragma unroll 1
  for (int i = threadIdx.x; i < (BT + p.parts - 1) / p.parts * kPer; i += kConsumers) {
    const int row = part + p.parts * (i / kPer), c = (i % kPer) * 4;
    if (row >= BT || k0 + row >= a.L) continue;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int src = 0; src < p.parts; ++src) {
      const float4 v = cluster_ld4(cluster_addr(stage + row * kStagePitch<HD> + c, (uint32_t)src));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const bool is_k = c < HD;
    const bma_tensor& t = is_k ? a.dk : a.dv;
    const float f = is_k ? a.scale : 1.f;
    const int64_t off = (int64_t)b * t.stride_b + (int64_t)(k0 + row) * t.stride_l + (int64_t)hk * t.stride_h + (is_k ? c : c - HD);
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(t.ptr) + off) = make_uint2(pack_bf16(s.x * f, s.y * f), pack_bf16(s.z * f, s.w * f));
  }
}

// SHARED: the CTAs of a cluster share a kv tile's walk.  BY_RANK: order of the CTAs of the others, see longest_first.
template <int HD, bool KB, bool SHARED, bool BY_RANK = false>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                const __grid_constant__ CUtensorMap map_dk, const __grid_constant__ CUtensorMap map_dv, const __grid_constant__ BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr uint32_t kTileBytes = kTileBytesOf<HD>;
  BwdSmem<HD>& sm = *reinterpret_cast<BwdSmem<HD>*>(smem_raw);

  const bma_attn_args& a = p.a;
  int kj, hk, b;   // (under a causal mask kv tile 0 sees the most q tiles)
  if constexpr (SHARED) cta_of_cluster(p.by_rank, kj, hk, b);
  else cta_of<BY_RANK>(kj, hk, b);
  hk += p.hk0;
  b += p.b0;
  const int G = a.Hq / a.Hkv;
  const int k0 = kj * BT;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // provably warp-uniform

  if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) report_device_error(p.status, 301);
    return;
  }

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUM_BARS; ++i) {
      uint32_t count = 1;
      if (i == BAR_P || i == BAR_DS || i == BAR_SYNC2 || i == BAR_STG) count = kConsumers;
      if (i == BAR_STAT0 || i == BAR_STAT1) count = 32;
      mbar_init(&sm.bar[i], count);
    }
    fence_barrier_init();
    // K and V of this kv tile do not depend on the block lists: the same thread that initialised the
    // barriers starts their loads at once, under the list reads and the TMEM allocation below
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    mbar_expect_tx(&sm.bar[BAR_KV], 2 * kTileBytes);
#pragma unroll
    for (int box = 0; box < HD / 64; ++box) {
      tma_load_4d(sm.k + box * kHalfTile, &map_k, &sm.bar[BAR_KV], box * 64, hk, k0, b);
      tma_load_4d(sm.v + box * kHalfTile, &map_v, &sm.bar[BAR_KV], box * 64, hk, k0, b);
    }
  }

  int total = 0;  // q tiles this CTA visits
  for (int g = 0; g < G; ++g) {
    const int h = hk * G + g;
    const int lb = p.l.B == 1 ? 0 : b, lh = p.l.H == 1 ? 0 : h;
    const int64_t row = ((int64_t)lb * p.l.H + lh) * p.l.NKV + kj;
    total += p.l.full_q_num[row] + p.l.q_num[row];
  }
  int skip = 0;
  if constexpr (SHARED) {   // this CTA's share of the walk
    const int part = (int)__clusterRelativeBlockRank(), all = total;
    skip = all * part / p.parts;
    total = all * (part + 1) / p.parts - skip;
  }
  if (warp == kWarpTma) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp >= kWarpTma) {
    setmaxnreg_dec_roles();
    if (warp == kWarpTma && lane == 0 && total > 0) {
      // ---------------------------------------------------------------- TMA producer
      prefetch_tensormap(&map_q);
      prefetch_tensormap(&map_do);
      auto load_tile = [&](const CUtensorMap* m, uint8_t* dst, uint64_t* bar, int head, int row0) {
#pragma unroll
        for (int box = 0; box < HD / 64; ++box) tma_load_4d(dst + box * kHalfTile, m, bar, box * 64, head, row0, b);
      };
      QTileIter loader(p.l, b, hk, G, kj, skip);
      bool ok = true;
      for (int n = 0; n < total && ok; ++n) {
        int h, qi; bool partial;
        loader.next(h, qi, partial);
        const int st = n & 1;
        // The Q stage is free once dK += dSt Q of tile n-2 has completed, the dO stage once dV += Pt dO has.  (One barrier
        // per stage: its next phase needs the load that this thread has not issued yet, so a phase cannot be missed.)
        // Q first: it is the operand the next tile needs first (K Q^T), and the one whose load the ring barely covers.
        if (n >= 2) ok = mbar_wait(&sm.bar[BAR_DK0 + st], ((n >> 1) - 1) & 1);
        if (!ok) break;
        mbar_expect_tx(&sm.bar[BAR_FULLQ0 + st], kTileBytes);
        load_tile(&map_q, sm.q[st], &sm.bar[BAR_FULLQ0 + st], h, qi * BT);
        if (n >= 2) ok = mbar_wait(&sm.bar[BAR_DV0 + st], ((n >> 1) - 1) & 1);
        if (!ok) break;
        mbar_expect_tx(&sm.bar[BAR_FULLDO0 + st], kTileBytes);
        load_tile(&map_do, sm.d_o[st], &sm.bar[BAR_FULLDO0 + st], h, qi * BT);
      }
      if (!ok) report_device_error(p.status, 305);
    } else if (warp == kWarpMma && total > 0) {
      // ---------------------------------------------------------------- MMA issuer: the whole warp runs the loop
      // (warp-uniform control flow and descriptors), one elected lane issues the tcgen05 instructions.  A loop run
      // by lane 0 alone costs ~60-70 cycles of issue per MMA under load — no slack against the 64 cycles an MMA takes.
      const bool leader = elect_one();
      constexpr uint32_t idesc_kk = make_idesc_bf16(BT, BT, 0, 0);  // both operands K-major
      constexpr uint32_t idesc_kn = make_idesc_bf16(BT, HD, 0, 1);  // B MN-major
      // descriptors are built once; per MMA only the 16-byte-unit start address moves
      const uint64_t dk = make_smem_desc(smem_u32(sm.k), 16, 1024), dv = make_smem_desc(smem_u32(sm.v), 16, 1024);
      const uint64_t dq0 = make_smem_desc(smem_u32(sm.q[0]), 16, 1024), ddo0 = make_smem_desc(smem_u32(sm.d_o[0]), 16, 1024);
      const uint64_t dqm0 = make_smem_desc(smem_u32(sm.q[0]), kHalfTile, 1024), ddom0 = make_smem_desc(smem_u32(sm.d_o[0]), kHalfTile, 1024);
      constexpr uint32_t kStageUnits = kTileBytes >> 4;
      auto gemm_st = [&](int st) {  // St = K Q^T
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = ((ks >> 2) * kHalfTile + (ks & 3) * 32) >> 4;
          if (leader) mma_ss(tmem + COL_ST, dk + off, dq0 + (uint32_t)(st * kStageUnits + off), idesc_kk, ks > 0);
        }
        if (leader) mma_commit(&sm.bar[BAR_S1]);
      };
      auto gemm_dpt = [&](int st) {  // dPt = V dO^T
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = ((ks >> 2) * kHalfTile + (ks & 3) * 32) >> 4;
          if (leader) mma_ss(tmem + COL_DPT, dv + off, ddo0 + (uint32_t)(st * kStageUnits + off), idesc_kk, ks > 0);
        }
        if (leader) mma_commit(&sm.bar[BAR_S2]);
      };
      bool ok = mbar_wait(&sm.bar[BAR_KV], 0) && mbar_wait(&sm.bar[BAR_FULLQ0], 0);
      if (ok) {
        tc_fence_after();
        gemm_st(0);
        ok = mbar_wait(&sm.bar[BAR_FULLDO0], 0);
        if (ok) { tc_fence_after(); gemm_dpt(0); }
      }
      for (int n = 0; n < total && ok; ++n) {
        const int st = n & 1;
        const uint32_t ph = n & 1;
        ok = mbar_wait(&sm.bar[BAR_P], ph);
        if (!ok) break;
        tc_fence_after();
        // dV += Pt dO      (A from TMEM, 8 columns per 16-query k-step; B = dO rows as K)
#pragma unroll
        for (int ks = 0; ks < BT / 16; ++ks)
          if (leader)
            mma_ts(tmem + COL_DV, tmem + COL_ST + packed_col(ks), ddom0 + (uint32_t)(st * kStageUnits + ks * (2048 >> 4)), idesc_kn, (n > 0) || (ks > 0));
        if (leader) mma_commit(&sm.bar[BAR_DV0 + st]);
        // the next St overwrites the columns Pt was read from; it is queued behind dV += Pt dO
        if (n + 1 < total) {
          ok = mbar_wait(&sm.bar[BAR_FULLQ0 + (st ^ 1)], ((n + 1) >> 1) & 1);
          if (!ok) break;
          tc_fence_after();
          gemm_st(st ^ 1);
        }
        ok = mbar_wait(&sm.bar[BAR_DS], ph);
        if (!ok) break;
        tc_fence_after();
        // dK += dSt Q
#pragma unroll
        for (int ks = 0; ks < BT / 16; ++ks)
          if (leader)
            mma_ts(tmem + COL_DK, tmem + COL_DPT + packed_col(ks), dqm0 + (uint32_t)(st * kStageUnits + ks * (2048 >> 4)), idesc_kn, (n > 0) || (ks > 0));
        if (leader) mma_commit(&sm.bar[BAR_DK0 + st]);
        // the next dPt overwrites the columns dSt was read from; it is queued behind dK += dSt Q
        if (n + 1 < total) {
          ok = mbar_wait(&sm.bar[BAR_FULLDO0 + (st ^ 1)], ((n + 1) >> 1) & 1);
          if (!ok) break;
          tc_fence_after();
          gemm_dpt(st ^ 1);
        }
      }
      if (!ok && leader) report_device_error(p.status, 310);
    } else if (warp == kWarpStat && total > 0) {
      // ---------------------------------------------------------------- row statistics of the coming q tiles
      QTileIter loader(p.l, b, hk, G, kj, skip);
      bool ok = true;
      for (int n = 0; n < total && ok; ++n) {
        int h, qi; bool partial;
        loader.next(h, qi, partial);
        const int st = n & 1;
        // the stage was last read for dSt of tile n-2, which its dK waited for
        if (n >= 2) ok = mbar_wait(&sm.bar[BAR_DK0 + st], ((n >> 1) - 1) & 1);
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int idx = lane * 4 + e;
          const int q = qi * BT + idx;
          const int64_t off = ((int64_t)b * a.Hq + h) * a.N + q;
          const float lv = q < a.N ? __ldg(a.lse + off) : -INFINITY;
          // +inf for rows that attend nothing or lie outside: their probabilities become exactly 0
          sm.lse2[st][idx] = (lv == -INFINITY) ? INFINITY : lv * kLog2e;
          sm.delta[st][idx] = q < a.N ? __ldg(a.delta + off) : 0.f;
        }
        mbar_arrive(&sm.bar[BAR_STAT0 + st]);
      }
      if (!ok && lane == 0) report_device_error(p.status, 315);
    } else if (warp == kWarpHand && p.ds_out != nullptr && total > 0) {
      // ---------------------------------------------------------------- dSt hand-over to the dQ replay kernel
      // BAR_STG says that all consumers have staged (and fenced) the dSt image of tile n in shared memory; one
      // bulk store moves it to its slot, and BAR_DSR tells the consumers that the buffer has been read.
      QTileIter loader(p.l, b, hk, G, kj, skip);
      const uint64_t policy = l2_evict_first();
      const int64_t first_head_base = __ldg(p.head_base + (int64_t)p.b0 * a.Hq + (int64_t)p.hk0 * G);
      bool ok = true;
      for (int n = 0; n < total && ok; ++n) {
        int h, qi; bool partial;
        loader.next(h, qi, partial);
        ok = mbar_wait(&sm.bar[BAR_STG], n & 1);
        if (!ok) break;
        if (lane == 0) {
          const int64_t lrow = ((int64_t)(p.l.B == 1 ? 0 : b) * p.l.H + (p.l.H == 1 ? 0 : h)) * p.l.NQ + qi;
          const int r = __ldg(p.rank + lrow * p.l.NKV + kj);
          const int64_t slot = __ldg(p.head_base + (int64_t)b * a.Hq + h) - first_head_base + __ldg(p.row_base + lrow) + r;
          if (r >= 0 && slot >= 0 && slot < p.capacity) {
            bulk_store_1d(p.ds_out + slot * (int64_t)kDsBytes, sm.ds, kDsBytes, policy);
            bulk_commit();
            bulk_wait_read0();
          } else {
            report_device_error(p.status, 319);   // the two list sides disagree, or the buffer is too small: nothing is written
          }
          mbar_arrive(&sm.bar[BAR_DSR]);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_device_error(p.status, 318);
    }
  } else {
    // ------------------------------------------------------------------ softmax-gradient warps
    setmaxnreg_inc_consumers();
    const int quarter = warp & 3, part = warp >> 2;
    const int row = quarter * 32 + lane;  // TMEM lane == key row of the tile
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t cols = lane_base + part * kCols;   // this thread's query columns of St and dPt
    const int k = k0 + row;
    bool ok = true;
    QTileIter walker(p.l, b, hk, G, kj, skip);
    int h = 0, qi = 0;
    bool partial = false;
    float pr[kCols];  // Pt of the current tile (this thread's key row, its query columns)

    // exponentials of one tile: Pt = exp2(St*c - lse2), handed to the MMA warp over the St columns
    auto exp_phase = [&](int n, int h_, int qi_, bool partial_) -> bool {
      const int st = n & 1;
      const int q0 = qi_ * BT;
      // per-head key bias times this thread's global key index, in log2 units (0 without a bias)
      const float kbk = KB ? __ldg(a.key_bias + h_) * kLog2e * (float)(p.spec.k_offset + k) : 0.f;
      uint32_t bits = 0xffffffffu;
      if (partial_) {
        const MaskView mv = make_mask_view(p.spec, b, h_);
        int jlo, jhi;
        col_interval(mv, k, q0, BT, jlo, jhi);
        const int lo = max(jlo - part * kCols, 0), hi = min(jhi - part * kCols, 31);
        bits = (lo <= hi) ? ((0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) : 0u;
        if (mv.flags & kTableTerms) bits &= table_bits_col32(mv, k, q0 + part * kCols);
      }
      if (!mbar_wait(&sm.bar[BAR_STAT0 + st], (n >> 1) & 1)) return false;
      if (!mbar_wait(&sm.bar[BAR_S1], n & 1)) return false;
      tc_fence_after();
      uint32_t s[32];
      tmem_ld32(tmem + COL_ST + cols, s);
      tmem_wait_ld();
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4) {
        const float4 lv4 = *reinterpret_cast<const float4*>(&sm.lse2[st][part * kCols + j4 * 4]);
        float lv[4] = {lv4.x, lv4.y, lv4.z, lv4.w};
        if constexpr (KB) {  // key bias of this thread's key row: the same shift for every query column
#pragma unroll
          for (int e = 0; e < 4; ++e) lv[e] -= kbk;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) pr[j4 * 4 + e] = ex2(fmaf(__uint_as_float(s[j4 * 4 + e]), p.scale_log2, -lv[e]));
      }
      if (partial_) {
#pragma unroll
        for (int j = 0; j < 32; ++j) pr[j] = (bits >> j) & 1u ? pr[j] : 0.f;
      }
      uint32_t pk[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) pk[j] = pack_bf16(pr[2 * j], pr[2 * j + 1]);
      // Pt takes the place of St values that this very thread has just read: no rendezvous of the consumers is needed
      tmem_st16(tmem + COL_ST + cols, pk);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[BAR_P]);
      return true;
    };

    if (total > 0) {
      walker.next(h, qi, partial);
      ok = exp_phase(0, h, qi, partial);
    }
    for (int n = 0; n < total && ok; ++n) {
      const int st = n & 1;

      // ---- dSt = Pt * (dPt - delta)
      ok = mbar_wait(&sm.bar[BAR_S2], n & 1);
      if (!ok) break;
      tc_fence_after();
      uint32_t dsp[16];
      {
        uint32_t d[32];
        tmem_ld32(tmem + COL_DPT + cols, d);
        tmem_wait_ld();
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 dl4 = *reinterpret_cast<const float4*>(&sm.delta[st][part * kCols + j4 * 4]);
          const float dl[4] = {dl4.x, dl4.y, dl4.z, dl4.w};
          float x[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = pr[j4 * 4 + e] * (__uint_as_float(d[j4 * 4 + e]) - dl[e]);
          dsp[j4 * 2] = pack_bf16(x[0], x[1]);
          dsp[j4 * 2 + 1] = pack_bf16(x[2], x[3]);
        }
      }
      tmem_st16(tmem + COL_DPT + cols, dsp);   // over columns of dPt that this very thread has just read
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.bar[BAR_DS]);
      if (p.ds_out != nullptr) {
        // Hand-over to the dQ replay kernel, off the MMAs' critical path: the thread's dSt values are part of one 128-byte
        // line of the tile image (key row `row`, box of 64 queries, 16-byte chunks swizzled like an MMA operand); the image
        // is staged in shared memory and leaves as one bulk store (warp kWarpHand).  Global stores issued by the consumer
        // warps themselves -- a line per thread, or 512 contiguous bytes per instruction after a turn through shared memory --
        // were measured 25 % and 9 % slower for the whole kernel: 32 KB per tile is more than the load/store path of
        // an SM absorbs without stalling the warps that issue it.
        if (n > 0) ok = mbar_wait(&sm.bar[BAR_DSR], (n - 1) & 1);  // the previous image has been read
        if (!ok) break;
        uint8_t* ds_row = sm.ds + (part >> 1) * kHalfTile + row * 128;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int chunk = ((part & 1) * 4 + u) ^ (row & 7);
          *reinterpret_cast<uint4*>(ds_row + chunk * 16) = make_uint4(dsp[u * 4], dsp[u * 4 + 1], dsp[u * 4 + 2], dsp[u * 4 + 3]);
        }
        fence_proxy_async();  // the bulk store reads the image through the async proxy
        mbar_arrive(&sm.bar[BAR_STG]);
      }

      // ---- exponentials of the next tile while the MMAs of this one run
      if (n + 1 < total) {
        walker.next(h, qi, partial);
        ok = exp_phase(n + 1, h, qi, partial);
      }
    }

    // ---- epilogue: dK (scaled) and dV of this kv tile
    if (ok && total > 0) ok = mbar_wait(&sm.bar[BAR_DK0 + ((total - 1) & 1)], ((total - 1) >> 1) & 1);  // the last MMA of all
    if (ok && total == 0) ok = mbar_wait(&sm.bar[BAR_KV], 0);  // the K/V loads must land before their buffers are reused below
    if (!ok) {
      report_device_error(p.status, 320 + warp);
    } else if constexpr (SHARED) {
      // the accumulators as they are, [128] rows of dK | dV in float32 over all of the tiles; the cluster adds them up below
      if (p.ds_out != nullptr && total > 0) ok = mbar_wait(&sm.bar[BAR_DSR], (total - 1) & 1);   // the last dSt image has been read
      if (!ok) report_device_error(p.status, 340 + warp);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; ok && c < HD / kParts / 16; ++c) {
        const int col = part * (HD / kParts) + c * 16;
        uint32_t rk[16], rv[16];
        if (total > 0) {
          tmem_ld16(tmem + COL_DK + lane_base + col, rk);
          tmem_ld16(tmem + COL_DV + lane_base + col, rv);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) { rk[j] = 0u; rv[j] = 0u; }
        }
        uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<float*>(smem_raw) + row * kStagePitch<HD> + col);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          dst[u] = make_uint4(rk[u * 4], rk[u * 4 + 1], rk[u * 4 + 2], rk[u * 4 + 3]);
          dst[HD / 4 + u] = make_uint4(rv[u * 4], rv[u * 4 + 1], rv[u * 4 + 2], rv[u * 4 + 3]);
        }
      }
    } else {
      tc_fence_after();
      // dK (scaled) and dV go through shared memory -- the K and V tiles are dead now -- in the 128-byte-swizzled
      // box layout and leave as TMA stores of whole lines (rows past the end of the tensor are clipped by the
      // tensor map).  Thread (row, part) owns HD / kParts columns of key row `row`, 16 at a time.
#pragma unroll
      for (int c = 0; c < HD / kParts / 16; ++c) {
        const int col = part * (HD / kParts) + c * 16;
        uint32_t rk[16], rv[16];
        if (total > 0) {
          tmem_ld16(tmem + COL_DK + lane_base + col, rk);
          tmem_ld16(tmem + COL_DV + lane_base + col, rv);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) { rk[j] = 0u; rv[j] = 0u; }
        }
        uint8_t* k_row = sm.k + (col >> 6) * kHalfTile + row * 128;
        uint8_t* v_row = sm.v + (col >> 6) * kHalfTile + row * 128;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = u * 8;
          uint4 ok4, ov4;
          ok4.x = pack_bf16(__uint_as_float(rk[j]) * a.scale, __uint_as_float(rk[j + 1]) * a.scale);
          ok4.y = pack_bf16(__uint_as_float(rk[j + 2]) * a.scale, __uint_as_float(rk[j + 3]) * a.scale);
          ok4.z = pack_bf16(__uint_as_float(rk[j + 4]) * a.scale, __uint_as_float(rk[j + 5]) * a.scale);
          ok4.w = pack_bf16(__uint_as_float(rk[j + 6]) * a.scale, __uint_as_float(rk[j + 7]) * a.scale);
          ov4.x = pack_bf16(__uint_as_float(rv[j]), __uint_as_float(rv[j + 1]));
          ov4.y = pack_bf16(__uint_as_float(rv[j + 2]), __uint_as_float(rv[j + 3]));
          ov4.z = pack_bf16(__uint_as_float(rv[j + 4]), __uint_as_float(rv[j + 5]));
          ov4.w = pack_bf16(__uint_as_float(rv[j + 6]), __uint_as_float(rv[j + 7]));
          const int chunk = (((col & 63) >> 3) + u) ^ (row & 7);
          *reinterpret_cast<uint4*>(k_row + chunk * 16) = ok4;
          *reinterpret_cast<uint4*>(v_row + chunk * 16) = ov4;
        }
      }
      fence_proxy_async();  // the TMA engine reads the staged tiles through the async proxy
      ok = consumer_sync(&sm.bar[BAR_SYNC2], 0);
      if (!ok) {
        report_device_error(p.status, 340 + warp);
      } else if (threadIdx.x == 0) {
#pragma unroll
        for (int box = 0; box < HD / 64; ++box) {
          tma_store_4d(&map_dk, sm.k + box * kHalfTile, box * 64, hk, k0, b);
          tma_store_4d(&map_dv, sm.v + box * kHalfTile, box * 64, hk, k0, b);
        }
        bulk_commit();
        bulk_wait_read0();  // shared memory must stay intact until the stores have read it
      }
    }
  }

  tc_fence_before();
  if constexpr (SHARED) cluster_sync();
  else __syncthreads();
  if (warp == kWarpTma) tmem_dealloc(tmem, kTmemCols);
  if constexpr (SHARED) {
    if (threadIdx.x < kConsumers) sum_parts<HD>(reinterpret_cast<const float*>(smem_raw), p, k0, hk, b);
    cluster_sync();   // shared memory stays until the others have read it
  }
}

bool aligned16(const bma_tensor& t) {
  return t.ptr && (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.stride_b % 8 == 0 && t.stride_l % 8 == 0 && t.stride_h % 8 == 0;
}

}  // namespace

// the query-major dQ kernel keeps a 1024-entry kv list in shared memory (L <= 131072)
bool sm100_bwd_supported(const bma_attn_args& a) { return sm100_supported(a) && ceil_div(a.L, BT) <= 1024; }

size_t sm100_bwd_workspace_bytes(const bma_attn_args&) { return 0; }

// tables + the largest (batch, kv head) unit: the smallest workspace that still takes the hand-over path
size_t sm100_bwd_scratch_min_bytes(const bma_attn_args& a, const bma_block_lists& lists, const int64_t* visited_host);

// A tile of a walk takes 1.7 us; a CTA takes about six tiles more for set-up, drain and the sum over a cluster.  The walks are those of the whole
// call, also in a launch of some of its heads.  (G = 8 query heads of 64 on one kv head, 3 x 1920 tokens, causal: 45 CTAs in 3 parts, the
// call 288 -> 180 us; 1 x 4096, 8/1 heads of 128 562 -> 214; 2 x 4096, 16/4 heads 665 -> 548; host path and launch order included.)
template <typename P>
static int launch_dkdv(const bma_attn_args& a, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                       const CUtensorMap& mdk, const CUtensorMap& mdv, P& p, const Walks& walks, int b0, int nb, int hk0, int nhk, cudaStream_t st) {
  p.b0 = b0; p.hk0 = hk0; p.nhk = nhk;
  p.by_rank = longest_first(ceil_div(a.L, BT), nhk, nb, (int64_t)4 * a.N * a.d * (a.Hq / a.Hkv));
  int rc;
  auto launch = [&](auto by_head, auto by_rank, auto shared, size_t smem) -> int {
    static ClusterCounts known[2][2];
    p.parts = walks.ctas > 4 * kSms ? 1 : share_walks(walks, 6.0, kMaxParts, [&](int parts) { return clusters_at_once(known[a.d == 128][a.key_bias != nullptr], shared, kThreads, smem, parts); });
    const auto kernel = p.parts > 1 ? shared : p.by_rank ? by_rank : by_head;
    BMA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = cta_grid(p.by_rank, ceil_div(a.L, BT), nhk, nb, p.parts);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = cluster_attribute(p.parts);
    if (p.parts > 1) { cfg.attrs = &attr; cfg.numAttrs = 1; }
    BMA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, mq, mk, mv, mdo, mdk, mdv, static_cast<const BwdParams&>(p)));
    return BMA_OK;
  };
  if (a.d == 128) rc = a.key_bias ? launch(bwd_dkdv_kernel<128, true, false>, bwd_dkdv_kernel<128, true, false, true>, bwd_dkdv_kernel<128, true, true>, sizeof(BwdSmem<128>))
                                  : launch(bwd_dkdv_kernel<128, false, false>, bwd_dkdv_kernel<128, false, false, true>, bwd_dkdv_kernel<128, false, true>, sizeof(BwdSmem<128>));
  else rc = a.key_bias ? launch(bwd_dkdv_kernel<64, true, false>, bwd_dkdv_kernel<64, true, false, true>, bwd_dkdv_kernel<64, true, true>, sizeof(BwdSmem<64>))
                       : launch(bwd_dkdv_kernel<64, false, false>, bwd_dkdv_kernel<64, false, false, true>, bwd_dkdv_kernel<64, false, true>, sizeof(BwdSmem<64>));
  if (rc) return rc;
  count_launches(1, p.parts);
  BMA_CUDA_TRY(cudaGetLastError());
  return BMA_OK;
}

// Visited blocks of one query head: from the caller's per-list-head counts, or the dense bound without them.
static int64_t head_blocks(const bma_attn_args& a, const bma_block_lists& l, const int64_t* visited, int b, int h) {
  if (!visited) return (int64_t)ceil_div(a.N, BT) * ceil_div(a.L, BT);
  return visited[(int64_t)(l.B == 1 ? 0 : b) * l.H + (l.H == 1 ? 0 : h)];
}
static int64_t unit_blocks(const bma_attn_args& a, const bma_block_lists& l, const int64_t* visited, int b, int hk) {
  const int G = a.Hq / a.Hkv;
  int64_t n = 0;
  for (int g = 0; g < G; ++g) n += head_blocks(a, l, visited, b, hk * G + g);
  return n;
}
// tables + one dSt image (32 KB) per visited block of the whole problem
size_t sm100_bwd_scratch_bytes(const bma_attn_args& a, const bma_block_lists& lists, const int64_t* visited_host) {
  if (lists.NKV > 1024 || lists.NQ <= 0 || lists.B <= 0 || lists.H <= 0) return 0;
  int64_t blocks = 0;
  for (int b = 0; b < a.B; ++b)
    for (int hk = 0; hk < a.Hkv; ++hk) blocks += unit_blocks(a, lists, visited_host, b, hk);
  return slot_tables_layout(a, lists, nullptr).bytes + (size_t)blocks * kDsBytes;
}

size_t sm100_bwd_scratch_min_bytes(const bma_attn_args& a, const bma_block_lists& lists, const int64_t* visited_host) {
  if (lists.NKV > 1024 || lists.NQ <= 0 || lists.B <= 0 || lists.H <= 0) return 0;
  int64_t largest = 0;
  for (int b = 0; b < a.B; ++b)
    for (int hk = 0; hk < a.Hkv; ++hk) largest = std::max(largest, unit_blocks(a, lists, visited_host, b, hk));
  return slot_tables_layout(a, lists, nullptr).bytes + (size_t)std::max<int64_t>(largest, 1) * kDsBytes;
}

int sm100_bwd(const bma_attn_args& a, const bma_mask_spec& spec, const bma_block_lists& lists, void* ws, size_t ws_bytes,
              const int64_t* visited_host, cudaEvent_t mark, const BwdPreprocess* pre, cudaStream_t st) {
  BMA_REQUIRE(lists.q_block == BT && lists.kv_block == BT && lists.q_num, BMA_ERR_ARG);
  BMA_REQUIRE(a.d_o.dtype == BMA_DTYPE_BF16, BMA_ERR_UNSUPPORTED);  // bma_attn_bwd_preprocess provides the bf16 copy
  BMA_REQUIRE(aligned16(a.d_o) && aligned16(a.dq) && aligned16(a.dk) && aligned16(a.dv), BMA_ERR_UNSUPPORTED);

  CUtensorMap mq, mk, mv, mdo;
  int rc;
  if ((rc = make_tile_map_bf16(&mq, a.q.ptr, a.B, a.N, a.Hq, a.d, a.q.stride_b, a.q.stride_l, a.q.stride_h, BT))) return rc;
  if ((rc = make_tile_map_bf16(&mk, a.k.ptr, a.B, a.L, a.Hkv, a.d, a.k.stride_b, a.k.stride_l, a.k.stride_h, BT))) return rc;
  if ((rc = make_tile_map_bf16(&mv, a.v.ptr, a.B, a.L, a.Hkv, a.d, a.v.stride_b, a.v.stride_l, a.v.stride_h, BT))) return rc;
  if ((rc = make_tile_map_bf16(&mdo, a.d_o.ptr, a.B, a.N, a.Hq, a.d, a.d_o.stride_b, a.d_o.stride_l, a.d_o.stride_h, BT))) return rc;
  CUtensorMap mdk, mdv;
  if ((rc = make_tile_map_bf16(&mdk, a.dk.ptr, a.B, a.L, a.Hkv, a.d, a.dk.stride_b, a.dk.stride_l, a.dk.stride_h, BT))) return rc;
  if ((rc = make_tile_map_bf16(&mdv, a.dv.ptr, a.B, a.L, a.Hkv, a.d, a.dv.stride_b, a.dv.stride_l, a.dv.stride_h, BT))) return rc;

  BwdParams p;
  p.a = a; p.spec = spec; p.l = lists;
  p.scale_log2 = a.scale * kLog2e;
  p.status = device_status_ptr();
  BMA_REQUIRE(p.status != nullptr, BMA_ERR_CUDA);
  p.ds_out = nullptr; p.head_base = nullptr; p.row_base = nullptr; p.rank = nullptr; p.capacity = 0;
  // A scratch buffer switches the dQ pass from recomputation to replaying the dSt tiles.  Behind the slot tables it
  // must hold at least the largest (batch, kv head) unit; when it is smaller than the whole problem the backward runs
  // as consecutive launches over ranges of whole batches (or, inside a batch that does not fit, of kv heads) that reuse
  // the slots.  Unit sizes come from the caller's visited-block counts (the dense bound without them); the kernels
  // address compactly either way, so a range never needs more than the host planned for it.
  const bool lists_fit = lists.NQ == ceil_div(a.N, BT) && lists.NKV == ceil_div(a.L, BT) && lists.NKV <= 1024;
  SlotTables tables = slot_tables_layout(a, lists, ws);
  int64_t capacity = 0;
  if (ws != nullptr && (reinterpret_cast<uintptr_t>(ws) & 255) == 0 && ws_bytes > tables.bytes && lists_fit)
    capacity = (int64_t)((ws_bytes - tables.bytes) / kDsBytes);
  int64_t largest = 0;
  for (int b = 0; b < a.B; ++b)
    for (int hk = 0; hk < a.Hkv; ++hk) largest = std::max(largest, unit_blocks(a, lists, visited_host, b, hk));
  const bool hand_over = capacity >= 1 && largest <= capacity;
  const bool many = (int64_t)ceil_div(a.L, BT) * a.Hkv * a.B > 4 * kSms;   // waves: nothing is shared
  const Walks walks = many ? Walks{4 * kSms + 1} : k_walks(a, spec);
  if (!hand_over) {
    if (pre && (rc = bma_attn_bwd_preprocess(&pre->a, pre->out, st))) return rc;
    rc = launch_dkdv(a, mq, mk, mv, mdo, mdk, mdv, p, walks, 0, a.B, 0, a.Hkv, st);
    if (rc) return rc;
    if (mark) BMA_CUDA_TRY(cudaEventRecord(mark, st));
    return sm100_bwd_dq(a, spec, lists, st);
  }
  if ((rc = slot_tables_build(a, lists, tables, pre, st))) return rc;
  p.ds_out = static_cast<uint8_t*>(ws) + tables.bytes;
  p.head_base = tables.head_base; p.row_base = tables.row_base; p.rank = tables.rank;
  p.capacity = capacity;
  bool first = true;
  auto run_range = [&](int b0, int nb, int hk0, int nhk, bool whole) -> int {
    int r = launch_dkdv(a, mq, mk, mv, mdo, mdk, mdv, p, walks, b0, nb, hk0, nhk, st);
    if (r) return r;
    if (mark && first && whole) BMA_CUDA_TRY(cudaEventRecord(mark, st));   // one boundary only when one range covers everything
    first = false;
    return sm100_bwd_dq_from_ds(a, lists, p.ds_out, tables, capacity, b0, nb, hk0, nhk, st);
  };
  auto batch_blocks = [&](int b) {
    int64_t n = 0;
    for (int hk = 0; hk < a.Hkv; ++hk) n += unit_blocks(a, lists, visited_host, b, hk);
    return n;
  };
  for (int b0 = 0; b0 < a.B;) {
    int nb = 0;
    int64_t used = 0;
    while (b0 + nb < a.B && used + batch_blocks(b0 + nb) <= capacity) used += batch_blocks(b0 + nb++);
    if (nb >= 1) {
      if ((rc = run_range(b0, nb, 0, a.Hkv, nb == a.B))) return rc;
      b0 += nb;
      continue;
    }
    for (int hk0 = 0; hk0 < a.Hkv;) {   // this batch alone does not fit: ranges of its kv heads
      int nhk = 0;
      used = 0;
      while (hk0 + nhk < a.Hkv && used + unit_blocks(a, lists, visited_host, b0, hk0 + nhk) <= capacity)
        used += unit_blocks(a, lists, visited_host, b0, hk0 + nhk++);
      if ((rc = run_range(b0, 1, hk0, nhk, false))) return rc;   // nhk >= 1: the largest unit fits
      hk0 += nhk;
    }
    b0 += 1;
  }
  return BMA_OK;

}

}  // namespace bma
