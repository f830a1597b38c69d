// Single-kernel backward of the softmax RBF attention for head dim 64 (sm_100a).
//
// A CTA owns 128 keys (K, V resident in shared memory) and streams the query tiles (Q, dO) past them. Per
// query tile it issues five MMAs - the algorithmic minimum - and evaluates every exponential once:
//   S^T  = K Q^T  (+ bias slab: -L[query] / scale)        smem x smem -> TMEM
//   dP^T = V dO^T (+ bias slab: -delta[query])            smem x smem -> TMEM
//   P^T  = exp2(S^T * 2c - ksq[key]),   dS^T = P^T * dP^T                        (registers)
//   dV  += P^T  dO               TMEM x smem   (P^T written to TMEM as 16-bit pairs)
//   dK  += dS^T Q                smem x smem   (dS^T stored to shared memory as a [key][query] tile)
//   dQ_partial = dS K            smem x smem   (the same tile read as an M-major A operand)
// The per-query statistics L and delta never pass through registers: the pre-pass stores them as three 16-bit
// parts per query ("bias slabs") and S^T / dP^T get one extra K = 16 MMA step against a slab of constants.
// dQ_partial leaves the CTA as fp32 reduce-adds into an accumulator in global memory; a small kernel converts it
// to the output type (times 2g) afterwards. dK gets the norm-gradient term on its way out:
// dK = 2g (acc - rowsum(dS^T)[key] * k).
//
// Roles: warps 0, 1, 3 MMA issuers (one thread sustains one MMA per ~60 cycles, the tensor pipe retires an N = 64
// product in 32; five issuers, one per product, measured slower than three), warp 2 TMA producer, warps 4-19 compute
// (thread = key row; group g owns query columns [32g, 32g+32) of the tile), warps 20-23 drain dQ_partial of every step
// and dV, dK of every item (thread = query / key row). Compute warpgroups take registers from the others.
//   issuer A: S^T(n+1) when P^T(n) is in TMEM (S^T(n) has been read by then)
//   issuer B: dV(n) when P^T(n) is in TMEM; dP^T(n+1) when dS^T(n) is in shared memory (dP^T(n) has been read by then)
//   issuer C: dK(n) when dS^T(n) is in shared memory, dQ_partial(n) when also dQ_partial(n-1) has been read by the drain
// A commit covers all MMAs its thread has issued before, so the products are ordered such that three waits (S^T; dP^T,
// which covers dV(n-1), that is the P^T columns; dQ(n-1), which covers dK(n-1), that is the dS^T tile) and two arrivals
// (P^T, dS^T) per step are enough. What bounds the kernel: the compute warps' own chain of a step (about 2900 clocks;
// traced, their waits are over when they get to them), in which TMEM and shared-memory latencies stretch with the MMA
// operand traffic; taking all MMAs out shortens the whole backward by 22 %, the exponentials by 4 %, the drain by 6 %.
// Between items they only wait for the next scores: the drain warps finish dK and dV. Measured against one item at a
// time with the epilogue on the compute warps (backward call, B8 H16 N4096 causal: 926 -> 897 us; B4 H12 N1000 full:
// 67.0 -> 61.4 us; N8192 B4 H16 training pass 2.71 -> 2.64 ms; N1028 B64 H8 about 480 us as before, bound by how
// fast loads and drains of items of five steps on average follow each other). With the short waits and the issue loops of
// four, which are less code: 892 -> 860 us and, at N1028, 453 -> 387 us (one box, replayed back to back).
// TMEM columns: S^T [0,128), dP^T [128,256), P^T [256,320), dV [320,384), dK [384,448), dQ_partial [448,512).
#include "common.cuh"
#include "launch.h"

namespace rbf {

namespace bwdf {


static constexpr int D = 64;
static constexpr int kThreads = 768;
static constexpr int kNumComputeWarps = 16;
static constexpr int kMmaWarpA = 0;
static constexpr int kMmaWarpB = 1;
static constexpr int kLoadWarp = 2;
static constexpr int kMmaWarpC = 3;
static constexpr int kComputeWarp0 = 4;
static constexpr int kDrainWarp0 = 20;
// Register budget: the launch allocates 80 per thread (768 threads); setmaxnreg may only redistribute that
// total: 512 * 96 + 128 * 32 + 128 * 64 = 768 * 80. (An increase beyond what the decreases released blocks
// forever, with no timeout.) The drain warps lag behind on short items; with 56 registers, dK finished after the last
// dQ_partial and scalar arithmetic the backward call took 42.2 us (now 41.1) at B4 H8 N1024, 62.6 (61.4) at B4 H12 N1000
// full, 907 (897) at B8 H16 N4096.
static constexpr int kComputeRegs = 96;
static constexpr int kOtherRegs = 32;
static constexpr int kDrainRegs = 64;
static_assert(512 * kComputeRegs + 128 * kOtherRegs + 128 * kDrainRegs <= 768 * 80, "setmaxnreg budget");
static constexpr int kDqBoxBytes = 32 * 128;        // 4 KB: 32 rows of 128 bytes of one drain warp

static constexpr int kTileBytes = kTile * D * 2;    // 16 KB: one 128 x 64 16-bit tile
static constexpr int kSlabBytes = kTile * 32;       // 4 KB: 128 rows x 16 x 16-bit
static constexpr int kQStages = 3;                  // ring of Q tiles (+ L slabs): a tile lives from S^T to dK
static constexpr int kDoStages = 2;                 // ring of dO tiles (+ delta slabs): from dP^T to dV
static constexpr int kDsBytes = kTile * kTile * 2;  // 32 KB: dS^T as [key][query], two 64-query boxes

struct Smem {
  static constexpr int kK = 0;                                 // two tiles: the current item's and the next one's
  static constexpr int kV = kK + 2 * kTileBytes;               // one tile: dead after the item's last dP^T
  static constexpr int kQ = kV + kTileBytes;
  static constexpr int kDo = kQ + kQStages * kTileBytes;
  static constexpr int kDs = kDo + kDoStages * kTileBytes;
  static constexpr int kLSlab = kDs + kDsBytes;
  static constexpr int kDSlab = kLSlab + kQStages * kSlabBytes;
  static constexpr int kOnes = kDSlab + kDoStages * kSlabBytes;
  static constexpr int kOutStage = kOnes + kSlabBytes;         // 32 KB: four drain warps, two 4 KB boxes each
  static constexpr int kRowsum = kOutStage + 8 * kDqBoxBytes;  // [2][4 groups][128] floats: partial row sums of an item
  static constexpr int kKsq = kRowsum + 2 * 4 * kTile * 4;     // [2][128] floats: key norms of the two K tiles
  static constexpr int kBars = kKsq + 2 * kTile * 4;
  static constexpr int kItemSlots = 4;                         // ring of work items, producer -> all other roles
  static constexpr int kNumBars = 6 + 2 * kQStages + 2 * kDoStages + 12 + 2 * kItemSlots;
  static constexpr int kMisc = kBars + kNumBars * 8;
  static constexpr int kItems = kMisc + 16;
  static constexpr int kTotal = kItems + 16 * kItemSlots;
  static constexpr int kDynamic = kTotal + 1024;
};
static_assert(Smem::kBars % 16 == 0 && Smem::kItems % 16 == 0 && Smem::kDynamic <= 232448, "shared memory layout");

static constexpr int kColS = 0, kColDP = 128, kColPT = 256, kColDV = 320, kColDK = 384, kColDQ = 448;

enum Site : uint32_t {
  kSiteKFull = 64, kSiteVFull, kSiteQFull, kSiteDoFull, kSiteQEmpty, kSiteDoEmpty, kSiteSFull, kSiteDPFull, kSitePFull,
  kSiteDSFull, kSiteDQFull, kSiteDQDrained, kSiteDVAcc, kSiteDKAcc, kSiteDVFree, kSiteDKFree, kSiteDsFree, kSiteRowsum,
  kSiteKFree, kSiteVFree, kSiteItemFull, kSiteItemEmpty
};

struct Params {
  const float* ksq;      // (B*H, n_pad), +inf on padding rows
  DeviceStatus* status;
  unsigned int* work;    // [0] items taken beyond the CTAs' first, [1] CTAs that have left; zero at launch and at its end
  int total_items;       // key tiles x (batch, head) pairs
  int plain_heads, group;   // order of the items (decode_item)
  int H, N, n_pad, causal;
  float scale2, grad_scale, slab_w;
};

// The launch is persistent and its items overlap: a CTA per SM, each starting with item blockIdx.x and taking further
// (key tile, batch-head) items from a global counter, in decode_item's order. TMEM, the barriers (their phases run on) and
// the Q / dO rings carry on from item to item; K and the key norms have two buffers, V is reloaded as soon as the item's last dP^T has read it, and the drain warps
// bring dK and dV out, so that the compute warps - the critical resource - go straight on to the next item's scores.
template <bool kBf16>
__global__ void __launch_bounds__(kThreads, 1)
rbf_bwd_fused_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                     const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                     const __grid_constant__ CUtensorMap tm_lslab, const __grid_constant__ CUtensorMap tm_dslab,
                     const __grid_constant__ CUtensorMap tm_dq_acc, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_k = smem + Smem::kK;
  uint8_t* s_v = smem + Smem::kV;
  uint8_t* s_q = smem + Smem::kQ;
  uint8_t* s_do = smem + Smem::kDo;
  uint8_t* s_ds = smem + Smem::kDs;
  uint8_t* s_lslab = smem + Smem::kLSlab;
  uint8_t* s_dslab = smem + Smem::kDSlab;
  uint8_t* s_ones = smem + Smem::kOnes;
  uint8_t* s_out = smem + Smem::kOutStage;
  float* s_rowsum = reinterpret_cast<float*>(smem + Smem::kRowsum);
  const float* s_ksq = reinterpret_cast<const float*>(smem + Smem::kKsq);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::kBars);
  uint64_t* k_full = bars;                   // [2] K tile and key norms of an item landed
  uint64_t* k_free = k_full + 2;             // [2] the item's last dQ_partial is drained (nothing reads K any more)
  uint64_t* v_full = k_free + 2;
  uint64_t* v_free = v_full + 1;             // the item's last dP^T has completed
  uint64_t* q_full = v_free + 1;             // [kQStages] Q tile + L slab landed
  uint64_t* q_empty = q_full + kQStages;     // dK has completed (it follows S^T)
  uint64_t* do_full = q_empty + kQStages;    // [kDoStages] dO tile + delta slab landed
  uint64_t* do_empty = do_full + kDoStages;  // dV has completed (it follows dP^T)
  uint64_t* s_full = do_empty + kDoStages;   // S^T(n) complete
  uint64_t* dp_full = s_full + 1;            // dP^T(n) and dV(n-1) complete: the P^T columns may be overwritten
  uint64_t* p_full = dp_full + 1;            // P^T(n) stored to TMEM, S^T(n) read
  uint64_t* ds_full = p_full + 1;            // dS^T(n) stored to shared memory, dP^T(n) read
  uint64_t* dq_full = ds_full + 1;           // dK(n) and dQ_partial(n) complete: dS^T tile free, dQ_partial readable
  uint64_t* dq_drained = dq_full + 1;        // drain warps have read dQ_partial(n) out of TMEM
  uint64_t* dv_acc = dq_drained + 1;         // the item's dV is complete
  uint64_t* dk_acc = dv_acc + 1;             // the item's dK is complete
  uint64_t* dv_free = dk_acc + 1;            // drain warps have read dV out of TMEM
  uint64_t* dk_free = dv_free + 1;           // drain warps have read dK out of TMEM
  uint64_t* rs_full = dk_free + 1;           // [2] the item's row sums of dS^T are in shared memory
  uint64_t* item_full = rs_full + 2;         // [kItemSlots] the producer has published the CTA's n-th item
  uint64_t* item_empty = item_full + Smem::kItemSlots;   // [kItemSlots] every other role has read it
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + Smem::kMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Smem::kMisc + 4);
  volatile int* s_item = reinterpret_cast<volatile int*>(smem + Smem::kMisc + 8);   // item a status word names
  volatile int4* s_items = reinterpret_cast<volatile int4*>(smem + Smem::kItems);   // {key tile (< 0: end), bh, b, h}

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int n_tiles = (p.N + kTile - 1) / kTile;
  // Every role walks the CTA's items by itself and keeps two counters: T counts the steps of its earlier items (step n of
  // the item is global step T + n: per-step barriers are in phase (T + n) & 1, a ring of R stages is at stage (T + n) % R
  // in phase ((T + n) / R) & 1), I counts the earlier items (per-item barriers are in phase I & 1; K buffer and row sums
  // I & 1 in phase (I >> 1) & 1; item slot I % kItemSlots in phase (I / kItemSlots) & 1).
  uint32_t T = 0, I = 0;
  // the current work item
  int bh = 0, b = 0, h = 0;
  int kt = 0;                                      // key tile; tile 0 is the heaviest under the causal mask
  int k_row0 = 0;
  int first = 0;                                   // first query tile that sees these keys
  int cnt = 0;
  auto set_tile = [&](int tile) {
    kt = tile;
    k_row0 = kt * kTile;
    first = p.causal ? kt : 0;
    cnt = n_tiles - first;
  };
  auto set_item = [&](int item) {
    int tile;
    decode_item(item, n_tiles, p.plain_heads, p.group, bh, tile);
    b = bh / p.H;
    h = bh % p.H;
    set_tile(tile);
  };
  // The next item as the issuer, drain and compute warps see it; false at the end of the sequence or when the launch is
  // being abandoned.
  constexpr int kItemReaders = 3 + 4 + kNumComputeWarps;
  auto next_item = [&]() -> bool {
    const int slot = I % Smem::kItemSlots;
    if (!mbar_wait_warp(&item_full[slot], (I / Smem::kItemSlots) & 1, abort_flag, kSiteItemFull))
      return false;
    const int tile = s_items[slot].x;
    bh = s_items[slot].y;
    b = s_items[slot].z;
    h = s_items[slot].w;
    mbar_arrive_warp(&item_empty[slot]);
    if (tile < 0) return false;
    set_tile(tile);
    return true;
  };
  auto publish_item = [&](bool more) {             // the producer's counterpart; I is the published item's number
    const int slot = I % Smem::kItemSlots;
    s_items[slot].x = more ? kt : -1;
    s_items[slot].y = bh;
    s_items[slot].z = b;
    s_items[slot].w = h;
    mbar_arrive(&item_full[slot]);
  };

  auto load_k = [&]() {
    const int kb = I & 1;
    mbar_arrive_expect_tx(&k_full[kb], kTileBytes + kTile * 4);
    tma_load_4d(s_k + kb * kTileBytes, &tm_k, &k_full[kb], 0, k_row0, h, b);
    bulk_load_1d(smem + Smem::kKsq + kb * kTile * 4, p.ksq + static_cast<int64_t>(bh) * p.n_pad + k_row0, kTile * 4,
                 &k_full[kb]);
  };
  auto load_v = [&]() {
    mbar_arrive_expect_tx(v_full, kTileBytes);
    tma_load_4d(s_v, &tm_v, v_full, 0, k_row0, h, b);
  };
  auto load_q = [&](int n) {
    const int row0 = (first + n) * kTile, st = (T + n) % kQStages;
    mbar_arrive_expect_tx(&q_full[st], kTileBytes + kSlabBytes);
    tma_load_4d(s_q + st * kTileBytes, &tm_q, &q_full[st], 0, row0, h, b);
    tma_load_3d(s_lslab + st * kSlabBytes, &tm_lslab, &q_full[st], 0, row0, bh);
  };
  auto load_do = [&](int n) {
    const int row0 = (first + n) * kTile, st = (T + n) % kDoStages;
    mbar_arrive_expect_tx(&do_full[st], kTileBytes + kSlabBytes);
    tma_load_4d(s_do + st * kTileBytes, &tm_do, &do_full[st], 0, row0, h, b);
    tma_load_3d(s_dslab + st * kSlabBytes, &tm_dslab, &do_full[st], 0, row0, bh);
  };
  // The producer warp sets the CTA up: it reads the launch's status word (a wait that ran out in an earlier CTA ends the
  // whole launch quickly: later CTAs leave at once), initialises the barriers while that load is in flight, and issues
  // the first loads before the CTA-wide synchronisation, so that K, V and the first query tiles travel while TMEM is
  // allocated and the constant slab is written.
  if (warp == kLoadWarp) {
    for (int i = lane; i < Smem::kNumBars; i += 32) {
      uint64_t* bar = &bars[i];
      uint32_t count = 1;                          // one MMA commit, TMA producer or publishing thread
      if (bar == p_full || bar == ds_full || bar == rs_full || bar == rs_full + 1) count = kNumComputeWarps;
      if (bar == dq_drained || bar == dv_free || bar == dk_free || bar == k_free || bar == k_free + 1) count = 4;
      if (bar >= item_empty) count = kItemReaders;
      mbar_init(bar, count);
    }
    fence_mbar_init();
    __syncwarp();
    if (lane == 0) {
      // the loads below complete on barriers that other lanes have just initialised; besides the warp-level
      // synchronisation, order those generic-proxy writes before this thread's async-proxy operations
      fence_proxy_async_smem();
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_do);
      tma_prefetch_desc(&tm_lslab);
      tma_prefetch_desc(&tm_dslab);
      grid_dependency_wait();                      // the pre-pass: slabs, norms, cleared accumulator, status word, counters
      const unsigned int earlier = *reinterpret_cast<volatile unsigned int*>(&p.status->code);
      *s_item = static_cast<int>(blockIdx.x);
      *abort_flag = earlier != 0u ? 1 : 0;
      if (earlier == 0u) {
        set_item(static_cast<int>(blockIdx.x));    // the launch never has more CTAs than items
        load_k();
        load_q(0);
        load_v();
        load_do(0);
        if (cnt > 1) {
          load_q(1);
          load_do(1);
        }
        publish_item(true);
      }
    }
  }
  if (warp == kMmaWarpA) {
    tmem_alloc(tmem_base_s, 512);
    tmem_relinquish();
  }
  if (tid < kTile) {
    // slab of constants (A operand of the bias-slab MMA steps): rows [w, w, w, 0 x5 | w, w, w, 0 x5]
    const uint4 v = make_uint4(pack2<kBf16>(p.slab_w, p.slab_w), pack2<kBf16>(p.slab_w, 0.f), 0u, 0u);
    *reinterpret_cast<uint4*>(s_ones + tid * 32) = v;
    *reinterpret_cast<uint4*>(s_ones + tid * 32 + 16) = v;
    fence_proxy_async_smem();
  }
  grid_dependency_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_base_s;
  const bool run = *abort_flag == 0;
  const bool queue = static_cast<int>(gridDim.x) < p.total_items;   // else: one item per CTA, no counter traffic

  if (warp < kComputeWarp0) {
    setmaxnreg_dec<kOtherRegs>();
  }
  if (warp == kLoadWarp) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0 && run) {
      bool ok = true;
      while (true) {
        if (I > 0) {
          // the K buffer's previous user is two items back
          if (I > 1) ok = mbar_wait(&k_free[I & 1], ((I >> 1) - 1) & 1, abort_flag, kSiteKFree);
          if (!ok) break;
          load_k();
        }
        for (int n = I == 0 ? 2 : 0; n < cnt; ++n) {
          const uint32_t g = T + n;
          if (g >= kQStages)
            ok = mbar_wait(&q_empty[g % kQStages], ((g / kQStages) - 1) & 1, abort_flag, kSiteQEmpty);
          if (!ok) break;
          load_q(n);
          if (n == 0) {
            ok = mbar_wait(v_free, (I - 1) & 1, abort_flag, kSiteVFree);
            if (!ok) break;
            load_v();
          }
          if (g >= kDoStages)
            ok = mbar_wait(&do_empty[g % kDoStages], ((g / kDoStages) - 1) & 1, abort_flag, kSiteDoEmpty);
          if (!ok) break;
          load_do(n);
        }
        if (!ok) break;
        T += cnt;
        ++I;
        // the next item is taken only now, with all loads of this one issued: taking items earlier leaves the launch's
        // last items reserved by CTAs that are still busy
        int item = p.total_items;
        if (queue) item = static_cast<int>(gridDim.x + atomicAdd(&p.work[0], 1u));
        const bool more = item < p.total_items;
        if (more) set_item(item);
        const int slot = I % Smem::kItemSlots;
        if (I >= Smem::kItemSlots &&
            !mbar_wait(&item_empty[slot], ((I / Smem::kItemSlots) - 1) & 1, abort_flag, kSiteItemEmpty))
          break;
        if (more) *s_item = item;
        publish_item(more);
        if (!more) break;
      }
    }
  } else if (warp == kMmaWarpA || warp == kMmaWarpB || warp == kMmaWarpC) {
    // ------------------------------------------------------------------ MMA issuers
    const bool el = elect_one();
    constexpr uint32_t idesc_s = make_idesc(kTile, kTile, kBf16, false, false);  // keys x queries, both K-major
    constexpr uint32_t idesc_acc = make_idesc(kTile, D, kBf16, false, true);     // A K-major (or TMEM), B N-major
    constexpr uint32_t idesc_dq = make_idesc(kTile, D, kBf16, true, true);       // A M-major (dS^T tile), B N-major
    const SmemDesc ones_desc = make_sdesc_slab32(smem_u32(s_ones));
    auto stage_of = [](SmemDesc d, int stage, uint32_t stage_bytes) {
      d.lo += static_cast<uint32_t>(stage) * (stage_bytes >> 4);
      return d;
    };
    // dst = A B^T over D (both K-major) plus the bias-slab step: dst[m][n] += w * (slab[n] hi + mid + lo)
    auto issue_scores = [&](uint32_t dst, const SmemDesc& a_desc, const SmemDesc& b_desc, const SmemDesc& slab) {
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        umma_ss(dst, sdesc_at(a_desc, kk * 32), sdesc_at(b_desc, kk * 32), idesc_s, kk > 0);
      umma_ss(dst, sdesc_at(ones_desc, 0), sdesc_at(slab, 0), idesc_s, 1u);
    };
    // The products of eight MMAs are loops of four: less code (see mbar_wait_limit) at the same rate of issue. Backward call,
    // unrolled altogether -> by four: B64 H8 N1028 393 -> 387 us, B4 N4100 H8 fp16 254 -> 246, B4 H8 N1024 37.9 -> 37.4.
    // Within an item the lanes wait each for itself (nothing there needs the whole warp) and agree on the outcome before
    // the next one. A vote at every wait cost the backward call 3 % at B8 H16 N4096 (994 -> 1024 us) and 7 % at B64 H8
    // N1028 (453 -> 488 us): three issuers wait in turn on the way from one step to the next.
    bool ok = run;
    while (__all_sync(0xffffffffu, ok) && next_item()) {
      if (warp == kMmaWarpA) {
        const SmemDesc k_kmaj = stage_of(make_sdesc_parts(smem_u32(s_k), 16, 1024), I & 1, kTileBytes);
        const SmemDesc q_kmaj0 = make_sdesc_parts(smem_u32(s_q), 16, 1024);
        const SmemDesc lslab0 = make_sdesc_slab32(smem_u32(s_lslab));
        ok = mbar_wait(&k_full[I & 1], (I >> 1) & 1, abort_flag, kSiteKFull);
        for (int n = 0; n < cnt && ok; ++n) {
          const uint32_t g = T + n, st = g % kQStages;
          ok = mbar_wait(&q_full[st], (g / kQStages) & 1, abort_flag, kSiteQFull);
          // S^T(n) may overwrite S^T(n-1) once every compute warp has stored P^T(n-1)
          if (ok && g > 0) ok = mbar_wait(p_full, (g - 1) & 1, abort_flag, kSitePFull);
          if (!ok) break;
          tc_fence_after_sync();
          if (el) {
            issue_scores(tmem + kColS, k_kmaj, stage_of(q_kmaj0, st, kTileBytes), stage_of(lslab0, st, kSlabBytes));
            umma_commit(s_full);
          }
        }
      } else if (warp == kMmaWarpB) {
        const SmemDesc v_kmaj = make_sdesc_parts(smem_u32(s_v), 16, 1024);
        const SmemDesc do_kmaj0 = make_sdesc_parts(smem_u32(s_do), 16, 1024);
        const SmemDesc do_nmaj0 = make_sdesc_parts(smem_u32(s_do), kTile * 128, 1024);
        const SmemDesc dslab0 = make_sdesc_slab32(smem_u32(s_dslab));
        ok = mbar_wait(v_full, I & 1, abort_flag, kSiteVFull);
        for (int n = 0; n < cnt && ok; ++n) {
          const uint32_t g = T + n, st = g % kDoStages;
          ok = mbar_wait(&do_full[st], (g / kDoStages) & 1, abort_flag, kSiteDoFull);
          // dP^T(n) may overwrite dP^T(n-1) once every compute warp has stored dS^T(n-1)
          if (ok && g > 0) ok = mbar_wait(ds_full, (g - 1) & 1, abort_flag, kSiteDSFull);
          if (!ok) break;
          tc_fence_after_sync();
          if (el) {
            issue_scores(tmem + kColDP, v_kmaj, stage_of(do_kmaj0, st, kTileBytes), stage_of(dslab0, st, kSlabBytes));
            umma_commit(dp_full);
            if (n == cnt - 1) umma_commit(v_free);
          }
          // dV += P^T dO, from zero once the previous item's dV has left
          ok = mbar_wait(p_full, g & 1, abort_flag, kSitePFull);
          if (ok && n == 0 && I > 0) ok = mbar_wait(dv_free, (I - 1) & 1, abort_flag, kSiteDVFree);
          if (!ok) break;
          tc_fence_after_sync();
          const SmemDesc do_n = stage_of(do_nmaj0, st, kTileBytes);
          if (el) {
#pragma unroll 4
            for (int kk = 0; kk < kTile / 16; ++kk)
              umma_ts(tmem + kColDV, tmem + kColPT + kk * 8, sdesc_at(do_n, kk * 2048), idesc_acc,
                      (n > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&do_empty[st]);
            if (n == cnt - 1) umma_commit(dv_acc);
          }
        }
      } else {
        // dK += dS^T Q : A = dS^T tile (K-major: 64-query boxes of 128-byte rows), B = Q read N-major
        const SmemDesc q_nmaj0 = make_sdesc_parts(smem_u32(s_q), kTile * 128, 1024);
        const SmemDesc ds_kmaj = make_sdesc_parts(smem_u32(s_ds), 16, 1024);            // rows = keys, K = queries
        // dQ_partial = dS K : A = the dS^T tile read M-major (rows = keys = reduction index), B = K read N-major
        const SmemDesc k_nmaj = stage_of(make_sdesc_parts(smem_u32(s_k), kTile * 128, 1024), I & 1, kTileBytes);
        const SmemDesc ds_mmaj = make_sdesc_parts(smem_u32(s_ds), kTile * 128, 1024);   // rows = reduction (keys)
        ok = mbar_wait(&k_full[I & 1], (I >> 1) & 1, abort_flag, kSiteKFull);
        for (int n = 0; n < cnt && ok; ++n) {
          const uint32_t g = T + n, st = g % kQStages;
          ok = mbar_wait(ds_full, g & 1, abort_flag, kSiteDSFull);
          if (ok && n == 0 && I > 0) ok = mbar_wait(dk_free, (I - 1) & 1, abort_flag, kSiteDKFree);
          if (!ok) break;
          tc_fence_after_sync();
          const SmemDesc q_n = stage_of(q_nmaj0, st, kTileBytes);
          if (el) {
#pragma unroll 4
            for (int kk = 0; kk < kTile / 16; ++kk)
              umma_ss(tmem + kColDK, sdesc_at(ds_kmaj, (kk >> 2) * (kTile * 128) + (kk & 3) * 32), sdesc_at(q_n, kk * 2048),
                      idesc_acc, (n > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&q_empty[st]);
            if (n == cnt - 1) umma_commit(dk_acc);   // the item's dK is complete
          }
          if (g > 0) ok = mbar_wait(dq_drained, (g - 1) & 1, abort_flag, kSiteDQDrained);
          if (!ok) break;
          tc_fence_after_sync();
          if (el) {
#pragma unroll 4
            for (int kk = 0; kk < kTile / 16; ++kk)
              umma_ss(tmem + kColDQ, sdesc_at(ds_mmaj, kk * 2048), sdesc_at(k_nmaj, kk * 2048), idesc_dq, kk > 0);
            umma_commit(dq_full);                    // dQ_partial readable; the dS^T tile's readers are done
          }
        }
    }
    T += cnt;
    ++I;
    }
  } else if (warp >= kDrainWarp0) {
    // ------------------------------------------------------------------ drain: dQ_partial of every step, dV and dK
    // Every warp owns 32 rows (query rows of dQ_partial, key rows of dV and dK) and two 4 KB boxes, used in turn without
    // any synchronisation between the warps: a [32 rows][32 floats] box per half of dQ_partial's head dim, reduced into
    // the accumulator by the TMA engine, and a [32 rows][64 x 16-bit] box each for dV and dK. (An SM pushes about 25
    // bytes per clock of reduce-adds into L2, measured: the 32 KB of a step take half as long as the step and must
    // overlap it. Reduce-adds straight from these warps' registers, 512 consecutive bytes per instruction into an
    // accumulator laid out for it, saved the staging and cost 9 % on the kernel.)
    setmaxnreg_dec<kDrainRegs>();
    const int wq = warp & 3;
    const uint32_t lane_sel = static_cast<uint32_t>(wq * 32) << 16;
    uint8_t* my_boxes = s_out + wq * (2 * kDqBoxBytes);
    uint32_t uses = 0;
    auto open_box = [&]() -> uint8_t* {
      if (lane == 0) tma_store_wait_read1();       // the box written two uses ago has been read by the bulk engine
      __syncwarp();
      return my_boxes + (uses++ & 1) * kDqBoxBytes;
    };
    auto drain_dq = [&](int n) -> bool {
      if (!mbar_wait_warp(dq_full, (T + n) & 1, abort_flag, kSiteDQFull)) return false;
      tc_fence_after_sync();
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint8_t* box = open_box();
        uint32_t v[32];
        tmem_ld_x32(tmem + kColDQ + lane_sel + hh * 32, v);
        tmem_ld_wait();
        if (hh == 1) {
          tc_fence_before_sync();
          mbar_arrive_warp(dq_drained);   // the next dQ_partial MMA may overwrite TMEM
        }
        uint8_t* row = box + lane * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(row + ((c ^ (lane & 7)) << 4)) =
              make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_reduce_add_4d(&tm_dq_acc, box, hh * 32, (first + n) * kTile + wq * 32, h, b);
          tma_store_commit();
        }
      }
      return true;
    };
    bool ok = run;
    while (ok && next_item()) {
      const int row0 = k_row0 + wq * 32;             // this warp's key rows
      for (int n = 0; n < cnt - 1 && ok; ++n) ok = drain_dq(n);
      // dV and dK are complete before the last dQ_partial, and the next item's products wait for their columns
      if (ok) ok = mbar_wait_warp(dv_acc, I & 1, abort_flag, kSiteDVAcc);
      if (!ok) break;
      tc_fence_after_sync();
      {
        uint8_t* box = open_box();
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t acc[32];
          tmem_ld_x32(tmem + kColDV + lane_sel + hh * 32, acc);
          tmem_ld_wait();
          if (hh == 1) {
            tc_fence_before_sync();
            mbar_arrive_warp(dv_free);
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o[i] = pack2<kBf16>(__uint_as_float(acc[q4 * 8 + 2 * i]), __uint_as_float(acc[q4 * 8 + 2 * i + 1]));
            *reinterpret_cast<uint4*>(box + sw128_offset(lane, hh * 4 + q4)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (row0 < p.N) tma_store_4d(&tm_dv, box, 0, row0, h, b);
          tma_store_commit();
        }
    }
    ok = mbar_wait_warp(dk_acc, I & 1, abort_flag, kSiteDKAcc) &&
         mbar_wait_warp(&k_full[I & 1], (I >> 1) & 1, abort_flag, kSiteKFull) &&
         mbar_wait_warp(&rs_full[I & 1], (I >> 1) & 1, abort_flag, kSiteRowsum);
    if (!ok) break;
    tc_fence_after_sync();
    {
      // dK = 2 gamma (acc - rowsum(dS^T) k): every compute group holds a quarter of the row sum
      uint8_t* box = open_box();
      const int r = wq * 32 + lane;
      const float* rs = s_rowsum + (I & 1) * 4 * kTile + r;
      const float w = (rs[0] + rs[kTile]) + (rs[2 * kTile] + rs[3 * kTile]);
      const uint8_t* k_tile = s_k + (I & 1) * kTileBytes;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t acc[32];
        tmem_ld_x32(tmem + kColDK + lane_sel + hh * 32, acc);
        tmem_ld_wait();
        if (hh == 1) {
          tc_fence_before_sync();
          mbar_arrive_warp(dk_free);
        }
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const uint4 k_raw = *reinterpret_cast<const uint4*>(k_tile + sw128_offset(r, hh * 4 + q4));
          const uint32_t kw[4] = {k_raw.x, k_raw.y, k_raw.z, k_raw.w};
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 kv = unpack2<kBf16>(kw[i]);
            float x0, x1;
            ffma2v(x0, x1, kv.x, kv.y, -w, -w, __uint_as_float(acc[q4 * 8 + 2 * i]), __uint_as_float(acc[q4 * 8 + 2 * i + 1]));
            fmul2(x0, x1, x0, x1, p.grad_scale, p.grad_scale);
            o[i] = pack2<kBf16>(x0, x1);
          }
          *reinterpret_cast<uint4*>(box + sw128_offset(lane, hh * 4 + q4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row0 < p.N) tma_store_4d(&tm_dk, box, 0, row0, h, b);
        tma_store_commit();
      }
    }
    ok = drain_dq(cnt - 1);
    if (!ok) break;
    mbar_arrive_warp(&k_free[I & 1]);        // the last dQ_partial was K's last reader
    T += cnt;
    ++I;
    }
    if (lane == 0) tma_store_wait_all();
  } else {
    // ------------------------------------------------------------------ compute groups (thread = key row)
    setmaxnreg_inc<kComputeRegs>();
    const int g = (warp - kComputeWarp0) >> 2;             // 32-column slice of the query tile
    const int r = tid & (kTile - 1);
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    bool ok = run;
    while (ok && next_item()) {
      ok = mbar_wait_warp(&k_full[I & 1], (I >> 1) & 1, abort_flag, kSiteKFull);
      if (!ok) break;
      const float neg_ksq = -s_ksq[(I & 1) * kTile + r];
      float ds_rowsum = 0.f;
      for (int n = 0; n < cnt; ++n) {
        ok = mbar_wait_warp(s_full, (T + n) & 1, abort_flag, kSiteSFull);
        if (!ok) break;
        tc_fence_after_sync();
        float pr[32];
        bool dp_ready;
        {
          uint32_t raw[32];
          tmem_ld_x32(tmem + kColS + lane_sel + g * 32, raw);
          dp_ready = mbar_test(dp_full, (T + n) & 1);
          tmem_ld_wait();
          // acc = k.q - L / scale2 ; P = exp2(acc * scale2 - ksq)
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float a0, a1;
            ffma2_bcast(a0, a1, __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]), p.scale2, neg_ksq);
            pr[i] = ex2_approx(a0);
            pr[i + 1] = ex2_approx(a1);
          }
        }
        if (p.causal && n == 0) {
          // diagonal tile: query column (32g + c) sees key row r iff column >= row
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (g * 32 + c < r) pr[c] = 0.f;
        }
        // dP^T(n) has landed, and with it dV(n-1): the P^T columns are free
        if (!__all_sync(0xffffffffu, dp_ready)) {
          ok = mbar_wait_warp(dp_full, (T + n) & 1, abort_flag, kSiteDPFull);
          if (!ok) break;
        }
        tc_fence_after_sync();
        {
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) packed[i] = pack2<kBf16>(pr[2 * i], pr[2 * i + 1]);
          tmem_st_x16(tmem + kColPT + lane_sel + g * 16, packed);
        }
        uint32_t ds_packed[16];
        bool ds_free;
        {
          uint32_t raw[32];
          tmem_ld_x32(tmem + kColDP + lane_sel + g * 32, raw);     // travels while the P^T store completes
          tmem_st_wait();
          tc_fence_before_sync();
          mbar_arrive_warp(p_full);
          // the dS^T tile is free once dK and dQ_partial of the previous step have completed
          ds_free = T + n == 0 || mbar_test(dq_full, (T + n - 1) & 1);
          tmem_ld_wait();
          // acc = v.dO - delta ; dS = P * acc
          float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float d0, d1;
            fmul2(d0, d1, pr[2 * i], pr[2 * i + 1], __uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1]));
            fadd2(rs0, rs1, rs0, rs1, d0, d1);
            ds_packed[i] = pack2<kBf16>(d0, d1);
          }
          ds_rowsum += rs0 + rs1;
        }
        if (!__all_sync(0xffffffffu, ds_free)) {
          ok = mbar_wait_warp(dq_full, (T + n - 1) & 1, abort_flag, kSiteDsFree);
          if (!ok) break;
        }
        // row r of the [key][query] tile, box g/2, 16-byte chunks 4(g%2) .. +3
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(s_ds + (g >> 1) * (kTile * 128) + sw128_offset(r, (g & 1) * 4 + ch)) =
              make_uint4(ds_packed[ch * 4 + 0], ds_packed[ch * 4 + 1], ds_packed[ch * 4 + 2], ds_packed[ch * 4 + 3]);
        tc_fence_before_sync();
        fence_proxy_async_smem();
        mbar_arrive_warp(ds_full);
    }

    if (ok) {
      // (the buffer's previous user, two items back, has been read: dK of the item in between has been started since)
      s_rowsum[((I & 1) * 4 + g) * kTile + r] = ds_rowsum;
      mbar_arrive_warp(&rs_full[I & 1]);
    }
    T += cnt;
    ++I;
    }
  }

  // ------------------------------------------------------------------ teardown
  grid_dependents_launch();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0) record_timeout(abort_flag, p.status, *s_item);
  if (warp == kMmaWarpA) tmem_dealloc(*tmem_base_s, 512);
  if (queue && tid == 0) {
    // the last CTA to leave puts the work counters back to zero for the next launch on this workspace
    __threadfence();
    if (atomicAdd(&p.work[1], 1u) == gridDim.x - 1) {
      p.work[0] = 0u;
      p.work[1] = 0u;
    }
  }
}

// dq[b,h,n,:] = scale * acc[b,h,n,:]  (acc fp32 contiguous, dq 16-bit with strides)
template <bool kBf16>
__global__ void __launch_bounds__(256) dq_convert_kernel(const float* acc, void* dq, int H, int N, int64_t sb,
                                                         int64_t sh, int64_t sn, float scale, int64_t total_chunks,
                                                         const void* q, int64_t qsb, int64_t qsh, int64_t qsn,
                                                         const float* delta, int n_pad,
                                                         const DeviceStatus* status, unsigned int* status_slot,
                                                         int head_dim) {
  grid_dependency_wait();
  if (status_slot != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) post_status_word(status, status_slot);
  // one thread per 8 consecutive elements of a row (D = 64: 8 chunks per row)
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total_chunks) return;
  const int64_t row = i >> 3;
  const int ch = static_cast<int>(i & 7);
  if (ch * 8 >= head_dim) return;
  const int64_t n = row % N;
  const int64_t bh = row / N;
  const int64_t b = bh / H, h = bh % H;
  const float4* src = reinterpret_cast<const float4*>(acc + row * D + ch * 8);
  float4 a = src[0], c = src[1];
  if (q != nullptr) {
    // non-softmax variant: subtract delta[row] * q[row, :]
    const float w = delta[bh * n_pad + n];
    const uint4 qv = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(q) + b * qsb + h * qsh +
                                                     n * qsn + ch * 8);
    const float2 q0 = unpack2<kBf16>(qv.x), q1 = unpack2<kBf16>(qv.y), q2 = unpack2<kBf16>(qv.z),
                 q3 = unpack2<kBf16>(qv.w);
    a.x = fmaf(-w, q0.x, a.x); a.y = fmaf(-w, q0.y, a.y); a.z = fmaf(-w, q1.x, a.z); a.w = fmaf(-w, q1.y, a.w);
    c.x = fmaf(-w, q2.x, c.x); c.y = fmaf(-w, q2.y, c.y); c.z = fmaf(-w, q3.x, c.z); c.w = fmaf(-w, q3.y, c.w);
  }
  uint4 o;
  o.x = pack2<kBf16>(a.x * scale, a.y * scale);
  o.y = pack2<kBf16>(a.z * scale, a.w * scale);
  o.z = pack2<kBf16>(c.x * scale, c.y * scale);
  o.w = pack2<kBf16>(c.z * scale, c.w * scale);
  uint16_t* dst = reinterpret_cast<uint16_t*>(dq) + b * sb + h * sh + n * sn + ch * 8;
  *reinterpret_cast<uint4*>(dst) = o;
}

template <bool kBf16>
static cudaError_t launch_t(const BwdFusedArgs& a, cudaStream_t stream) {
  auto kernel = rbf_bwd_fused_kernel<kBf16>;
  constexpr int smem = Smem::kDynamic;
  static PerDeviceFlags configured{};
  {
    const cudaError_t ce = ensure_dynamic_smem(kernel, smem, configured);
    if (ce != cudaSuccess) return ce;
  }
  // the pre-pass has cleared the dQ accumulator
  cudaError_t e = cudaSuccess;
  Params p{};
  p.ksq = a.ksq; p.status = a.status;
  p.H = a.H; p.N = a.N; p.n_pad = a.n_pad; p.causal = a.causal;
  p.scale2 = a.scale2; p.grad_scale = a.grad_scale; p.slab_w = a.slab_w;
  p.work = a.work;
  const int n_tiles = (a.N + kTile - 1) / kTile;
  p.total_items = n_tiles * a.B * a.H;
  p.group = item_group(n_tiles, a.B * a.H, a.causal, a.sm_count);
  p.plain_heads = a.B * a.H - p.group;
  dim3 grid(p.total_items < a.sm_count ? p.total_items : a.sm_count);
  e = launch_dependent(kernel, grid, kThreads, smem, stream, a.tm_k, a.tm_v, a.tm_q, a.tm_do, a.tm_dk, a.tm_dv, a.tm_lslab,
                       a.tm_dslab, a.tm_dq_acc, p);
  if (e != cudaSuccess) return e;
  const int64_t chunks = static_cast<int64_t>(a.B) * a.H * a.N * 8;
  return launch_dependent(
      dq_convert_kernel<kBf16>, static_cast<unsigned>((chunks + 255) / 256), 256, 0, stream, a.dq_acc, a.dq, a.H, a.N, a.dq_strides[0], a.dq_strides[1], a.dq_strides[2], a.grad_scale, chunks, a.q_rows,
      a.q_strides[0], a.q_strides[1], a.q_strides[2], a.delta, a.n_pad, a.status, a.status_slot, a.head_dim);
}

}  // namespace bwdf


cudaError_t launch_bwd_fused(const BwdFusedArgs& a, bool bf16, cudaStream_t stream) {
  return bf16 ? bwdf::launch_t<true>(a, stream) : bwdf::launch_t<false>(a, stream);
}

}  // namespace rbf
