// bf16 GEMM on CTA pairs (tcgen05 cta_group::2) for sm_100a: one 256 x 256 output tile per pair of SMs, or one of 256 x 128 where
// that is the shorter way (half_tiles_pay), with half of B and of the accumulator.
//
// Two CTAs of a cluster work on one tile.  Each CTA stages ITS half of the A tile (128 rows) and ITS half of the B
// tile (128 rows of B, i.e. 128 output columns) with ordinary per-CTA TMA loads, and holds the accumulator rows
// of its A half (128 lanes x 256 fp32 columns) in its own tensor memory.  One thread of the even CTA (the leader)
// issues tcgen05.mma.cta_group::2: the tensor cores of both SMs read both halves of B, so every byte of B is
// fetched from L2 and written to shared memory once per PAIR instead of once per SM, and a stage of the ring is
// 32 KiB per CTA instead of 48 KiB (six stages instead of four).
//
//   warp 0      : TMA producer of this CTA's halves; byte counts are reported to the leader's "full" barrier
//   warp 1      : leader only: MMA issuer; completion is committed to BOTH CTAs' barriers (two commits, no multicast)
//   warps 2..5  : epilogue of this CTA's 128 rows, 32 each (tcgen05.ld -> bias / residual -> swizzled staging -> TMA store),
//                 then a (remote) arrive on the leader's "accumulator free" barrier
// The issuing threads are elected with elect.sync: of a thread picked by its lane number the compiler does not know that it
// is alone, and moves every descriptor to uniform registers by way of a loop, which the main loop then waits for (16321 x
// 16384 x 2048: 760 us, elected 679; the twelve products of a 2048-wide layer over 16321 tokens: 4.40 ms, now 4.05).
// Two accumulators (all 512 TMEM columns of each CTA) alternate, so the epilogue of one tile overlaps the main
// loop of the next.  Every copy in this file is an ordinary per-CTA TMA copy into that CTA's own shared memory.  Every wait is
// bounded and reports through the status word; a pair whose partner gave up runs into its own bounded waits and leaves the same way.
//
// Operand layouts, edge handling and the epilogue are those of the single-CTA kernel (gemm_tcgen05.cu).
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdlib.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "api.h"
#include "launch.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace odc {
namespace gemm_pair {

using namespace sm100;

constexpr int BMH = 128, BNH = 128, BN = 256, BK = 64;   // per-CTA halves; the pair's tile is 256 x 256
constexpr int kStages = 6;
constexpr int kATile = BMH * BK * 2;                     // 16 KiB
constexpr int kBTile = BNH * BK * 2;                     // 16 KiB
constexpr int kStageBytes = kATile + kBTile;             // 32 KiB per CTA
constexpr int kStagingBytes = 128 * 128;
constexpr int kOutRows = 32;                             // rows of an output box: those of one epilogue warp
constexpr int kSmemBytes = kStages * kStageBytes + 2 * kStagingBytes + 1024 + 768;
constexpr uint32_t kTmemCols = 512;
constexpr uint64_t kWaitBudgetNs = 4000000000ull;
constexpr int kThreads = 192;
constexpr int kMaxGroup = kMaxGroupProducts;

struct Params {
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  int M, N, K;
  int c_is_f32, accumulate;
  int a_mn, b_mn;
  int tiles_m, tiles_n;   // in units of the pair's 256 x 256 tile (256 x 128 in half-width ones)
  int bn;                 // modes with tiles of either width: columns of a tile
  // kModePlain, kModeScatter: the first `whole` tiles are work items of their own; the k-blocks of every other are divided
  // over `splits` items, kb_split each.  In kModePlain item whole + i writes its fp32 partial tile at row 256 * i of a
  // 256-column scratch (owners.m[0])
  int whole, splits, kb_split;
  int* status;
  // kModeScatter: the epilogue adds every 128-row output box into the fp32 accumulator of the rank that owns those rows
  const long long* ctr_ptrs;   // [nranks] arrival counters
  int rows_per_rank;           // output rows owned by one rank (a multiple of 128)
  int nranks;
  float scale;
  unsigned int* done_slot;     // self-resetting CTA completion counter
  // kModeGather: operand B (a row-sharded weight) is assembled from the owners' shards while the GEMM runs
  const long long* shard_ptrs; // [nranks] base address of each owner's [rows_per_rank, w_cols] bf16 shard
  unsigned char* b_local;      // local [w_rows, w_cols] bf16 buffer the shards are gathered into (tensor map B covers it)
  unsigned int* panel_flags;   // [ceil(w_rows / 256)] chunks landed per 256-row group (zeroed before the launch)
  // kModeSwiglu (N = F): tensor maps c: activation [M, F], owners.m[0] / [1]: gate / up half of the projection [M, 2F]
  int store_gate_up;
  // kModeLogits
  const long long* labels;     // [M]
  float2* row_stats;           // [tiles_n, M]: largest scaled logit of the tile's columns and the sum of 2^(logit - it)
  float* label_logits;         // [M]
  float inv_temp;
  int store_logits;
  // kModeRope: the columns below rot_cols are heads of head_dim, rotated by the row's position
  const long long* pos;        // [M]
  int rot_cols, head_dim;
  float log2_theta;
  int w_rows, w_cols;          // gathered matrix: [N, K] when B is K-major (y = x W^T), [K, N] when MN-major (dx = dy W)
  // Rotation of the work order by this rank's position in the group.  Without it every rank would pull the first
  // owner's rows first (and push into the first owner's accumulator first): one GPU's links saturated, seven idle.
  // Each rank starts at the rows it owns itself and walks the owners from there, like the stand-alone kernels do.
  int rot_m, rot_n;            // tile rows / tile columns by which the tile order is rotated
  int rot_kb;                  // k-blocks by which the k loop is rotated (gathered reduction dimension)
  long long fetch_rot;         // 64 KiB chunks by which the fetch order is rotated
};

// kModeSwiglu: B holds the gate rows and, F rows further on, the up rows.  The even CTA stages 128 gate rows and the odd one
// the matching 128 up rows, so a tile's accumulator holds both halves of 128 activations and the epilogue forms them: the
// activation is not a pass of its own (16384 x 8192: 0.12 ms of reading and writing), and without gradients the
// projection itself is never written.
// kModeLogits: the epilogue leaves the softmax statistics of every row of a tile and the label's logit, so the log-sum-exp
// needs no pass over the logits, and where no gradient follows they are not written at all.  From the logits as rounded to
// bf16, as the pass that forms the gradient reads them.  The arithmetic (one exponential per logit) runs under the next tile's
// products, where these are long enough (logits_stats_pay).  Log-probabilities of 6000 tokens, 151936 words, 1536 wide, forward and backward: 9.62 ms, now 8.99; forward only,
// 16321 tokens, 128256 words: four passes of 0.24 ms and as many writes of the logits less (36.6 -> 35.3 ms with the decoder).
constexpr int kModePlain = 0, kModeScatter = 1, kModeGather = 2, kModeSwiglu = 3, kModeLogits = 4, kModeSwigluBwd = 5, kModeGroup = 6, kModeRope = 7;
// kModeSwigluBwd (N = F): the product is the gradient of the activations; the epilogue turns it, rounded to bf16, with the
// projection [M, 2F] (tensor map c) into the projection's gradient (owners.m[0] / [1]: its halves).  A warp of its own brings
// boxes of gate and up into two buffers, for which the ring gives up a stage.  Forward and backward of a layer, both forms in
// turn: 16321 tokens, 2048 and 8192 wide: 6.92 ms with the pass, 6.76 without; 30000 tokens, 4096 and 14336 wide, all under the
// power cap: 34.4 and 34.6, the same within the spread of either.
template <int kMode> struct Ring {
  static constexpr int kDepth = kMode == kModeSwigluBwd ? 5 : 6;
  static constexpr int kGateUpBytes = kMode == kModeSwigluBwd ? 2 * kStagingBytes : 0;
};
static_assert(kStageBytes == 2 * kStagingBytes, "the boxes of gate and up take the place of one stage");
constexpr int kFetchWarps = 4;
constexpr int kFetchWarpBytes = 16384;                  // moved by one fetch warp between two flag updates
constexpr int kFetchChunkBytes = kFetchWarps * kFetchWarpBytes;
template <int kMode> struct Roles {
  static constexpr int kThreadsTotal = kThreads + (kMode == kModeGather ? 32 * kFetchWarps : kMode == kModeSwigluBwd ? 32 : 0);
};
constexpr int kMaxOwners = 8;
struct OwnerMaps {   // one fp32 tensor map per owner's accumulator region (kModeScatter)
  CUtensorMap m[kMaxOwners];
};

// kModeGroup: up to three products that do not depend on one another (the input and weight gradients of a layer) in one launch.
// Apart, each fills the machine by itself or not at all: 1000 tokens, 1536 and 8960 wide, are 24, 420 and 210 tiles of 280, 16
// and 16 k-blocks on 74 pairs.  The items of the longest product come first and a pair takes the next one from a counter, so the
// short ones fill what the long ones leave.  One by one / together, us on the GPU: input and weight gradient of 1000 x 1536 x 2048
// 19.0 / 17.5, of 1000 x 1536 x 1536 14.9 / 14.9, of 2000 x 512 x 512 (fp32 sum) 14.5 / 10.1; the three of an MLP over 2000 tokens, 512
// and 1536 wide, 32.0 / 18.3, 300 tokens, 2048 and 8192 wide, 70 / 67 (fp32 sums 123 / 106), 1000 tokens, 1536 and 8960 wide,
// 109 / 106 (134 / 130).  Called from a program, smaller ones gain the launches: MLP of 512 and 1536, 300 tokens, forward and backward,
// 93 / 85.  One product by itself costs 0.7 us more than in kModePlain, and some 0.2 us an item where items are short.
struct GroupProblem {
  int M, N, K, tiles_m, tiles_n;
  int a_mn, b_mn, bn;
  int out;                  // 0: bf16, 1: fp32, 2: added to fp32
  float scale;              // of the result, times *scale_ptr unless that is null
  const float* scale_ptr;
  const float* addend;      // bf16 results: fp32 [M, N] that joins the sum before it is rounded, or null
  int first;                // its first item
  // the first `whole` tiles are items, each of the `divided` others is `splits` of kb_split k-blocks each
  int whole, divided, splits, kb_split;
  int first_split_tile, first_part;   // bf16 with divided tiles: of the first of them, among the divided tiles and parts of the launch
};
struct Group {
  CUtensorMap a[kMaxGroup], b[kMaxGroup], c[kMaxGroup];
  GroupProblem prob[kMaxGroup];
  int count, items;
  // bf16 tiles in parts: each part is left in fp32 scratch, and the CTA that finds its part to be the last of the tile adds them
  // up in order.  arrived: parts that are there, per divided tile and CTA of a pair; zero before and after the launch.
  float4* parts;
  unsigned int* arrived;
  unsigned int* next;       // items handed out so far beyond the first of every pair; zero before and after the launch
  int arrivals;             // contributions to report to ctr_ptrs[0] when all is added
};
__device__ __forceinline__ int owners_rows(const OwnerMaps&, int) { return 0; }
__device__ __forceinline__ int owners_rows(const Group& g, int i) { return g.prob[i].M; }
template <int kMode> struct Extra { using type = OwnerMaps; };
template <> struct Extra<kModeGroup> { using type = Group; };
constexpr uint32_t kItemSlots = 16;   // see the item loop

// Tile order: groups of kGroupM tile rows are walked column by column (rows fastest inside a group), so the pairs
// that run at the same time share a few A row panels and a few B column panels and both stay in L2 however large
// the whole operands are.
constexpr int kGroupM = 16;
template <typename P>
__device__ __forceinline__ void tile_coords(int tile, const P& p, int rot_m, int rot_n, int* tm, int* tn) {
  const int per_group = kGroupM * p.tiles_n;
  const int group = tile / per_group;
  const int first_m = group * kGroupM;
  const int gsize = min(p.tiles_m - first_m, kGroupM);
  const int in_group = tile - group * per_group;
  int m = first_m + in_group % gsize + rot_m;
  int n = in_group / gsize + rot_n;
  *tm = m >= p.tiles_m ? m - p.tiles_m : m;
  *tn = n >= p.tiles_n ? n - p.tiles_n : n;
}
__device__ __forceinline__ void tile_coords(int tile, const Params& p, int* tm, int* tn) {
  tile_coords(tile, p, p.rot_m, p.rot_n, tm, tn);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// One thread's walk over the k-blocks of an item.  What a k-block takes is instructions one behind the other: with the stage's
// number, address and parity worked out from a running count, the operands' layouts asked for and the leader's barrier looked up
// at each, loading one took 465 clocks, nearly as much as multiplying a whole tile's (512) and more than a half tile's (256).
// Stepped, with the layouts as types and the first tile worked out before the pair meets: 1900 x 512 x 512 6.3 us, now 5.3, 1000 x
// 1536 x 1536 10.2 and 8.1, with K = 8960 and an fp32 result 38.5 and 28.0; whole tiles gain half a microsecond a launch.
template <int kStages, bool kAMn, bool kBMn>
__device__ __forceinline__ bool load_blocks(const CUtensorMap* map_a, const CUtensorMap* map_b, int kb0, int kb1, int m0, int n0, bool whole_b,
                                            uint32_t it, uint32_t base, uint32_t empty0, uint32_t full0, uint32_t leader_full0, bool leader,
                                            uint32_t bytes, const WaitCtx& wc) {
  uint32_t s = it % kStages, parity = ((it / kStages) & 1) ^ 1;
  for (int k0 = kb0 * BK; k0 < kb1 * BK; k0 += BK) {
    if (!mbar_wait(empty0 + 8 * s, parity, wc, 11)) return false;
    const uint32_t sa = base + s * kStageBytes, sb = sa + kATile, bar = leader_full0 + 8 * s;
    if (leader) mbar_arrive_expect_tx(full0 + 8 * s, bytes);   // of both CTAs
    if constexpr (!kAMn) {
      tma_load_2d_pair(sa, map_a, bar, k0, m0);                 // box {64 k, 128 rows}
    } else {
      tma_load_2d_pair(sa, map_a, bar, m0, k0);
      tma_load_2d_pair(sa + 8192, map_a, bar, m0 + 64, k0);
    }
    if constexpr (!kBMn) {
      tma_load_2d_pair(sb, map_b, bar, k0, n0);                 // box {64 k, 128 (64) rows}
    } else {
      tma_load_2d_pair(sb, map_b, bar, n0, k0);
      if (whole_b) tma_load_2d_pair(sb + 8192, map_b, bar, n0 + 64, k0);
    }
    if (++s == kStages) { s = 0; parity ^= 1; }
  }
  return true;
}
template <int kStages, typename... Rest>
__device__ __forceinline__ bool load_blocks(int a_mn, int b_mn, Rest... rest) {
  if (a_mn) return load_blocks<kStages, true, true>(rest...);   // "tn"
  return b_mn ? load_blocks<kStages, false, true>(rest...) : load_blocks<kStages, false, false>(rest...);
}
// The products of an item's k-blocks into the accumulator at d_tmem; the stages are reusable in BOTH CTAs once they have been read.
template <int kStages>
__device__ __forceinline__ bool multiply_blocks(int blocks, uint32_t it, uint32_t d_tmem, uint32_t idesc, int a_mn, int b_mn, uint32_t base,
                                                uint32_t full0, uint32_t empty0, const WaitCtx& wc) {
  const uint32_t leader_empty0 = mapa_shared(empty0, 0), partner_empty0 = mapa_shared(empty0, 1);
  const uint64_t da0 = make_smem_desc(base, a_mn ? 8192u : 16u, 1024), db0 = make_smem_desc(base + kATile, b_mn ? 8192u : 16u, 1024);
  const uint64_t a_kstep = a_mn ? 128 : 2, b_kstep = b_mn ? 128 : 2;  // 16-byte units per K = 16
  uint32_t s = it % kStages, parity = (it / kStages) & 1;
  for (int n = 0; n < blocks; ++n) {
    if (!mbar_wait(full0 + 8 * s, parity, wc, 13)) return false;
    tc_fence_after();
    const uint64_t da = da0 + s * (kStageBytes / 16), db = db0 + s * (kStageBytes / 16);
#pragma unroll
    for (int j = 0; j < BK / 16; ++j) umma_f16_pair(d_tmem, da + j * a_kstep, db + j * b_kstep, idesc, (n > 0 || j > 0) ? 1u : 0u);
    umma_commit_pair(leader_empty0 + 8 * s);
    umma_commit_pair(partner_empty0 + 8 * s);
    if (++s == kStages) { s = 0; parity ^= 1; }
  }
  return true;
}

template <int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Roles<kMode>::kThreadsTotal, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ typename Extra<kMode>::type owners,
                      const Params p) {
  constexpr int kStages = Ring<kMode>::kDepth;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  uint8_t* staging = smem + kStages * kStageBytes + Ring<kMode>::kGateUpBytes;
  const uint32_t staging_u32 = base + kStages * kStageBytes + Ring<kMode>::kGateUpBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + 2 * kStagingBytes);
  const uint32_t full0 = smem_u32(bars);                    // [kStages]  used in the leader: both CTAs' bytes landed
  const uint32_t empty0 = full0 + 8 * kStages;              // [kStages]  per CTA: the MMAs have read this stage
  const uint32_t tfull0 = empty0 + 8 * kStages;             // [2]        per CTA: accumulator complete
  const uint32_t tempty0 = tfull0 + 16;                     // [2]        used in the leader: both epilogues drained it
  const uint32_t gfull = tempty0 + 16, gempty = gfull + 8;  // boxes of gate and up
  const uint32_t islot0 = gempty + 8;                       // [kItemSlots] per CTA: an item is written down
  const uint32_t pready = islot0 + 8 * kItemSlots, pcounted = pready + 8;   // a part is in memory / has been counted
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 6 + kItemSlots + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* part_last = abort_flag + 1;
  volatile int* item_slots = part_last + 1;                 // [kItemSlots]
  float* rope_freq = reinterpret_cast<float*>(const_cast<int*>(item_slots) + kItemSlots);   // [64]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();                   // 0: leader
  const WaitCtx wc{abort_flag, p.status, kWaitBudgetNs};

  constexpr bool kDivides = kMode == kModePlain || kMode == kModeScatter;
  const int bn = kMode == kModePlain || kMode == kModeRope || kMode == kModeSwiglu ? p.bn : BN;   // of a group: its products'
  const int num_tiles = p.tiles_m * p.tiles_n;
  int num_items = kDivides ? p.whole + (num_tiles - p.whole) * p.splits : num_tiles;   // the parts of a tile are adjacent
  if constexpr (kMode == kModeGroup) num_items = owners.items;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  // kModeGroup, leader's producer: every pair asks until it is told that there is nothing left, `items` questions in all, and the
  // last one clears the counter.  `taken` is apart from the question: looking at the answer waits for it.
  [[maybe_unused]] auto take = [&]() -> int {
    if constexpr (kMode == kModeGroup)
      if (num_items > num_pairs && lane == 0) return num_pairs + static_cast<int>(atomicAdd(owners.next, 1u));
    return num_items;
  };
  [[maybe_unused]] auto taken = [&](int i) {
    if constexpr (kMode == kModeGroup)
      if (num_items > num_pairs && lane == 0 && i == num_pairs + num_items - 1) *owners.next = 0;
  };

  if (threadIdx.x == 0) {
    if constexpr (kMode != kModeGroup) {
      prefetch_tmap(&tmap_a);   // the descriptors are on their way while the barriers are set up
      prefetch_tmap(&tmap_b);
      prefetch_tmap(&tmap_c);
    }
    mbar_init(gfull, 1);
    mbar_init(gempty, 4);
    if constexpr (kMode == kModeGroup) {
      for (uint32_t s = 0; s < kItemSlots; ++s) mbar_init(islot0 + 8 * s, 1);
      mbar_init(pready, 4);
      mbar_init(pcounted, 1);
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 8);   // four epilogue warps in each CTA of the pair
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if constexpr (kMode == kModeGroup) {
    if (warp == 2 && lane < owners.count) {
      prefetch_tmap(&owners.a[lane]);
      prefetch_tmap(&owners.b[lane]);
      prefetch_tmap(&owners.c[lane]);
    }
  }
  if constexpr (kMode == kModeRope) {
    if (threadIdx.x >= 128 && threadIdx.x < 128 + p.head_dim / 2)
      rope_freq[threadIdx.x - 128] = exp2f(-p.log2_theta * (2.0f * (threadIdx.x - 128)) / p.head_dim);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  const int all_k_blocks = (p.K + BK - 1) / BK;
  auto is_part = [&](int item) { return kDivides && item >= p.whole; };
  auto tile_of = [&](int item) { return is_part(item) ? p.whole + (item - p.whole) / p.splits : item; };
  auto k_range = [&](int item, int* kb0, int* kb1) {
    *kb0 = 0;
    *kb1 = all_k_blocks;
    if (is_part(item)) {
      *kb0 = (item - p.whole) % p.splits * p.kb_split;
      *kb1 = min(all_k_blocks, *kb0 + p.kb_split);
    }
  };
  // where an item lies; group modes only
  struct Place { int pi, tm, tn, kb0, kb1, part, divided; };   // divided: which of its product's divided tiles, or -1
  [[maybe_unused]] auto place_of = [&](int item) -> Place {
    Place w{};
    if constexpr (kMode == kModeGroup) {
      while (w.pi + 1 < owners.count && item >= owners.prob[w.pi + 1].first) ++w.pi;
      const GroupProblem& q = owners.prob[w.pi];
      const int local = item - q.first, beyond = local - q.whole;
      // the first parts of all tiles, then the second ones: what runs at the same time reads the same k-blocks of A and B
      w.part = beyond < 0 ? 0 : beyond / q.divided;
      w.divided = beyond < 0 ? -1 : beyond - w.part * q.divided;
      tile_coords(beyond < 0 ? local : q.whole + w.divided, q, 0, 0, &w.tm, &w.tn);
      w.kb0 = w.part * q.kb_split;
      w.kb1 = (q.K + BK - 1) / BK;
      if (beyond >= 0) w.kb1 = min(w.kb1, w.kb0 + q.kb_split);
    }
    return w;
  };

  // the producer's first tile, worked out before the CTAs of the pair meet
  [[maybe_unused]] int first_tm = 0, first_tn = 0;
  [[maybe_unused]] Place first_place{};
  if (warp == 0) {
    if constexpr (kMode == kModeGroup) first_place = place_of(pair);
    else tile_coords(tile_of(pair), p, &first_tm, &first_tn);
  }
  [[maybe_unused]] int ahead = 0;   // kModeGroup: what the leader's producer (its lane 0) has asked for beyond the next item
  if constexpr (kMode == kModeGroup) {
    if (warp == 0 && cta == 0) ahead = take();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_barriers();   // the partner's barriers exist before anything is reported to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Work items.  kModeGroup: the leader's producer takes them from a counter and writes the next one down for the other roles of
  // both CTAs before it loads the current one.  A slot is written again kItemSlots items later.  By then all have read it: once the
  // loads of an item have been issued, all but kStages (6) of the k-blocks so far have been multiplied, so at most 6 items are
  // still to come for the multiplying thread, and at most two more (the accumulators) for the epilogues.
  uint32_t item_seq = 0;
  [[maybe_unused]] auto written_item = [&]() -> int {
    if (num_items <= num_pairs) return num_items;   // one each, nothing is written down
    const uint32_t slot = item_seq % kItemSlots, ph = (item_seq / kItemSlots) & 1;
    ++item_seq;
    const bool there = cta == 0 ? mbar_wait(islot0 + 8 * slot, ph, wc, 22) : mbar_wait_cluster(islot0 + 8 * slot, ph, wc, 22);
    const int item = there ? item_slots[slot] : num_items;
    return __shfl_sync(0xffffffffu, item, 0);   // the same in all lanes, also for the compiler
  };
  auto following = [&](int item) -> int {
    if constexpr (kMode == kModeGroup) return written_item();
    return item + num_pairs;
  };
  if (kMode == kModeGroup && warp == 0) {
    // ------------------------------------------------------------------ TMA producer of a group (both CTAs)
    // The whole warp walks the items, so that what depends on them stays in uniform registers, and one thread issues.
    if constexpr (kMode == kModeGroup) {
      uint32_t it = 0;
      int item = pair, next = num_items;
      Place w = first_place, w_next{};
      const uint32_t leader_full0 = mapa_shared(full0, 0);
      for (; item < num_items; item = next, w = w_next) {
        if (cta == 0 && num_items > num_pairs) {   // the next item is written down and the one after it asked for before this one is loaded
          taken(ahead);
          next = __shfl_sync(0xffffffffu, ahead, 0);
          const uint32_t slot = item_seq++ % kItemSlots;
          if (lane == 0) {
            item_slots[slot] = next;
            mbar_arrive(islot0 + 8 * slot);
            st_async_arrive(mapa_shared(smem_u32(const_cast<int*>(item_slots + slot)), 1), next, mapa_shared(islot0 + 8 * slot, 1));
          }
          if (next < num_items) ahead = take();
        }
        const GroupProblem& q = owners.prob[w.pi];
        const CUtensorMap *map_a = &owners.a[w.pi], *map_b = &owners.b[w.pi];
        const int a_mn = q.a_mn, b_mn = q.b_mn, q_bn = q.bn;
        const int m0 = w.tm * 256 + static_cast<int>(cta) * BMH, n0 = w.tn * q_bn + static_cast<int>(cta) * (q_bn / 2);
        bool ok = true;
        auto load = [&](int kb0, int kb1) {
          ok = load_blocks<kStages>(a_mn, b_mn, map_a, map_b, kb0, kb1, m0, n0, q_bn == BN, it, base, empty0, full0, leader_full0, cta == 0,
                                    static_cast<uint32_t>(2 * kATile + q_bn * BK * 2), wc);
        };
        const int head = min(w.kb1, w.kb0 + kStages);
        if (elect_one()) load(w.kb0, head);
        it += head - w.kb0;
        __syncwarp();
        // the rest of the item is loaded as the ring empties: time to find the place of the next one
        if (cta != 0) next = written_item();
        if (next < num_items) w_next = place_of(next);
        if (elect_one() && ok) load(head, w.kb1);
        it += w.kb1 - head;
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      if (cta == 0 && lane == 0 && item < num_items) {   // given up: the counter is left as the next launch expects it
        taken(ahead);   // the answer that had not been looked at may be the last one
        while (ahead < num_items) taken(ahead = take());
      }
    }
  } else if (kMode == kModeGroup && warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of a group (leader only)
    if constexpr (kMode == kModeGroup) {
      if (cta == 0) {
        uint32_t it = 0, local_tile = 0;
        int item = pair, next;
        Place w = place_of(item), w_next{};
        for (; item < num_items; item = next, w = w_next, ++local_tile) {
          next = written_item();   // ahead of the products: they are issued without a pause between two items
          if (next < num_items) w_next = place_of(next);
          const GroupProblem& q = owners.prob[w.pi];
          const uint32_t acc = local_tile & 1, acc_ph = (local_tile >> 1) & 1;
          const uint32_t idesc = make_idesc_bf16(256, q.bn, q.a_mn != 0, q.b_mn != 0);
          const uint32_t d_tmem = tmem_base + acc * BN;
          bool ok = true;
          if (elect_one()) {
            ok = mbar_wait(tempty0 + 8 * acc, acc_ph ^ 1, wc, 12);
            tc_fence_after();
            ok = ok && multiply_blocks<kStages>(w.kb1 - w.kb0, it, d_tmem, idesc, q.a_mn, q.b_mn, base, full0, empty0, wc);
            if (ok) {
              umma_commit_pair(mapa_shared(tfull0 + 8 * acc, 0));
              umma_commit_pair(mapa_shared(tfull0 + 8 * acc, 1));
            }
          }
          if (!__all_sync(0xffffffffu, ok)) break;
          it += w.kb1 - w.kb0;
        }
      }
    }
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      // gather mode: wait (bounded) until every chunk of 256-row group `g` of the gathered matrix is in local memory
      // groups already known complete: in address order a running count is enough (the reduction dimension is
      // walked front to back); a rotated walk keeps a bitmask of the first 512 groups (later ones are re-checked)
      int groups_ready = 0;
      uint32_t ready[16] = {0};
      const bool rotated = p.rot_kb != 0 || p.rot_n != 0;
      auto wait_group = [&](int g) -> bool {
        if (!rotated) {
          if (g < groups_ready) return true;
        } else if (g < 512 && ((ready[g >> 5] >> (g & 31)) & 1u)) {
          return true;
        }
        const long long group_bytes = static_cast<long long>(min(BN, p.w_rows - g * BN)) * p.w_cols * 2;
        const unsigned int target =
            static_cast<unsigned int>((group_bytes + kFetchChunkBytes - 1) / kFetchChunkBytes) * kFetchWarps;
        const uint64_t t0 = globaltimer_ns();
        unsigned int seen;
        while (true) {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.panel_flags + g) : "memory");
          if (seen >= target) break;
          if (*abort_flag) return false;
          if (globaltimer_ns() - t0 > kWaitBudgetNs) {
            *abort_flag = 1;
            report(p.status, kErrPipelineTimeout, 25, g);
            return false;
          }
          __nanosleep(64);
        }
        asm volatile("fence.proxy.async;" ::: "memory");  // generic-proxy stores -> visible to TMA reads
        if (!rotated) {
          if (p.b_mn) groups_ready = g + 1;
        } else if (g < 512) {
          ready[g >> 5] |= 1u << (g & 31);
        }
        return true;
      };
      uint32_t it = 0;
      bool ok = true;
      const uint32_t leader_full0 = mapa_shared(full0, 0);
      int tm = first_tm, tn = first_tn;
      for (int item = pair; item < num_items && ok; item += num_pairs) {
        int kb0, k_blocks;
        k_range(item, &kb0, &k_blocks);
        const int m0 = tm * 256 + static_cast<int>(cta) * BMH;   // this CTA's rows of A and C
        const int n0 = kMode == kModeSwiglu ? tn * (bn / 2) + static_cast<int>(cta) * p.N
                                            : tn * bn + static_cast<int>(cta) * (bn / 2);   // this CTA's rows of B
        if constexpr (kMode == kModeGather) {
          // B K-major (forward): the 256 weight rows this tile multiplies must have landed in local memory first
          if (!p.b_mn && !(ok = wait_group(tn))) break;
          for (int kb = kb0; kb < k_blocks; ++kb, ++it) {
            // B MN-major (input gradient): the gathered rows are the reduction dimension, 4 k-blocks per group
            const int at = p.rot_kb ? (kb + p.rot_kb) % k_blocks : kb;
            if (p.b_mn && !(ok = wait_group(at * BK / BN))) break;
            if (!(ok = load_blocks<kStages>(p.a_mn, p.b_mn, &tmap_a, &tmap_b, at, at + 1, m0, n0, true, it, base, empty0, full0, leader_full0,
                                            cta == 0, static_cast<uint32_t>(2 * kStageBytes), wc))) break;
          }
        } else {
          ok = load_blocks<kStages>(p.a_mn, p.b_mn, &tmap_a, &tmap_b, kb0, k_blocks, m0, n0, bn == BN, it, base, empty0, full0, leader_full0,
                                    cta == 0, static_cast<uint32_t>(2 * kATile + bn * BK * 2), wc);
          it += k_blocks - kb0;
        }
        if (item + num_pairs < num_items) tile_coords(tile_of(item + num_pairs), p, &tm, &tn);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    if (cta == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(256, bn, p.a_mn != 0, p.b_mn != 0);
      uint32_t it = 0, local_tile = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += num_pairs, ++local_tile) {
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_ph = (local_tile >> 1) & 1;
        if (!(ok = mbar_wait(tempty0 + 8 * acc, acc_ph ^ 1, wc, 12))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        int kb0, k_blocks;
        k_range(item, &kb0, &k_blocks);
        ok = multiply_blocks<kStages>(k_blocks - kb0, it, d_tmem, idesc, p.a_mn, p.b_mn, base, full0, empty0, wc);
        it += k_blocks - kb0;
        if (ok) {
          umma_commit_pair(mapa_shared(tfull0 + 8 * acc, 0));
          umma_commit_pair(mapa_shared(tfull0 + 8 * acc, 1));
        }
      }
    }
  } else if (kMode == kModeGather && warp >= 6) {
    // ------------------------------------------------------------------ shard fetch (every CTA of the grid)
    // The owners' shards are copied into the local B buffer in address order (= group order): 64 KiB per step and
    // CTA, 16 KiB per warp with 16 x 16-byte peer loads in flight per lane; after its part a warp makes the stores
    // visible and counts them on the group's flag.
    const int fw = warp - 6;
    const long long total_bytes = static_cast<long long>(p.w_rows) * p.w_cols * 2;
    const long long shard_bytes = static_cast<long long>(p.rows_per_rank) * p.w_cols * 2;
    const long long panel_bytes_full = static_cast<long long>(BN) * p.w_cols * 2;  // a multiple of the chunk size
    const long long n_chunks = (total_bytes + kFetchChunkBytes - 1) / kFetchChunkBytes;
    for (long long c0 = blockIdx.x; c0 < n_chunks; c0 += gridDim.x) {
      // rotated: this rank's own rows first, then the next owner's, ...
      const long long c = p.fetch_rot ? (c0 + p.fetch_rot) % n_chunks : c0;
      const long long byte0 = c * kFetchChunkBytes + fw * kFetchWarpBytes;
      const long long last = min(byte0 + kFetchWarpBytes, total_bytes) - 1;
      const int owner0 = static_cast<int>(byte0 / shard_bytes);
      const bool one_owner = byte0 < total_bytes && owner0 == static_cast<int>(last / shard_bytes);
      const unsigned char* src0 = one_owner
          ? reinterpret_cast<const unsigned char*>(p.shard_ptrs[owner0]) - static_cast<long long>(owner0) * shard_bytes
          : nullptr;
      uint4 r[16];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int v = 0; v < 16; ++v) {
          const long long b = byte0 + (static_cast<long long>(half * 16 + v) * 32 + lane) * 16;
          if (b < total_bytes) {
            if (one_owner) {
              r[v] = ld_stream_v4(src0 + b);
            } else {
              const int owner = static_cast<int>(b / shard_bytes);
              r[v] = ld_stream_v4(reinterpret_cast<const unsigned char*>(p.shard_ptrs[owner]) + (b - owner * shard_bytes));
            }
          }
        }
#pragma unroll
        for (int v = 0; v < 16; ++v) {
          const long long b = byte0 + (static_cast<long long>(half * 16 + v) * 32 + lane) * 16;
          if (b < total_bytes) *reinterpret_cast<uint4*>(p.b_local + b) = r[v];
        }
      }
      __threadfence();
      __syncwarp();
      if (lane == 0) {
        const int panel = static_cast<int>((c * kFetchChunkBytes) / panel_bytes_full);
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.panel_flags + panel) : "memory");
      }
    }
  } else if (kMode == kModeSwigluBwd && warp == 6) {
    // ------------------------------------------------------------------ boxes of gate and up (both CTAs)
    if (elect_one()) {
      uint32_t n = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += num_pairs) {
        int tm, tn;
        tile_coords(item, p, &tm, &tn);
        const int m0 = tm * 256 + static_cast<int>(cta) * BMH;
        if (m0 >= p.M) continue;
        for (int col = tn * BN; col < min(p.N, tn * BN + BN); col += 64, ++n) {
          if (!(ok = mbar_wait(gempty, (n & 1) ^ 1, wc, 19))) break;
          mbar_arrive_expect_tx(gfull, 2 * kStagingBytes);
          const uint32_t dst = base + kStages * kStageBytes;
          tma_load_2d(dst, &tmap_c, gfull, col, m0);
          tma_load_2d(dst + kStagingBytes, &tmap_c, gfull, p.N + col, m0);
        }
      }
    }
  } else if (warp >= 2 && warp < 6) {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int quad = warp & 3;  // TMEM lanes [32*quad, 32*quad+32) belong to this warp
    uint32_t local_tile = 0;
    uint32_t box_ctr = 0;
    int last_boxes = 0;
    [[maybe_unused]] uint32_t gu_ctr = 0;
    bool ok = true;
    const uint32_t tempty_leader0 = mapa_shared(tempty0, 0);
    [[maybe_unused]] uint32_t part_ctr = 0;
    for (int item = pair, next_item; item < num_items && ok; item = next_item, ++local_tile) {
      int tm, tn;
      [[maybe_unused]] Place place{};
      if constexpr (kMode == kModeGroup) {
        place = place_of(item);
        tm = place.tm; tn = place.tn;
      } else {
        tile_coords(tile_of(item), p, &tm, &tn);
      }
      const bool part = kMode == kModePlain && is_part(item), f32 = part || p.c_is_f32;
      next_item = following(item);   // kModeGroup: written down when the loads of this one were issued
      // The ring is idle under the last epilogue of the CTA: every box gets a place of its own there and none waits for the
      // one before it to be read.
      const bool last = next_item >= num_items;
      const int m0 = tm * 256 + static_cast<int>(cta) * BMH;
      int tile_cols = bn;
      if constexpr (kMode == kModeGroup) tile_cols = owners.prob[place.pi].bn;
      const int n0 = tn * tile_cols;
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      const int my_row = quad * 32 + lane;
      const int row = m0 + my_row;
      [[maybe_unused]] const bool row_ok = row < p.M;
      // the first `n` (a multiple of 8) of 64 values of a row, and their addition
      [[maybe_unused]] auto load64 = [](const __nv_bfloat16* src, int n, uint4* v) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 8 * i < n ? *reinterpret_cast<const uint4*>(src + 8 * i) : make_uint4(0, 0, 0, 0);
      };
      [[maybe_unused]] auto add64 = [](uint32_t* r, const uint4* v) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t o[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            r[8 * i + 2 * k] = __float_as_uint(__uint_as_float(r[8 * i + 2 * k]) + lo(o[k]));
            r[8 * i + 2 * k + 1] = __float_as_uint(__uint_as_float(r[8 * i + 2 * k + 1]) + hi(o[k]));
          }
        }
      };
      // The tile's bias is asked for while the products run, eight columns a lane, and passed around by shuffles.
      [[maybe_unused]] uint4 bias8 = make_uint4(0, 0, 0, 0);
      constexpr bool kBias = kMode == kModePlain || kMode == kModeGather || kMode == kModeRope;
      [[maybe_unused]] const bool biased = kBias && p.bias != nullptr && !part;
      if constexpr (kBias) {
        if (biased && n0 + 8 * lane < p.N) {
          const __nv_bfloat16* from = p.bias + n0 + 8 * lane;
          // a bias may be a view of anything; kModeRope is only launched with one that starts on a 16-byte boundary
          if (kMode == kModeRope || (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
            bias8 = *reinterpret_cast<const uint4*>(from);
          } else {
            const auto two = [&](int i) {
              return static_cast<uint32_t>(__bfloat16_as_ushort(from[i])) | static_cast<uint32_t>(__bfloat16_as_ushort(from[i + 1])) << 16;
            };
            bias8 = make_uint4(two(0), two(2), two(4), two(6));
          }
        }
      }
      // its values of `kCols` columns from `col` on (multiples of 16), added to accumulators
      [[maybe_unused]] auto add_bias = [&](auto n_cols, int col, auto* r) {
        const uint32_t b4[4] = {bias8.x, bias8.y, bias8.z, bias8.w};
#pragma unroll
        for (int i = 0; i < decltype(n_cols)::value / 2; ++i) {
          const uint32_t b = __shfl_sync(0xffffffffu, b4[i & 3], (col >> 3) + (i >> 2));
          if constexpr (sizeof(r[0]) == sizeof(uint32_t) && std::is_integral_v<std::remove_reference_t<decltype(r[0])>>) {
            r[2 * i] = __float_as_uint(__uint_as_float(r[2 * i]) + lo(b));
            r[2 * i + 1] = __float_as_uint(__uint_as_float(r[2 * i + 1]) + hi(b));
          } else {
            r[2 * i] += lo(b);
            r[2 * i + 1] += hi(b);
          }
        }
      };
      // The angles of a row's heads: those of narrow heads, four of which share a tile, are worked out while the products run (for
      // wide ones there are not the registers, and a row of a tile has only two heads).
      [[maybe_unused]] float at = 0.f, cosines[kMode == kModeRope ? 32 : 1], sines[kMode == kModeRope ? 32 : 1];
      if constexpr (kMode == kModeRope) {
        at = row_ok ? static_cast<float>(p.pos[row]) : 0.f;
        if (p.head_dim == 64) {
#pragma unroll
          for (int i = 0; i < 32; ++i) sincosf(at * rope_freq[i], &sines[i], &cosines[i]);
        }
      }
      [[maybe_unused]] float result_scale = 1.f;
      if constexpr (kMode == kModeGroup) {
        const GroupProblem& q = owners.prob[place.pi];
        result_scale = q.scale;
        if (q.scale_ptr != nullptr) result_scale *= *q.scale_ptr;
      }
      // the residual's first box is asked for while the products run (1000 x 1536 x 1536: 3 us more than without a residual, box by box)
      [[maybe_unused]] const __nv_bfloat16* rrow = nullptr;
      [[maybe_unused]] uint4 res[8];
      if constexpr (kMode == kModePlain || kMode == kModeGather) {
        if (p.residual != nullptr && !part && row_ok) rrow = p.residual + static_cast<long long>(row) * p.ldr + n0;
        if (rrow != nullptr) load64(rrow, p.N - n0, res);
      }
      if (!(ok = mbar_wait(tfull0 + 8 * acc, acc_ph, wc, 14))) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN;
      // A warp's 32 rows of one box, 64 columns of bf16 or 32 of fp32 (32 registers per row), are staged in shared memory of its own
      // and handed to the TMA unit by the warp itself: no warp waits for another, as all four did at every box of 128 rows.  What
      // a last epilogue waited for besides was the release of its accumulator to the other CTA (1500 clocks, and nobody takes it any
      // more) and the residual and bias box by box.  From the first launch of a chain to the next, before and now: 1900 x 512 x 512
      // 8.3 and 7.4 us, 1000 x 1536 x 1536 13.2 and 12.3, with a residual 16.1 and 13.7, with a bias 22.1 and 13.5; 16321 x 3072 x
      // 2048 with a bias 167 and 133; fp32 results, in four times as many boxes, 16320 x 2048 x 2048 96 and 96, K = 512 47 and 38, added
      // 102 and 103, 68 and 64, 2048 x 2048 x 8192 53 and 52.
      const bool rows_in = m0 + quad * 32 < (kMode == kModeGroup ? owners_rows(owners, place.pi) : p.M);
      auto emit = [&](const uint32_t* v32, const CUtensorMap* map, int col0, int row0, bool add = false) {
        uint8_t* slab = (last ? smem + last_boxes * kStagingBytes : staging + (box_ctr & 1u) * kStagingBytes) + quad * 4096;
        if (!last && box_ctr >= 2) {   // the box before the last one has been read
          if (elect_one()) bulk_wait_group_read1();
          __syncwarp();
        }
        uint8_t* srow = slab + lane * 128;
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<uint4*>(srow + ((v ^ (lane & 7)) << 4)) =
              make_uint4(v32[4 * v], v32[4 * v + 1], v32[4 * v + 2], v32[4 * v + 3]);
        fence_proxy_async();
        __syncwarp();
        if (elect_one()) {
          if (rows_in) {
            if (add) tma_reduce_add_2d(map, smem_u32(slab), col0, row0 + quad * 32);
            else tma_store_2d(map, smem_u32(slab), col0, row0 + quad * 32);
          }
          bulk_commit_group();
        }
        if (last) ++last_boxes; else ++box_ctr;
      };
      if constexpr (kMode == kModeSwiglu || kMode == kModeLogits || kMode == kModeSwigluBwd || kMode == kModeGroup || kMode == kModeRope) {
        if constexpr (kMode == kModeRope) {
          const int cols = m0 >= p.M ? 0 : min(tile_cols, p.N - n0);
          auto read16 = [&](int col, float* x) {   // 16 columns of this row, with their bias
            uint32_t r[16];
            tmem_ld_32x16(t_row + col, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(r[i]);
            if (biased) add_bias(std::integral_constant<int, 16>{}, col, x);
          };
          auto rounded = [](float x) { return __bfloat162float(__float2bfloat16(x)); };
          // one head: halves of kHalf columns, packed next to one another; `angle` gives cosine and sine
          auto head = [&](auto half, int col, uint32_t* v, auto angle) {
            constexpr int kHalf = decltype(half)::value;
#pragma unroll
            for (int c = 0; c < kHalf; c += 16) {
              float a[16], b[16];
              read16(col + c, a);
              read16(col + kHalf + c, b);
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                float sn, cn;
                angle(c + i, &sn, &cn);
                rotate_pair(rounded(a[i]), rounded(b[i]), cn, sn, &a[i], &b[i]);   // as the stand-alone pass reads them
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                v[c / 2 + i] = pack2(a[2 * i], a[2 * i + 1]);
                v[(kHalf + c) / 2 + i] = pack2(b[2 * i], b[2 * i + 1]);
              }
            }
          };
#pragma unroll 1
          for (int col = 0; col < cols;) {
            uint32_t v[64];
            if (n0 + col >= p.rot_cols) {   // v heads
#pragma unroll
              for (int c = 0; c < 64; c += 16) {
                float a[16];
                read16(col + c, a);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[c / 2 + i] = pack2(a[2 * i], a[2 * i + 1]);
              }
              emit(v, &tmap_c, n0 + col, m0);
              col += 64;
            } else if (p.head_dim == 64) {
              head(std::integral_constant<int, 32>{}, col, v, [&](int i, float* sn, float* cn) { *sn = sines[i]; *cn = cosines[i]; });
              emit(v, &tmap_c, n0 + col, m0);
              col += 64;
            } else {
              head(std::integral_constant<int, 64>{}, col, v, [&](int i, float* sn, float* cn) { sincosf(at * rope_freq[i], sn, cn); });
              emit(v, &tmap_c, n0 + col, m0);
              emit(v + 32, &tmap_c, n0 + col + 64, m0);
              col += 128;
            }
          }
        } else if constexpr (kMode == kModeGroup) {
          const GroupProblem& q = owners.prob[place.pi];
          const CUtensorMap* map = &owners.c[place.pi];
          const int cols = m0 >= q.M ? 0 : min(tile_cols, q.N - n0);
          if (q.out != 0) {
            const bool add = q.out == 2;
#pragma unroll 1
            for (int col = 0; col < cols; col += 32) {
              uint32_t r[32];
              tmem_ld_32x32(t_row + col, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * result_scale);
              emit(r, map, n0 + col, m0, add);
            }
          } else {
            // A part: 16 bytes of 128 rows next to one another, so that a warp writes and reads whole lines.
            const float4* others = nullptr;
            bool mine = true;
            if (place.divided >= 0) {
              const int tile = q.first_split_tile + place.divided;
              // parts of the tile, this CTA's half of each
              float4* at = owners.parts + ((q.first_part + static_cast<long long>(place.divided) * q.splits) * 2 + cta) * (64 * 128) + my_row;
              float4* own = at + static_cast<long long>(place.part) * (2 * 64 * 128);
#pragma unroll 1
              for (int col = 0; col < cols; col += 32) {
                uint32_t r[32];
                tmem_ld_32x32(t_row + col, r);
                tmem_ld_wait();
#pragma unroll
                for (int v = 0; v < 8; ++v)
                  __stcg(own + (col / 4 + v) * 128, make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]),
                                                                __uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3])));
              }
              __threadfence();
              __syncwarp();
              if (lane == 0) mbar_arrive(pready);
              if (warp == 2 && lane == 0 && mbar_wait(pready, part_ctr & 1, wc, 23)) {
                __threadfence();
                unsigned int* ctr = owners.arrived + 2 * tile + cta;
                const bool all = atomicInc(ctr, q.splits - 1) == static_cast<unsigned int>(q.splits) - 1;   // and back to zero
                __threadfence();
                *part_last = all;
                mbar_arrive(pcounted);
              }
              __syncwarp();
              if (!(ok = mbar_wait(pcounted, part_ctr & 1, wc, 24))) break;
              ++part_ctr;
              mine = *part_last != 0;
              others = at;
            }
            if (mine) {
#pragma unroll 1
              for (int col = 0; col < cols; col += 64) {
                uint32_t r[64], v[32];
                tmem_ld_32x32(t_row + col, r);
                tmem_ld_32x32(t_row + col + 32, r + 32);
                tmem_ld_wait();
                if (others != nullptr) {
                  // in the order of the parts; this one's from the accumulator
                  float f[64];
#pragma unroll
                  for (int i = 0; i < 64; ++i) f[i] = 0.f;
#pragma unroll 1
                  for (int s = 0; s < q.splits; ++s) {
                    if (s == place.part) {
#pragma unroll
                      for (int i = 0; i < 64; ++i) f[i] += __uint_as_float(r[i]);
                    } else {
                      const float4* src = others + static_cast<long long>(s) * (2 * 64 * 128) + (col / 4) * 128;
                      float4 x[16];
#pragma unroll
                      for (int i = 0; i < 16; ++i) x[i] = __ldcg(src + i * 128);
#pragma unroll
                      for (int i = 0; i < 16; ++i) {
                        f[4 * i] += x[i].x; f[4 * i + 1] += x[i].y; f[4 * i + 2] += x[i].z; f[4 * i + 3] += x[i].w;
                      }
                    }
                  }
#pragma unroll
                  for (int i = 0; i < 64; ++i) r[i] = __float_as_uint(f[i]);
                }
                if (q.addend != nullptr) {
                  if (row < q.M) {
                    const float* from = q.addend + static_cast<long long>(row) * q.N + n0 + col;
                    const int left = cols - col;   // a multiple of 8
                    float4 x[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                      x[i] = 4 * i < left ? *reinterpret_cast<const float4*>(from + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                      r[4 * i] = __float_as_uint(__uint_as_float(r[4 * i]) + x[i].x);
                      r[4 * i + 1] = __float_as_uint(__uint_as_float(r[4 * i + 1]) + x[i].y);
                      r[4 * i + 2] = __float_as_uint(__uint_as_float(r[4 * i + 2]) + x[i].z);
                      r[4 * i + 3] = __float_as_uint(__uint_as_float(r[4 * i + 3]) + x[i].w);
                    }
                  }
                }
                if (result_scale != 1.f) {
#pragma unroll
                  for (int i = 0; i < 64; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * result_scale);
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                emit(v, map, n0 + col, m0);
              }
            }
          }
        } else
        if constexpr (kMode == kModeSwigluBwd) {
          const int n_boxes = m0 >= p.M ? 0 : min(BN, p.N - n0 + 63) / 64;
#pragma unroll 1
          for (int bx = 0; bx < n_boxes; ++bx, ++gu_ctr) {
            uint32_t d[32], g[32], u[32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t r[32];
              tmem_ld_32x32(t_row + bx * 64 + 32 * h, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) d[16 * h + i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            }
            if (!(ok = mbar_wait(gfull, gu_ctr & 1, wc, 21))) break;
            const uint8_t* row_gu = smem + kStages * kStageBytes + my_row * 128;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              const uint4 a = *reinterpret_cast<const uint4*>(row_gu + ((v ^ (my_row & 7)) << 4));
              const uint4 b = *reinterpret_cast<const uint4*>(row_gu + kStagingBytes + ((v ^ (my_row & 7)) << 4));
              g[4 * v] = a.x; g[4 * v + 1] = a.y; g[4 * v + 2] = a.z; g[4 * v + 3] = a.w;
              u[4 * v] = b.x; u[4 * v + 1] = b.y; u[4 * v + 2] = b.z; u[4 * v + 3] = b.w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(gempty);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              float dg[2], du[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float df = e ? hi(d[i]) : lo(d[i]), gf = e ? hi(g[i]) : lo(g[i]), uf = e ? hi(u[i]) : lo(u[i]);
                const float sig = 1.f / (1.f + __expf(-gf)), silu = gf * sig;
                du[e] = df * silu;
                dg[e] = df * uf * (sig + silu * (1.f - sig));
              }
              g[i] = pack2(dg[0], dg[1]);
              u[i] = pack2(du[0], du[1]);
            }
            emit(g, &owners.m[0], n0 + bx * 64, m0);
            emit(u, &owners.m[1], n0 + bx * 64, m0);
          }
        } else if constexpr (kMode == kModeLogits) {
          const long long label = row_ok ? p.labels[row] - n0 : -1;
          const int n_boxes = m0 >= p.M ? 0 : min(BN, p.N - n0 + 63) / 64;
          const float log2e_t = 1.4426950408889634f * p.inv_temp;
          float m = -INFINITY, s = 0.f;   // logits in units of log2(e)
#pragma unroll 1
          for (int bx = 0; bx < n_boxes; ++bx) {
            uint32_t v[32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t r[32];
              tmem_ld_32x32(t_row + bx * 64 + 32 * h, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) v[16 * h + i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            }
            const int left = p.N - n0 - bx * 64;   // a multiple of 8
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (2 * i < left) mx4[i & 3] = fmaxf(mx4[i & 3], fmaxf(lo(v[i]) * log2e_t, hi(v[i]) * log2e_t));
            const float m_new = fmaxf(m, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
            const float m_sub = m_new == -INFINITY ? 0.f : m_new;   // nothing but -inf so far: the sum stays zero, NaN stays NaN
            float s4[4] = {s * exp2f(m - m_sub), 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (2 * i < left) s4[i & 3] += exp2f(fmaf(lo(v[i]), log2e_t, -m_sub)) + exp2f(fmaf(hi(v[i]), log2e_t, -m_sub));
            s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
            m = m_new;
            if (label >= bx * 64 && label < bx * 64 + 64) {
              float x = 0.f;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (label - bx * 64 == 2 * i) x = lo(v[i]);
                if (label - bx * 64 == 2 * i + 1) x = hi(v[i]);
              }
              p.label_logits[row] = x;
            }
            if (p.store_logits) emit(v, &tmap_c, n0 + bx * 64, m0);
          }
          if (row_ok) p.row_stats[static_cast<long long>(tn) * p.M + row] = make_float2(m, s);
        } else {
#pragma unroll 1
        for (int bx = 0; bx < bn / 128; ++bx) {
          uint32_t gate[32], up[32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[64];
            tmem_ld_32x32(t_row + bx * 64 + 32 * h, r);
            tmem_ld_32x32(t_row + bn / 2 + bx * 64 + 32 * h, r + 32);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              gate[16 * h + i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
              up[16 * h + i] = pack2(__uint_as_float(r[32 + 2 * i]), __uint_as_float(r[32 + 2 * i + 1]));
            }
          }
          const int col0 = tn * (bn / 2) + bx * 64;
          if (col0 >= p.N || m0 >= p.M) continue;
          if (p.store_gate_up) {
            emit(gate, &owners.m[0], col0, m0);
            emit(up, &owners.m[1], col0, m0);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) {   // from the rounded halves, as the stand-alone pass reads them
            const float g0 = __uint_as_float(gate[i] << 16), g1 = __uint_as_float(gate[i] & 0xffff0000u);
            const float u0 = __uint_as_float(up[i] << 16), u1 = __uint_as_float(up[i] & 0xffff0000u);
            gate[i] = pack2(g0 / (1.f + __expf(-g0)) * u0, g1 / (1.f + __expf(-g1)) * u1);
          }
          emit(gate, &tmap_c, col0, m0);
        }
        }
      } else {
        const int cols = m0 >= p.M ? 0 : min(tile_cols, p.N - n0);
        if (f32) {
          // a CTA's 128 rows never straddle two owners (rows_per_rank is a multiple of 128)
          const int owner = kMode == kModeScatter ? m0 / p.rows_per_rank : 0;
          const CUtensorMap* map = kMode == kModeScatter || part ? &owners.m[owner] : &tmap_c;
          const int row0 = kMode == kModeScatter ? m0 - owner * p.rows_per_rank
                           : part ? (item - p.whole) * 256 + static_cast<int>(cta) * BMH : m0;
          const int first_col = part ? 0 : n0;
          const bool add = kMode == kModeScatter || (!part && p.accumulate);
#pragma unroll 1
          for (int col = 0; col < cols; col += 32) {
            uint32_t r[32];
            tmem_ld_32x32(t_row + col, r);
            tmem_ld_wait();
            if constexpr (kMode == kModeScatter) {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * p.scale);
            }
            if (biased) add_bias(std::integral_constant<int, 32>{}, col, r);
            emit(r, map, first_col + col, row0, add);
          }
        } else if (!biased && p.residual == nullptr) {
#pragma unroll 1
          for (int col = 0; col < cols; col += 64) {
            uint32_t r[64];
            tmem_ld_32x32(t_row + col, r);
            tmem_ld_32x32(t_row + col + 32, r + 32);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            emit(r, &tmap_c, n0 + col, m0);
          }
        } else {
#pragma unroll 1
          for (int col = 0; col < cols; col += 64) {
            uint32_t r[64];
            tmem_ld_32x32(t_row + col, r);
            tmem_ld_32x32(t_row + col + 32, r + 32);
            tmem_ld_wait();
            if (biased) add_bias(std::integral_constant<int, 64>{}, col, r);
            if (rrow != nullptr) {
              add64(r, res);
              load64(rrow + col + 64, cols - col - 64, res);   // of the next box, under the rest of this one
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            emit(r, &tmap_c, n0 + col, m0);
          }
        }
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      // the leader may overwrite this accumulator, if it has a use for it
      if (lane == 0 && (kMode == kModeGroup ? !last : item + 2 * num_pairs < num_items)) mbar_arrive_cluster_tmem(tempty_leader0 + 8 * acc);
    }
    if (elect_one()) {   // the thread that issued them: all output boxes have been read, or are in memory before an arrival is reported
      if constexpr (kMode == kModeScatter || kMode == kModeGroup) bulk_wait_group0();
      else bulk_wait_group_read0();
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  // Nothing is reported to the partner's barriers, or read from its shared memory, after this.  Where all that a thread reported has
  // been waited for, nothing is left to be ordered (a release waits 1000 clocks for the memory system); in a group with further
  // items the last accumulator but one is given back to nobody.
  if (kMode != kModeGroup || num_items <= num_pairs) cluster_sync_exit();
  else cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
  if constexpr (kMode == kModeScatter || kMode == kModeGroup) {
    // the last CTA to finish reports to every owner's counter, unless any CTA of the launch gave up
    unsigned long long arrivals = 1;
    if constexpr (kMode == kModeGroup) arrivals = owners.arrivals;
    if (arrivals > 0)
      finish_and_signal(p.ctr_ptrs, p.nranks, p.done_slot, arrivals,
                        [&] { return !*abort_flag && (p.status == nullptr || *reinterpret_cast<volatile int*>(p.status) == 0); });
  }
}

// The divided tiles of C: the sum of their fp32 partial tiles, in order, + bias + residual, narrowed to bf16.  Eight columns
// per thread, 32 CTAs per tile.
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ c, long long ldc,
                 const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ residual, const Params p) {
  const int i = blockIdx.x >> 5;
  int tm, tn;
  tile_coords(p.whole + i, p, &tm, &tn);
  const int r = (blockIdx.x & 31) * 8 + (threadIdx.x >> 5), k8 = (threadIdx.x & 31) * 8;
  const int row = tm * 256 + r, col = tn * BN + k8;
  if (row >= p.M || col >= p.N) return;
  const float* src = partial + (static_cast<long long>(i) * p.splits * 256 + r) * BN + k8;
  float f[8] = {};
  for (int s = 0; s < p.splits; ++s, src += 256 * BN) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
    f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
  }
  if (bias != nullptr) {
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] += __bfloat162float(bias[col + k]);
  }
  if (residual != nullptr) {
    const uint4 res = *reinterpret_cast<const uint4*>(residual + row * p.ldr + col);
    const uint32_t u[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      f[2 * k] += __uint_as_float(u[k] << 16);
      f[2 * k + 1] += __uint_as_float(u[k] & 0xffff0000u);
    }
  }
  *reinterpret_cast<uint4*>(c + row * ldc + col) =
      make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

}  // namespace gemm_pair

// ODC_GEMM_ROTATE: 0 (default) every rank walks the owners in address order; 1: the forward gather and the
// weight-gradient scatter start at the rank's own rows and walk the owners from there; 2: the input-gradient
// gather (rotated k loop) as well.  Measured on 8 GPUs with all ranks launching the same kernel at once, rotation
// makes the forward kernels faster (0.863 -> 0.799 ms and 1.247 -> 0.766 ms on the two widest weights) and the
// input-gradient kernel slower; a whole training step, where ranks are not in lock-step anyway, measured slower with
// it, so it is off unless asked for.
static int rotate_mode() {
  static const int mode = [] {
    const char* e = getenv("ODC_GEMM_ROTATE");
    return e == nullptr ? 0 : atoi(e);
  }();
  return mode;
}

// Which tiles are divided, and how many ways, where the last round of tiles (or the only one) leaves pairs idle.  In units of
// a k-block (512 clocks of the tensor cores, 0.28 us): a product takes as many rounds as its items need, each as long as its
// longest item.  Dividing a bf16 product adds a second launch (3 us: 11 units) and writes and reads the fp32 partials once
// (at 5 TB/s, 1.4 MB per unit); a scattered one only adds the parts to the accumulators, once more each, and what other ranks
// own crosses the link (770 GB/s, 0.216 MB per unit; priced as if nothing ran meanwhile, not measured on several GPUs).  All
// tiles are divided only where that is a tenth faster, those of the last rounds where it is a twentieth.
// All tiles: 765 x 1536 with K = 8960: 59 us whole, 29 us divided by four with the sum.  The last rounds, weight gradients
// over 16321 rows: 3072 x 2048 (96 tiles on 74 pairs) 197 us whole, now 158; 2048 x 8192 410 and 370; over 30000 rows
// 4096 x 4096 750 and 709.
struct SplitPlan {
  int whole, splits, kb_split;
};
struct SplitCost {   // in units: of dividing at all, and per MB of fp32 parts
  double fixed, per_mb;
};
constexpr SplitCost kPartialsCost{11.0, 2 / 1.4};
static SplitCost scatter_cost(int nranks) {
  const double remote = static_cast<double>(nranks - 1) / nranks;
  return {2.0, (1 - remote) / 1.4 + remote / 0.216};
}
static SplitPlan plan_splits(int M, int N, int K, int sm_count, const SplitCost& dividing, bool tail) {
  using namespace gemm_pair;
  const int tiles = (M + 255) / 256 * ((N + BN - 1) / BN), pairs = sm_count / 2;
  const int kb = (K + BK - 1) / BK, rounds = (tiles + pairs - 1) / pairs;
  double best = (tail ? 0.95 : 0.9) * rounds * kb;
  SplitPlan plan{tiles, 1, kb};
  for (int full = tail ? std::max(0, tiles / pairs - 1) : 0; full <= tiles / pairs; ++full) {
    const int rest = tiles - full * pairs;
    if (rest == 0 || (!tail && tiles >= pairs)) continue;
    for (int want = 2; want <= 8; ++want) {
      const int each = (kb + want - 1) / want, s = (kb + each - 1) / each;   // no empty part
      if (s < 2) break;
      const long long items = static_cast<long long>(rest) * s;
      const double mb = items * 0.262144;
      const double cost = static_cast<double>(full) * kb + static_cast<double>((items + pairs - 1) / pairs) * each +
                          dividing.fixed + mb * dividing.per_mb;
      if (cost < best) { best = cost; plan = SplitPlan{full * pairs, s, each}; }
    }
  }
  return plan;
}

// Whether an undivided product is taken in tiles of 256 x 128: a k-block of one takes 0.6 of the time, its epilogue half, so it is
// where as many rounds of them are shorter.  Twice as many tiles that still have a pair each: 300 x 512 x 512 6.8 us, half as wide
// 5.1, 1000 x 1536 x 1536 11.9 and 8.0, 512 x 4096 x 4096 24.3 and 15.1; three rounds instead of two: 1500 x 4096 x 4096 45.0 and
// 38.4, 4000 x 1536 x 1536 20.0 and 17.9; two instead of one 1900 x 2048 x 2048 15.5 and 15.8, six instead of three 6000 x 2048 x
// 2048 36.4 and 40.0.  Weight gradients, whose two operands take three loads a k-block, 0.75: 3000 x 2048 x 2048 26.1 and 30.0.
// The logits have many rounds of tiles at any number of tokens; the SwiGLU backward, scattered weight gradients and gathered weights
// were not tried in half tiles and keep whole ones.
static double half_tile_time(int layout) { return layout == 2 ? 0.75 : 0.6; }
static bool half_tiles_pay(int tiles, int half_tiles, int layout, int sm_count) {
  const int pairs = sm_count / 2;
  return (half_tiles + pairs - 1) / pairs * half_tile_time(layout) < 0.95 * ((tiles + pairs - 1) / pairs);
}
static bool half_tiles_pay_for(int M, int N, int layout, int sm_count) {
  const int rows = (M + 255) / 256;
  return half_tiles_pay(rows * ((N + 255) / 256), rows * ((N + 127) / 128), layout, sm_count);
}

// The plan of a bf16 product: all tiles divided where they are fewer than the pairs, else those of its last rounds.
static SplitPlan product_plan(int M, int N, int K, int sm_count) {
  const SplitPlan all = plan_splits(M, N, K, sm_count, kPartialsCost, false);
  return all.splits > 1 || M < 256 ? all : plan_splits(M, N, K, sm_count, kPartialsCost, true);
}

GemmPlan gemm_plan(int M, int N, int K, int c_kind, int sm_count) {
  using namespace gemm_pair;
  const int tiles = (M + 255) / 256 * ((N + BN - 1) / BN);
  if (c_kind != kBF16 || M < 1 || N < 256 || K < BK || sm_count < 2) return {tiles, tiles, 1, 0};
  const SplitPlan plan = product_plan(M, N, K, sm_count);
  return {tiles, plan.whole, plan.splits, static_cast<size_t>(tiles - plan.whole) * plan.splits * 256 * BN * sizeof(float)};
}

// Returns cudaErrorNotSupported when the shape is not worth a CTA pair (the caller then uses the single-CTA kernel).
cudaError_t gemm_bf16_pair(const void* a, const void* b, void* c, int c_kind, const void* bias, int M, int N, int K,
                           int layout, bool accumulate, long long lda, long long ldb, long long ldc, int* status,
                           int sm_count, cudaStream_t stream, const void* residual, long long ldr, float* split_ws) {
  using namespace gemm_pair;
  // fewer rows than a tile are worth a pair only where several share the reduction (136 x 1536, K = 8960: 61 us on the
  // single-CTA kernel, 23 us; 200 x 2048, K = 8192: 57 us, 25 us)
  if ((M < 256 && split_ws == nullptr) || N < 256 || K < BK || sm_count < 2) return cudaErrorNotSupported;
  const bool a_mn = (layout == 2);
  const bool b_mn = (layout != 0);
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15)
    return cudaErrorMisalignedAddress;
  if ((lda % 8) || (ldb % 8) || (N % 8) || (ldc % (c_kind == kF32 ? 4 : 8))) return cudaErrorInvalidDevicePointer;
  if (c_kind != kF32 && accumulate) return cudaErrorNotSupported;

  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModePlain>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;

  CUtensorMap ta, tb, tc;
  if (!a_mn) {
    if (!encode_tile_map_2d(&ta, a, K, M, lda * 2, 64, BMH)) return cudaErrorInvalidPitchValue;
  } else {
    if (!encode_tile_map_2d(&ta, a, M, K, lda * 2, 64, 64)) return cudaErrorInvalidPitchValue;
  }
  SplitPlan plan{(M + 255) / 256 * ((N + BN - 1) / BN), 1, 0};
  if (split_ws != nullptr) plan = product_plan(M, N, K, sm_count);
  const int bn = plan.splits == 1 && half_tiles_pay_for(M, N, layout, sm_count) ? BN / 2 : BN;
  if (!b_mn) {
    if (!encode_tile_map_2d(&tb, b, K, N, ldb * 2, 64, bn / 2)) return cudaErrorInvalidTexture;
  } else {
    if (!encode_tile_map_2d(&tb, b, N, K, ldb * 2, 64, 64)) return cudaErrorInvalidTexture;
  }
  Params p{};
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (N + bn - 1) / bn;
  p.bn = bn;
  if (plan.splits == 1) plan.whole = p.tiles_m * p.tiles_n;
  p.whole = plan.whole; p.splits = plan.splits; p.kb_split = plan.kb_split;
  OwnerMaps scratch{};
  const int parts = (p.tiles_m * p.tiles_n - p.whole) * p.splits;
  if (parts > 0 && !encode_tile_map_2d_f32(&scratch.m[0], split_ws, BN, static_cast<uint64_t>(parts) * 256, BN * 4, 32, kOutRows))
    return cudaErrorInvalidValue;
  if (c_kind == kF32) {
    if (!encode_tile_map_2d_f32(&tc, c, N, M, ldc * 4, 32, kOutRows)) return cudaErrorInvalidValue;
  } else {
    if (!encode_tile_map_2d(&tc, c, N, M, ldc * 2, 64, kOutRows)) return cudaErrorInvalidValue;
  }
  p.bias = static_cast<const __nv_bfloat16*>(bias);   // the sum of the parts adds it where there are any
  p.M = M; p.N = N; p.K = K;
  p.c_is_f32 = c_kind == kF32;
  p.accumulate = accumulate ? 1 : 0;
  p.a_mn = a_mn; p.b_mn = b_mn;
  p.status = status;
  if (residual != nullptr) {
    if (c_kind != kBF16 || (ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15)) return cudaErrorInvalidValue;
    p.residual = static_cast<const __nv_bfloat16*>(residual);
    p.ldr = ldr;
  }
  const int items = p.whole + parts;
  const int pairs = items < sm_count / 2 ? items : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModePlain>, 2 * pairs, kThreads, kSmemBytes, stream, ta, tb, tc, scratch, p);
  if (parts > 0) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    launch(split_sum_kernel, parts / p.splits * 32, 256, 0, stream, static_cast<const float*>(split_ws),
        static_cast<__nv_bfloat16*>(c), ldc, p.bias, p.residual, p);
  }
  return cudaGetLastError();
}

// act[M, F] = silu(x Wg^T) * (x Wu^T) for w = [Wg; Wu], [2F, K]; gate_up [M, 2F] receives both products unless it is null.
// cudaErrorNotSupported where the plain product followed by the activation is the better form: fewer rows than a tile, or a
// reduction that is worth dividing.
cudaError_t gemm_swiglu_pair(const void* x, const void* w, void* gate_up, void* act, int M, int F, int K, long long ldx,
                             long long ldw, int* status, int sm_count, cudaStream_t stream) {
  using namespace gemm_pair;
  if (M < 256 || F < BNH || K < BK || sm_count < 2 || plan_splits(M, 2 * F, K, sm_count, kPartialsCost, false).splits > 1)
    return cudaErrorNotSupported;
  if ((ldx % 8) || (ldw % 8) || (F % 8) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gate_up) |
        reinterpret_cast<uintptr_t>(act)) & 15))
    return cudaErrorNotSupported;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeSwiglu>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb, tc;
  OwnerMaps halves{};
  const int row_tiles = (M + 255) / 256;   // 128 activations a tile, or 64
  const int bn = half_tiles_pay(row_tiles * ((F + 127) / 128), row_tiles * ((F + 63) / 64), 0, sm_count) ? BN / 2 : BN;
  const uint64_t ld_gu = static_cast<uint64_t>(F) * 4;
  if (!encode_tile_map_2d(&ta, x, K, M, ldx * 2, 64, BMH) || !encode_tile_map_2d(&tb, w, K, 2ull * F, ldw * 2, 64, bn / 2) ||
      !encode_tile_map_2d(&tc, act, F, M, static_cast<uint64_t>(F) * 2, 64, kOutRows))
    return cudaErrorInvalidValue;
  if (gate_up != nullptr) {  // each half clipped at its own last column
    if (!encode_tile_map_2d(&halves.m[0], gate_up, F, M, ld_gu, 64, kOutRows) ||
        !encode_tile_map_2d(&halves.m[1], static_cast<__nv_bfloat16*>(gate_up) + F, F, M, ld_gu, 64, kOutRows))
      return cudaErrorInvalidValue;
  }
  Params p{};
  p.M = M; p.N = F; p.K = K;
  p.store_gate_up = gate_up != nullptr;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (F + bn / 2 - 1) / (bn / 2);
  p.bn = bn;
  p.status = status;
  const int tiles = p.tiles_m * p.tiles_n;
  const int pairs = tiles < sm_count / 2 ? tiles : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeSwiglu>, 2 * pairs, kThreads, kSmemBytes, stream, ta, tb, tc, halves, p);
  return cudaGetLastError();
}

// The kernel is at the limit of 255 registers and spills 60 bytes of stores and 100 of loads a thread; what these cost was not measured
// apart (with the angles of all heads of a tile in registers it was 340 bytes and a tenth of its time, 10.4 -> 11.5 us).
// out[M, N] = x w^T (+ bias), w [N, K], with the columns below rot_cols, heads of 64 or 128, rotated by pos[row] (rotary base theta;
// halves of a head are the pairs, as in launch_rope_qkv): the rotation is not a pass over the projection (16321 tokens, 32 + 16
// heads of 64: 45 us), and runs while the next tile is multiplied.  The same bytes as the two passes: rounded, rotated, rounded.
// cudaErrorNotSupported where the product by itself would be divided, all of it or its last round (528 to 608 x 7168 x 5120): then the
// product and the pass.
cudaError_t gemm_rope_pair(const void* x, const void* w, const void* bias, void* out, const long long* pos, int M, int N, int K,
                           long long ldx, long long ldw, int rot_cols, int head_dim, float theta, int* status, int sm_count,
                           cudaStream_t stream) {
  using namespace gemm_pair;
  if (M < 256 || N < 256 || K < BK || sm_count < 2 || product_plan(M, N, K, sm_count).splits > 1) return cudaErrorNotSupported;
  if ((head_dim != 64 && head_dim != 128) || rot_cols % head_dim || N % 64 || rot_cols > N || (ldx % 8) || (ldw % 8) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out) |
        reinterpret_cast<uintptr_t>(bias)) & 15))
    return cudaErrorNotSupported;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeRope>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb, tc;
  const int bn = half_tiles_pay_for(M, N, 0, sm_count) ? BN / 2 : BN;   // a head is 128 columns at most
  if (!encode_tile_map_2d(&ta, x, K, M, ldx * 2, 64, BMH) || !encode_tile_map_2d(&tb, w, K, N, ldw * 2, 64, bn / 2) ||
      !encode_tile_map_2d(&tc, out, N, M, static_cast<uint64_t>(N) * 2, 64, kOutRows))
    return cudaErrorNotSupported;
  Params p{};
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.M = M; p.N = N; p.K = K;
  p.pos = pos; p.rot_cols = rot_cols; p.head_dim = head_dim; p.log2_theta = log2f(theta);
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (N + bn - 1) / bn;
  p.bn = bn;
  p.status = status;
  const int tiles = p.tiles_m * p.tiles_n;
  const int pairs = tiles < sm_count / 2 ? tiles : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeRope>, 2 * pairs, kThreads, kSmemBytes, stream, ta, tb, tc, OwnerMaps{}, p);
  return cudaGetLastError();
}

// dgate_up[M, 2F] = gradient of swiglu(gate_up) where the gradient of its result is dy w, w [K, F]: the activations' gradient is
// never written.  cudaErrorNotSupported where the plain product followed by the pass is the better form.  16321 tokens, 2048 and
// 8192 wide: the product 0.38 ms and the pass 0.22 (1.6 GB).
cudaError_t gemm_swiglu_bwd_pair(const void* dy, const void* w, const void* gate_up, void* dgate_up, int M, int F, int K,
                                 long long lddy, long long ldw, int* status, int sm_count, cudaStream_t stream) {
  using namespace gemm_pair;
  if (M < 256 || F < 256 || K < BK || sm_count < 2 || plan_splits(M, F, K, sm_count, kPartialsCost, false).splits > 1)
    return cudaErrorNotSupported;
  if ((lddy % 8) || (ldw % 8) || (F % 8) ||
      ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gate_up) |
        reinterpret_cast<uintptr_t>(dgate_up)) & 15))
    return cudaErrorNotSupported;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeSwigluBwd>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb, tc;
  OwnerMaps halves{};
  const uint64_t ld_gu = static_cast<uint64_t>(F) * 4;
  if (!encode_tile_map_2d(&ta, dy, K, M, lddy * 2, 64, BMH) || !encode_tile_map_2d(&tb, w, F, K, ldw * 2, 64, 64) ||
      !encode_tile_map_2d(&tc, gate_up, 2ull * F, M, ld_gu, 64, BMH) ||
      !encode_tile_map_2d(&halves.m[0], dgate_up, F, M, ld_gu, 64, kOutRows) ||   // each half clipped at its own last column
      !encode_tile_map_2d(&halves.m[1], static_cast<__nv_bfloat16*>(dgate_up) + F, F, M, ld_gu, 64, kOutRows))
    return cudaErrorNotSupported;
  Params p{};
  p.M = M; p.N = F; p.K = K;
  p.b_mn = 1;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (F + BN - 1) / BN;
  p.status = status;
  const int tiles = p.tiles_m * p.tiles_n;
  const int pairs = tiles < sm_count / 2 ? tiles : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeSwigluBwd>, 2 * pairs, Roles<kModeSwigluBwd>::kThreadsTotal, kSmemBytes, stream, ta, tb, tc,
      halves, p);
  return cudaGetLastError();
}

// Where the statistics in the epilogue are the better form of a head of M rows, N words and width K.  Against the plain product
// and the pass over its logits (times of that form over this one, log-probabilities / loss and its gradient):
//   - They lengthen the last epilogue by 3 us, so there has to be more than one round of tiles, or enough rows to keep the pass
//     busy for some waves: 256 rows and 4096 words, width 512: 0.81 / 0.77; 300 and 8192, 2048: 0.98 / 0.94; 800 and 4096: 1.07 /
//     1.00; 300 and 32000, 2048: 1.07 / 1.05; 4096 and 4096: 1.52 / 1.23.
//   - The product must not be one that is divided: 256 and 1024, width 4096: 0.52 / 0.51; 1200 and 1024: 0.87 / 0.84.
//   - With the logits to be stored as well an epilogue takes as long as 16 k-blocks of the next tile's products.  Below that width
//     the passes win where rows are long: 4096 and 128256, width 512: 0.94, 768 0.94, 1024 0.96, 1536 1.15; rows up to 16384 words
//     gain at any width (1.03 to 1.7 from 2000 rows on).
bool logits_stats_pay(int M, int N, int K, bool store_logits, int sm_count) {
  using namespace gemm_pair;
  if (M < 256 || N < 256 || K < BK || sm_count < 2) return false;
  const long long tiles = static_cast<long long>((M + 255) / 256) * logits_stat_tiles(N);
  if (tiles <= sm_count / 2 && M < 5 * sm_count) return false;
  if (store_logits && K < 1024 && N > 16384) return false;
  return product_plan(M, N, K, sm_count).splits == 1;
}

int logits_stat_tiles(int N) { return (N + gemm_pair::BN - 1) / gemm_pair::BN; }

cudaError_t gemm_logits_pair(const void* h, const void* w, void* logits, const long long* labels, float* row_stats,
                             float* label_logits, int M, int N, int K, long long ldh, long long ldw, long long ldl, float inv_temp,
                             int* status, int sm_count, cudaStream_t stream) {
  using namespace gemm_pair;
  if (M < 256 || N < 256 || K < BK || sm_count < 2) return cudaErrorNotSupported;
  if ((ldh % 8) || (ldw % 8) || (ldl % 8) || (N % 8) ||
      ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(logits)) & 15))
    return cudaErrorNotSupported;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeLogits>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb, tc;
  if (!encode_tile_map_2d(&ta, h, K, M, ldh * 2, 64, BMH) || !encode_tile_map_2d(&tb, w, K, N, ldw * 2, 64, BNH))
    return cudaErrorNotSupported;
  tc = ta;
  if (logits != nullptr && !encode_tile_map_2d(&tc, logits, N, M, ldl * 2, 64, kOutRows)) return cudaErrorNotSupported;
  Params p{};
  p.M = M; p.N = N; p.K = K;
  p.labels = labels;
  p.row_stats = reinterpret_cast<float2*>(row_stats); p.label_logits = label_logits;
  p.inv_temp = inv_temp;
  p.store_logits = logits != nullptr;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = logits_stat_tiles(N);
  p.status = status;
  const int tiles = p.tiles_m * p.tiles_n;
  const int pairs = tiles < sm_count / 2 ? tiles : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeLogits>, 2 * pairs, kThreads, kSmemBytes, stream, ta, tb, tc, OwnerMaps{}, p);
  return cudaGetLastError();
}

// Words for the launches of groups, zero at load and left zero by each: the counter of items, the count of finished CTAs, and two
// per divided tile.  Every stream has a set of its own, so the order of its launches keeps one from the words of another that still
// runs.  A launch that gives up may leave some as they are: from then on the streams of the device get new sets.  Who comes
// after kGroupSets of them gets none.
constexpr int kGroupSets = 1000;
__device__ unsigned int g_group_words[kGroupSets * kGroupLaunchWords];
struct GroupSets {
  std::mutex mu;
  unsigned int* base = nullptr;
  int used = 0;
  std::unordered_map<unsigned long long, int> of_stream;   // by a number that no other stream of the process ever has
};
static GroupSets* group_sets() {
  static GroupSets sets[64];
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? &sets[dev] : nullptr;
}
unsigned int* gemm_group_words(cudaStream_t stream) {
  GroupSets* sets = group_sets();
  unsigned long long id = 0;
  if (sets == nullptr) return nullptr;
  if (cudaStreamGetId(stream, &id) != cudaSuccess) {
    (void)cudaGetLastError();   // the launch that follows, with counters of its own, is not to answer for it
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(sets->mu);
  if (sets->base == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_group_words) != cudaSuccess) return nullptr;
    sets->base = static_cast<unsigned int*>(p);
  }
  auto set = sets->of_stream.find(id);
  if (set == sets->of_stream.end()) {
    if (sets->used == kGroupSets) return nullptr;
    set = sets->of_stream.emplace(id, sets->used++).first;
  }
  return sets->base + static_cast<size_t>(set->second) * kGroupLaunchWords;
}
void gemm_group_new_words() {
  if (GroupSets* sets = group_sets()) {
    std::lock_guard<std::mutex> lock(sets->mu);
    sets->of_stream.clear();
  }
}

// How wide the tiles of each product are, and into how many parts its sum is divided unless that is given (group_split).  In units of a
// k-block (0.28 us): the items go to the pairs that are free first, longest first, so the group takes the work per pair and half of
// its last item, but at least its longest item, and a second round besides costs 6 (the items are handed on from CTA to CTA, the
// first epilogues are in the way).  An item takes at least what its epilogue does (6) and 2 to begin with; a part of a bf16 tile
// writes and reads 256 KB of fp32 (6), the parts of an fp32 sum meet in memory.  The longest item is made half as wide, or
// divided, as long as that gains a twentieth.  300 tokens, 1536 wide: half as wide 15.3 -> 12.5 us (projection), MLP of 512 and 1536
// 19.5 -> 15.4.
struct GroupShape {
  int tiles, kb;
  SplitPlan plan;
  bool bf16, may_divide;        // may_divide: into other parts than the plan's
  int bn, half_tiles, layout;   // columns of a tile; how many tiles of half the width there are
  int divided() const { return tiles - plan.whole; }
  int parts() const { return divided() * plan.splits; }
  double time(int k_blocks, bool part) const {
    return std::max(6.0, k_blocks * (bn == 128 ? half_tile_time(layout) : 1.0)) + 2 + (part ? (bf16 ? 6.0 : 1.0) : 0.0);
  }
  double item() const { return plan.whole > 0 ? time(kb, false) : time(plan.kb_split, true); }   // the longest
  double sum() const { return bf16 && parts() > 0 ? 12.0 + 8.0 * (plan.splits - 1) : 0.0; }
  double work() const { return plan.whole * time(kb, false) + (parts() > 0 ? parts() * time(plan.kb_split, true) : 0.0); }
};
// Long sums are divided as in a launch of their own, so that they are no longer than there, and the bytes of a bf16 result are the
// same either way.  The tensor cores drop what does not fit behind an accumulator's last bit, 1e-9 of the result for every product in
// one sum: 8e-6 over 8192, 1.8e-5 over 17920, 1.3e-4 over 131072.  Left whole under the other products' arithmetic, as three parts
// had not been, the hidden states' gradient over 151936 words went from 8.3e-5 to 1.2e-4 (2.3526e-3 to 2.3602e-3 from 64 bits in
// all), the input gradient of a layer of 4096 and 14336 from 7.3445e-3 to 7.3461e-3; of one of 2048 and 8192, a sum over 16384, it
// stayed at 4.190e-3.  Shorter sums are divided as the group needs it: parts of a product's own are too many here (MLP of 512 and
// 1536, fp32 sums, 2000 tokens 35 us with them and 20 without; projection of 6144 x 4096, 300 tokens, 48 and 45).  Sums in one
// order and addends stay whole over any length.
constexpr int kGroupShortSum = 16384;
static SplitPlan group_split(const GemmProduct& q, int tiles, int sm_count) {
  using namespace gemm_pair;
  if (q.K > kGroupShortSum && !q.whole) {
    if (q.c_kind == kBF16 && q.addend == nullptr) return product_plan(q.M, q.N, q.K, sm_count);
    if (q.c_kind == kF32 && q.accumulate) return plan_splits(q.M, q.N, q.K, sm_count, scatter_cost(1), true);
  }
  return {tiles, 1, (q.K + BK - 1) / BK};
}
static void plan_group(GroupShape* g, int n, int pairs) {
  auto cost = [&] {
    int order[kMaxGroupProducts];
    for (int i = 0; i < n; ++i) order[i] = i;
    std::sort(order, order + n, [&](int a, int b) { return g[a].item() > g[b].item(); });
    double work = 0, span = 0;
    int all = 0;
    for (int i = 0; i < n; ++i) {
      const GroupShape& q = g[order[i]];
      const int items = q.plan.whole + q.parts();
      work += q.work();
      all += items;
      const double end = all <= pairs ? q.item() : i == 0 ? (items + pairs - 1) / pairs * (q.work() / items) : work / pairs + 0.5 * q.item();
      span = std::max(span, end + q.sum());
    }
    return span + (all > pairs ? 6.0 : 0.0);
  };
  for (double best = cost();;) {
    int longest = 0;
    for (int i = 1; i < n; ++i)
      if (g[i].item() > g[longest].item()) longest = i;
    GroupShape& q = g[longest];
    const GroupShape before = q;
    GroupShape better = before;
    double least = 0.95 * best;
    const auto consider = [&] {
      if (const double c = cost(); c < least) { least = c; better = q; }
      q = before;
    };
    if (q.bn == 256 && q.parts() == 0) {
      q.bn = 128;
      q.tiles = q.plan.whole = q.half_tiles;
      consider();
    }
    for (int want = before.plan.splits + 1; want <= 8 && q.may_divide; ++want) {
      const int each = (q.kb + want - 1) / want, s = (q.kb + each - 1) / each;   // no empty part
      if (s <= before.plan.splits || each < 4 || (q.bf16 && q.tiles > kMaxGroupDivided / kMaxGroupProducts)) continue;
      q.plan = {0, s, each};
      consider();
    }
    if (better.bn == before.bn && better.plan.splits == before.plan.splits) return;
    q = better;
    best = least;
  }
}

// What is taken together, by types and sizes.
static bool group_admits(const GemmProduct* g, int n, int sm_count) {
  using namespace gemm_pair;
  if (n < 1 || n > kMaxGroup || sm_count < 2) return false;
  // A group saves the launches and last rounds of its products, 30 to 100 units.  With more work than this for a pair that is no
  // gain any more, and pairs that are not in step with one another share less of L2 (16321 tokens, 2048 and 8192 wide, 4400 units:
  // the layer 0.5 % slower together; 5120 and 13824 wide, 32000 units: 7.62 ms one by one, 7.83 together).  fp32 results, 256 KB a
  // tile to be added to memory, run under the other products' arithmetic (head of 16384 tokens, 128256 words, 2048 wide, 7000
  // units a chunk: 20.5 ms with its forward, 20.0 together).
  long long work = 0;
  bool f32 = false;
  int rounds = 0, shortest = (g[0].K + BK - 1) / BK;
  for (int i = 0; i < n; ++i) {
    const GemmProduct& q = g[i];
    if (q.M < 1 || q.N < 256 || q.K < BK || (q.c_kind != kF32 && (q.c_kind != kBF16 || q.accumulate)) || (q.addend != nullptr && q.c_kind != kBF16)) return false;
    const int tiles = (q.M + 255) / 256 * ((q.N + BN - 1) / BN), kb = (q.K + BK - 1) / BK;
    work += static_cast<long long>(tiles) * kb;
    f32 = f32 || q.c_kind == kF32 || q.addend != nullptr;
    rounds += tiles;
    shortest = std::min(shortest, kb);
  }
  if (work > (f32 ? 12000ll : 2700ll) * (sm_count / 2)) return false;
  // Handing an item on costs 0.2 to 0.5 us that a product of its own does not pay, and in many rounds of items that is more than the
  // launches and last rounds are, the sooner the shorter the items.  Products one by one and together, us, in bf16 (k-blocks of the
  // weight gradients, rounds of items): MLP of 4096 and 14336, 256 tokens (4, 36) 164 and 167, 768 (12, 36) 333 and 325; of 5120
  // and 13824, 64 (1, 44) 161 and 171, 1000 (16, 44) 493 and 494, 2000 (32, 44) 925 and 971; of 2048 and 8192, 64 (1, 10) 57 and 53;
  // head of 128256 words, 2048 wide, 256 (4, 54) 253 and 271, 1500 (24, 54) 1070 and 1133, of 32000, 4096 wide, 400 (7, 27) 198 and
  // 202, 768 (12, 27) 296 and 288.  (All with long sums whole; with parts of their own the two that gained are level, 323 and 325, 285 and
  // 288.)  fp32 gradients gain at all of them: their additions to memory run under the other items.
  rounds /= sm_count / 2;
  return n == 1 || f32 || rounds < std::min(40, std::max(20, 7 * shortest / 2));
}

GemmGroupPlan gemm_group_plan(const GemmProduct* g, int n, int sm_count) {
  using namespace gemm_pair;
  GemmGroupPlan plan{};
  if (!group_admits(g, n, sm_count)) return plan;
  plan.taken = true;
  GroupShape shapes[kMaxGroup];
  for (int i = 0; i < n; ++i) {
    const GemmProduct& q = g[i];
    const int rows = (q.M + 255) / 256, tiles = rows * ((q.N + BN - 1) / BN);
    shapes[i] = GroupShape{tiles, (q.K + BK - 1) / BK, group_split(q, tiles, sm_count), q.c_kind == kBF16,
                           !q.whole && q.K <= kGroupShortSum && (q.c_kind == kBF16 ? q.addend == nullptr : q.accumulate), BN,
                           rows * ((q.N + BN / 2 - 1) / (BN / 2)), q.layout};
  }
  plan_group(shapes, n, sm_count / 2);
  for (int i = 0; i < n; ++i) {
    const SplitPlan& split = shapes[i].plan;
    plan.order[i] = i;
    plan.parts[i] = split.whole > 0 ? 1 : split.splits;
    plan.columns[i] = shapes[i].bn;
    plan.tiles[i] = {shapes[i].tiles, split.whole, split.splits, 0};
    plan.kb_split[i] = split.kb_split;
    if (shapes[i].bf16) plan.scratch_bytes += static_cast<size_t>(shapes[i].parts()) * 256 * BN * sizeof(float);
  }
  std::stable_sort(plan.order, plan.order + n, [&](int x, int y) { return shapes[x].item() > shapes[y].item(); });
  return plan;
}

// what the tensor maps and the epilogue ask for
static bool group_aligned(const GemmProduct* g, int n) {
  for (int i = 0; i < n; ++i) {
    const GemmProduct& q = g[i];
    if ((reinterpret_cast<uintptr_t>(q.a) | reinterpret_cast<uintptr_t>(q.b) | reinterpret_cast<uintptr_t>(q.c) |
         reinterpret_cast<uintptr_t>(q.addend)) & 15)
      return false;
    if ((q.lda % 8) || (q.ldb % 8) || (q.N % 8) || (q.layout == 2 && q.M % 8) || (q.ldc % (q.c_kind == kF32 ? 4 : 8))) return false;
  }
  return true;
}
bool gemm_group_takes(const GemmProduct* g, int n, int sm_count) { return group_admits(g, n, sm_count) && group_aligned(g, n); }

cudaError_t gemm_group(const GemmProduct* g, int n, const GemmGroupPlan& plan, float* scratch, unsigned int* words,
                       const long long* ctr_ptrs, int arrivals, int* status, int sm_count, cudaStream_t stream) {
  using namespace gemm_pair;
  if (!plan.taken || !group_aligned(g, n)) return cudaErrorNotSupported;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeGroup>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  Group group{};
  int divided = 0, parts = 0;
  for (int i = 0; i < n; ++i) {
    const GemmProduct& q = g[plan.order[i]];
    const GemmPlan& tiles = plan.tiles[plan.order[i]];
    const int bn = plan.columns[plan.order[i]];
    const bool a_mn = q.layout == 2, b_mn = q.layout != 0;
    if (!(a_mn ? encode_tile_map_2d(&group.a[i], q.a, q.M, q.K, q.lda * 2, 64, 64) : encode_tile_map_2d(&group.a[i], q.a, q.K, q.M, q.lda * 2, 64, BMH)) ||
        !(b_mn ? encode_tile_map_2d(&group.b[i], q.b, q.N, q.K, q.ldb * 2, 64, 64) : encode_tile_map_2d(&group.b[i], q.b, q.K, q.N, q.ldb * 2, 64, bn / 2)) ||
        !(q.c_kind == kF32 ? encode_tile_map_2d_f32(&group.c[i], q.c, q.N, q.M, q.ldc * 4, 32, kOutRows) : encode_tile_map_2d(&group.c[i], q.c, q.N, q.M, q.ldc * 2, 64, kOutRows)))
      return cudaErrorInvalidValue;
    GroupProblem& t = group.prob[i];
    t.M = q.M; t.N = q.N; t.K = q.K;
    t.tiles_m = (q.M + 255) / 256; t.tiles_n = (q.N + bn - 1) / bn;
    t.a_mn = a_mn; t.b_mn = b_mn; t.bn = bn;
    t.out = q.c_kind == kBF16 ? 0 : q.accumulate ? 2 : 1;
    t.scale = q.scale; t.scale_ptr = q.scale_ptr; t.addend = q.addend;
    t.first = group.items;
    t.whole = tiles.whole; t.divided = tiles.tiles - tiles.whole; t.splits = tiles.parts; t.kb_split = plan.kb_split[plan.order[i]];
    if (q.c_kind == kBF16) {
      t.first_split_tile = divided; t.first_part = parts;
      divided += t.divided; parts += t.divided * t.splits;
    }
    group.items += t.whole + t.divided * t.splits;
  }
  group.count = n;
  if (divided > kMaxGroupDivided || (divided > 0 && scratch == nullptr)) return cudaErrorNotSupported;
  group.parts = reinterpret_cast<float4*>(scratch);
  if (words == nullptr) return cudaErrorInvalidValue;
  group.next = words;
  group.arrived = words + 2;
  group.arrivals = arrivals;
  Params p{};
  p.status = status;
  p.ctr_ptrs = ctr_ptrs; p.nranks = 1; p.done_slot = words + 1;
  const int pairs = group.items < sm_count / 2 ? group.items : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeGroup>, 2 * pairs, kThreads, kSmemBytes, stream, group.a[0], group.b[0], group.c[0], group, p);
  return cudaGetLastError();
}

GemmPlan scatter_plan(int n_out, int k_in, int tokens, int nranks, int sm_count) {
  using namespace gemm_pair;
  const SplitPlan plan = plan_splits(n_out, k_in, tokens, sm_count, scatter_cost(nranks), true);
  return {(n_out + 255) / 256 * ((k_in + BN - 1) / BN), plan.whole, plan.splits, 0};
}

// dW[n_out, k_in] = dY^T X on CTA pairs; every 128 x 32 fp32 output box is added (x scale) into the accumulator of the
// rank that owns its rows by the TMA unit, through the peer mapping; then one arrival per owner.  Same contract as
// gemm_wgrad_scatter_tma; returns cudaErrorNotSupported for shapes it does not take.
cudaError_t gemm_wgrad_scatter_pair(const void* dy, const void* x, int tokens, int n_out, int k_in, long long ld_dy,
                                    long long ld_x, const long long* acc_addrs_host, const long long* ctr_ptrs,
                                    long long acc_offset, int rows_per_rank, int nranks, float scale,
                                    unsigned int* done_slot, int* status, int sm_count, cudaStream_t stream,
                                    int start_rank, bool fixed_order) {
  using namespace gemm_pair;
  if (n_out < 256 || k_in < 256 || tokens < BK || sm_count < 2) return cudaErrorNotSupported;
  if (nranks > kMaxOwners || (rows_per_rank % BMH) != 0) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x)) & 15) return cudaErrorMisalignedAddress;
  if ((ld_dy % 8) || (ld_x % 8) || (k_in % 8) || (acc_offset % 4)) return cudaErrorInvalidValue;
  if (static_cast<long long>(rows_per_rank) * nranks < n_out) return cudaErrorInvalidValue;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeScatter>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb;
  // "tn": A = dY viewed as [K = tokens rows, M = n_out cols], B = X as [K = tokens rows, N = k_in cols]
  if (!encode_tile_map_2d(&ta, dy, n_out, tokens, ld_dy * 2, 64, 64)) return cudaErrorInvalidValue;
  if (!encode_tile_map_2d(&tb, x, k_in, tokens, ld_x * 2, 64, 64)) return cudaErrorInvalidValue;
  OwnerMaps owners{};
  for (int r = 0; r < nranks; ++r) {
    float* base = reinterpret_cast<float*>(static_cast<uintptr_t>(acc_addrs_host[r])) + acc_offset;
    if (!encode_tile_map_2d_f32(&owners.m[r], base, k_in, rows_per_rank, static_cast<uint64_t>(k_in) * 4, 32, kOutRows))
      return cudaErrorInvalidValue;
  }
  Params p{};
  p.M = n_out; p.N = k_in; p.K = tokens;
  p.c_is_f32 = 1;
  p.a_mn = 1; p.b_mn = 1;
  p.tiles_m = (n_out + 255) / 256;
  p.tiles_n = (k_in + BN - 1) / BN;
  p.status = status;
  p.ctr_ptrs = ctr_ptrs;
  p.rows_per_rank = rows_per_rank; p.nranks = nranks; p.scale = scale; p.done_slot = done_slot;
  if (rotate_mode() >= 1)
    p.rot_m = static_cast<int>((static_cast<long long>(start_rank) * rows_per_rank / 256) % p.tiles_m);
  SplitPlan plan{p.tiles_m * p.tiles_n, 1, 0};
  if (!fixed_order) plan = plan_splits(n_out, k_in, tokens, sm_count, scatter_cost(nranks), true);
  p.whole = plan.whole; p.splits = plan.splits; p.kb_split = plan.kb_split;
  const int items = p.whole + (p.tiles_m * p.tiles_n - p.whole) * p.splits;
  const int pairs = items < sm_count / 2 ? items : sm_count / 2;
  launch(gemm_bf16_pair_kernel<kModeScatter>, 2 * pairs, kThreads, kSmemBytes, stream, ta, tb, ta, owners, p);
  return cudaGetLastError();
}

// Y[M, N] = X[M, K] W[N, K]^T (dgrad = false) or dX[M, K_in] = dY[M, N_out] W[N_out, K_in] (dgrad = true) on CTA pairs,
// with W row-sharded over nranks owners and pulled into w_local by four extra warps per CTA while the GEMM runs.
// Same contracts as gemm_gather_nt / gemm_gather_nn; cudaErrorNotSupported for shapes it does not take.
cudaError_t gemm_gather_pair(bool dgrad, const void* a, const long long* shard_ptrs, void* w_local, void* out,
                             const void* bias, int M, int w_rows, int w_cols, long long lda, long long ldo,
                             int rows_per_rank, int nranks, unsigned int* group_flags, int* status, int sm_count,
                             cudaStream_t stream, const void* residual, long long ldr, int start_rank) {
  using namespace gemm_pair;
  const int N = dgrad ? w_cols : w_rows;   // output columns
  const int K = dgrad ? w_rows : w_cols;   // reduction length
  if (M < 256 || N < 256 || K < BK || sm_count < 2) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w_local) | reinterpret_cast<uintptr_t>(out)) & 15)
    return cudaErrorMisalignedAddress;
  if ((lda % 8) || (ldo % 8) || (N % 8) || (w_cols % 128)) return cudaErrorInvalidValue;
  if (static_cast<long long>(rows_per_rank) * nranks < w_rows) return cudaErrorInvalidValue;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_pair_kernel<kModeGather>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemBytes);
  });
  if (attr_err != cudaSuccess) return attr_err;
  CUtensorMap ta, tb, tc;
  if (!encode_tile_map_2d(&ta, a, K, M, lda * 2, 64, BMH)) return cudaErrorInvalidValue;
  if (!dgrad) {
    if (!encode_tile_map_2d(&tb, w_local, w_cols, w_rows, static_cast<uint64_t>(w_cols) * 2, 64, BNH)) return cudaErrorInvalidValue;
  } else {  // B is MN-major: rows = reduction index, box {64 output columns, 64 reduction rows}
    if (!encode_tile_map_2d(&tb, w_local, w_cols, w_rows, static_cast<uint64_t>(w_cols) * 2, 64, 64)) return cudaErrorInvalidValue;
  }
  if (!encode_tile_map_2d(&tc, out, N, M, ldo * 2, 64, kOutRows)) return cudaErrorInvalidValue;
  Params p{};
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.M = M; p.N = N; p.K = K;
  p.b_mn = dgrad ? 1 : 0;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (N + BN - 1) / BN;
  p.status = status;
  p.shard_ptrs = shard_ptrs;
  p.b_local = static_cast<unsigned char*>(w_local);
  p.panel_flags = group_flags;
  p.rows_per_rank = rows_per_rank; p.nranks = nranks;
  p.w_rows = w_rows; p.w_cols = w_cols;
  if (rotate_mode() >= (dgrad ? 2 : 1)) {
    const int groups = (w_rows + BN - 1) / BN;
    const int rot_group = static_cast<int>((static_cast<long long>(start_rank) * rows_per_rank / BN) % groups);
    if (!dgrad) p.rot_n = rot_group % p.tiles_n;
    else p.rot_kb = (rot_group * (BN / BK)) % ((K + BK - 1) / BK);
    p.fetch_rot = static_cast<long long>(rot_group) * (static_cast<long long>(BN) * w_cols * 2 / kFetchChunkBytes);
  }
  if (residual != nullptr) {
    if ((ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15)) return cudaErrorInvalidValue;
    p.residual = static_cast<const __nv_bfloat16*>(residual);
    p.ldr = ldr;
  }
  cudaError_t e = cudaMemsetAsync(group_flags, 0, sizeof(unsigned int) * ((w_rows + BN - 1) / BN), stream);
  if (e != cudaSuccess) return e;
  const int grid = sm_count & ~1;  // every CTA also fetches, so the whole machine runs even when there are few tiles
  gemm_bf16_pair_kernel<kModeGather><<<grid, Roles<kModeGather>::kThreadsTotal, kSmemBytes, stream>>>(ta, tb, tc, OwnerMaps{}, p);
  return cudaGetLastError();
}

}  // namespace odc
