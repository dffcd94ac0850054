// Causal attention over packed variable-length sequences on tcgen05 tensor cores (sm_100a).
//
// Forward: one or two tiles of 128 query rows of one sequence per CTA.
//   warp 0     TMA producer: Q tiles once, then K and V tiles of 128 keys through two small rings
//   warp 1     MMA issuer:   S = Q K^T into TMEM, then O += P V
//   warps 2-   softmax:      eight warps per tile, two threads per query row, 64 keys each; S from TMEM, online softmax in
//                            base 2 with lazy rescaling of O (only when a row maximum grows by more than 2^8),
//                            P written back to TMEM as the bf16 A operand of P V
// The TMA and MMA warps elect their thread with elect.sync: of a thread picked by its lane number the compiler does not
// know that it is alone, and moves the operands of every tcgen05 and TMA instruction to uniform registers by way of a loop.
// Eight MMAs of 64 clocks each then took 690 clocks to issue and the tensor cores waited for them; elected, 410.
// K and V tiles share one TMA box shape: K is read as
// a K-major operand (Q K^T) and V as an N-major operand (P V), so nothing is transposed in memory.
// Rows/keys outside the sequence are masked; grouped-query attention maps query head h to
// key/value head h / (Hq/Hkv).
//
// Backward: a pre-pass computes delta = rowsum(dO * O); the main kernel owns one (128 keys, kv
// head) tile, keeps dK and dV in TMEM across all query tiles and query heads of the group, and
// recomputes P from the saved log-sum-exp.  dQ tiles are staged in shared memory as fp32 and added into a
// global fp32 buffer by the TMA unit (bulk reduce-add), then scaled and converted to bf16 by a post-pass.
//
// The reference calls flash-attn 2 for this op (examples/llm_training/torch_fsdp2.py:85-103).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "api.h"
#include "launch.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace odc {

using namespace sm100;

namespace {

constexpr int kBlockQ = 128, kBlockKV = 128;
constexpr uint64_t kWaitBudgetNs = 4000000000ull;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// byte offset of element (row, col) inside a [128 rows][128 cols] bf16 operand stored as two
// 128-byte-swizzled slabs of 64 columns (the layout TMA produces and the K-major descriptor reads)
__device__ __forceinline__ uint32_t swz_chunk_offset(int row, int chunk16 /*0..15*/) {
  const int slab = chunk16 >> 3, ch = chunk16 & 7;
  return slab * 16384 + row * 128 + ((ch ^ (row & 7)) << 4);
}

struct FwdParams {
  const int* cu_seqlens;
  int num_seqs;
  int n_q, n_kv;
  int heads_per_cta;
  __nv_bfloat16* o;
  long long o_stride;
  float* lse;  // [n_q, total_tokens]
  int total_tokens;
  float scale_log2;
  int causal;
  int* status;
};

// The idx-th tile of the pack, longest work first; false if there are fewer.  A tile's work w is the number of tiles it meets
// under the causal mask, 1 .. n for the n tiles of a sequence (query tiles from the front, key tiles from the back), so
// sum over sequences of max(0, n - w + 1) tiles have at least w.  Tiles of a long sequence then start before those of
// short ones wherever it lies in the pack: started in pack order, the last long tiles ran alone (T = 8192 in one
// sequence, 16/4 heads: SMs idle for 23 % of the forward and 36 % of the backward; 16210 tokens in 12 sequences up to 8192, 32/8 heads, D = 64:
// forward 0.600 ms, now 0.479, backward 1.388 ms, now 1.196).  Called by whole warps.
__device__ __forceinline__ bool locate_tile(const int* cu, int num_seqs, int idx, int tile_rows, int* start, int* len, int* work) {
  const int lane = threadIdx.x & 31;
  auto tiles = [&](int s) { return s < num_seqs ? (cu[s + 1] - cu[s] + tile_rows - 1) / tile_rows : 0; };
  const int own = tiles(lane);
  auto at_least = [&](int w) {
    int c = max(0, own - w + 1);
    for (int s = lane + 32; s < num_seqs; s += 32) c += max(0, tiles(s) - w + 1);
    return __reduce_add_sync(0xffffffffu, c);
  };
  int longest = own;
  for (int s = lane + 32; s < num_seqs; s += 32) longest = max(longest, tiles(s));
  int lo = 1, hi = __reduce_max_sync(0xffffffffu, longest);
  if (hi < 1 || idx >= at_least(1)) return false;
  while (lo < hi) {  // the largest w that more than idx tiles reach
    const int mid = (lo + hi + 1) / 2;
    if (at_least(mid) > idx) lo = mid; else hi = mid - 1;
  }
  int rank = idx - at_least(lo + 1);
  for (int first = 0; first < num_seqs; first += 32) {  // the rank-th sequence with at least lo tiles
    const bool has = (first == 0 ? own : tiles(first + lane)) >= lo;
    const unsigned int m = __ballot_sync(0xffffffffu, has);
    if (rank < __popc(m)) {
      const bool mine = has && __popc(m & ((1u << lane) - 1u)) == rank;
      const int s = first + __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
      *start = cu[s];
      *len = cu[s + 1] - cu[s];
      *work = lo;
      return true;
    }
    rank -= __popc(m);
  }
  return false;  // not reached while cu_seqlens stays as it is
}

// Two 128-row query tiles per SM keep the exponential units and the tensor cores busy at the same time: while the softmax
// warps of one tile work, the products of the other run.  P goes back to tensor memory as the A operand of O += P V, so
// it costs no shared memory and no shared-memory bandwidth.
//   D = 64:  one tile per CTA in 256 TMEM columns, two CTAs per SM (tiles of short sequences see only 1-3 key blocks: the
//            start of one CTA hides under the other).  P has its own columns, so S(j+1) is issued as soon as S(j) has
//            been read and runs under the exponentials of block j.
//   D = 128: two tiles in one CTA that read the same K and V tiles: two heads of a key/value group, or with an odd number
//            of heads per group two consecutive tiles of one head.  All 512 TMEM columns are taken: P(j) overwrites the
//            scores it came from, and S(j+1) follows P V(j) in the tensor cores' issue order.  Where pairs would leave SMs
//            without work (attn_fwd_pairs) a CTA takes one tile, with P in columns of its own as at D = 64.
// Bound by the chain around the exponentials (scores out of TMEM, maximum, exponentials, P into TMEM): with none of them
// computed at all a pass is only 12 (D = 128) to 18 % (D = 64) faster.  Two threads per row halve that chain, a few of the
// exponentials go to the FMA pipe, and the first half of P V starts before the other half of P is there.  Against one thread
// per row and MMAs issued by lane 0: 32768 tokens, 40/8 heads, D = 128 9.65 ms, now 8.92 (1233 TFLOP/s), under the power cap
// 10.77 and 10.05 (1094); 16 sequences of 1024 357 us, now 327; 40 of 300 297 and 299.  32/8 heads, D = 64: 16 sequences of
// 1024 180 us, now 164; 40 of 300 125 and 112; one of 32768 5.53 ms and 5.56, under the power cap 5.83 and 5.94.
template <int D, int Tiles>
struct FwdCfg {
  static constexpr int kTiles = Tiles;
  static constexpr int kCtasPerSm = (D == 64) ? 2 : 1;
  static constexpr int kStages = (D == 128 && Tiles == 1) ? 3 : 2;  // of K and of V, each with barriers of its own
  static constexpr bool kPrivateP = (Tiles == 1);
  static constexpr int kTmemCols = (D == 64) ? 256 : 512;
  static constexpr int kOCol = kTiles * 128;
  // P of the first / the other 64 keys of tile t
  __host__ __device__ static constexpr int p_col(int t, int half) {
    return kPrivateP ? 128 + D + 32 * half : 128 * t + 64 * half;
  }
  // Of 16 pairs of exponentials, how many the FMA pipe takes instead of the special-function unit (13 instructions a pair).
  // 32768 tokens, 40/8 heads, D = 128: none 8974 us, one 9069, two 8916 (under the power cap 10076, 10184, 10047); 4096 tokens,
  // 12/2 heads: none 72, two 69, four 70, six 74.  32/8 heads, D = 64, 32768 tokens: none 5756 us, one 5559, two 5646, three
  // 5639 (under the power cap 6035, 5942, 6042, 6086); 16 sequences of 1024: 167, 164, 165, 166.
  static constexpr int kPolyPairs = (D == 64) ? 1 : 2;
  static constexpr int kThreads = 64 + 256 * kTiles;
  static constexpr int kQBytes = kBlockQ * D * 2;
  static constexpr int kKBytes = kBlockKV * D * 2;
  static constexpr int kStageBytes = 2 * kKBytes;
  static constexpr int kBarBytes = 256;
  // the alignment slack is trimmed so that two CTAs fit in one SM's 228 KiB (the dynamic window starts 1024-byte aligned
  // in practice; the kernel checks and reports otherwise)
  static constexpr int kAlignSlack = 768;
  static constexpr int kExchangeBytes = kTiles * 2 * 2 * 128 * 4;  // row maxima, [tile][step & 1][half][row]
  static constexpr int kSmem = kTiles * kQBytes + kStages * kStageBytes + kBarBytes + kExchangeBytes + kAlignSlack;
};

// a * b + c on two fp32 values in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// 2^x for x <= 127 on the FMA pipe: x = n + f with |f| <= 1/2, a polynomial in f (degree 5, the minimax fit of the relative
// error with a constant term of one: 1.7e-7 in fp32, the special-function unit's is 2.4e-7) times 2^n.  Adding 1.5 * 2^23
// rounds x to n and leaves n + 127 in the low bits, which shifted are 2^n; n = -127 gives zero, as the unit's flush does,
// and NaN stays NaN.
__device__ __forceinline__ float2 exp2_poly(float2 x) {
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x.x));  // -127
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x.y));
  constexpr float kRound = 12582912.f + 127.f;
  const float2 t = add2(x, make_float2(kRound, kRound));
  const float2 f = fma2(add2(t, make_float2(-kRound, -kRound)), make_float2(-1.f, -1.f), x);
  float2 p = make_float2(0.0013264593435451388f, 0.0013264593435451388f);
  p = fma2(p, f, make_float2(0.0096714673563838f, 0.0096714673563838f));
  p = fma2(p, f, make_float2(0.05550733581185341f, 0.05550733581185341f));
  p = fma2(p, f, make_float2(0.24022242426872253f, 0.24022242426872253f));
  p = fma2(p, f, make_float2(0.6931470036506653f, 0.6931470036506653f));
  p = fma2(p, f, make_float2(1.f, 1.f));
  return mul2(p, make_float2(__uint_as_float(__float_as_uint(t.x) << 23), __uint_as_float(__float_as_uint(t.y) << 23)));
}

// exp2_poly on its own, for tests of its error
__global__ void __launch_bounds__(256) exp2_poly_kernel(const float2* x, float2* y, long long n2) {
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i < n2) y[i] = exp2_poly(x[i]);
}

template <int D, int Tiles>
__global__ void __launch_bounds__(FwdCfg<D, Tiles>::kThreads, FwdCfg<D, Tiles>::kCtasPerSm)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const FwdParams p) {
  using C = FwdCfg<D, Tiles>;
  // the tiles of one CTA: heads_per_cta heads, or consecutive query tiles of one head
  const int rows = p.heads_per_cta == C::kTiles ? kBlockQ : kBlockQ * C::kTiles;
  // heads vary fastest: the longest tiles of all heads start first
  const int head_groups = p.n_q / p.heads_per_cta;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  if (base - raw > static_cast<uint32_t>(C::kAlignSlack)) {  // cannot happen with a 1024-aligned window
    if (threadIdx.x == 0) report(p.status, kErrBounds, 42, static_cast<int>(base - raw));
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kTiles * C::kQBytes + C::kStages * C::kStageBytes);
  const uint32_t q_smem = base;
  const uint32_t kv_smem = q_smem + C::kTiles * C::kQBytes;
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t q_full = bar0;
  const uint32_t k_full0 = bar0 + 8;                       // [kStages]
  const uint32_t k_empty0 = k_full0 + 8 * C::kStages;      // [kStages]
  const uint32_t v_full0 = k_empty0 + 8 * C::kStages;      // [kStages]
  const uint32_t v_empty0 = v_full0 + 8 * C::kStages;      // [kStages]
  const uint32_t s_full0 = v_empty0 + 8 * C::kStages;      // [2] per tile: scores complete
  const uint32_t s_empty0 = s_full0 + 16;                  // [2] scores have been read
  const uint32_t p_full0 = s_empty0 + 16;                  // [2][2] P of the first / the other 64 keys is in tensor memory
  const uint32_t o_ready0 = p_full0 + 32;                  // [2] P V complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * C::kStages + 12);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitCtx wc{abort_flag, p.status, kWaitBudgetNs};

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(k_full0 + 8 * s, 1);
      mbar_init(k_empty0 + 8 * s, 1);
      mbar_init(v_full0 + 8 * s, 1);
      mbar_init(v_empty0 + 8 * s, 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(s_full0 + 8 * t, 1);
      mbar_init(s_empty0 + 8 * t, 8);
      mbar_init(p_full0 + 16 * t, 4);
      mbar_init(p_full0 + 16 * t + 8, 4);
      mbar_init(o_ready0 + 8 * t, 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  // One warp finds the tile, while the others set up: the walks of ten or eighteen warps over the lengths took 8-20 % of the
  // time of short sequences.  300 sequences of 20 tokens, 32/8 heads: D = 64 268 us, now 214; D = 128 352, now 307; 100 of
  // 100 tokens: 102, now 84, and 139, now 131.
  int* found = reinterpret_cast<int*>(bars + C::kBarBytes / 8) - 4;
  if (warp == 2) {
    int start = 0, len = 0, w = 0;
    if (!locate_tile(p.cu_seqlens, p.num_seqs, blockIdx.x / head_groups, rows, &start, &len, &w)) w = 0;
    if (lane == 0) found[0] = start, found[1] = len, found[2] = w;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int seq_start = found[0], seq_len = found[1], work = found[2];
  if (work == 0) {
    if (warp == 1) tmem_dealloc(tmem_base, C::kTmemCols);
    return;
  }
  const int q_first = (work - 1) * rows;
  const int head0 = (blockIdx.x % head_groups) * p.heads_per_cta;
  const int kv_head = head0 / (p.n_q / p.n_kv);
  auto tile_head = [&](int t) { return p.heads_per_cta == C::kTiles ? head0 + t : head0; };
  auto tile_q0 = [&](int t) { return p.heads_per_cta == C::kTiles ? q_first : q_first + t * kBlockQ; };
  auto tile_blocks = [&](int t) {  // key blocks that tile t sees; 0 if it lies past the end of the sequence
    const int q0 = tile_q0(t);
    if (q0 >= seq_len) return 0;
    return ((p.causal ? min(seq_len, q0 + kBlockQ) : seq_len) + kBlockKV - 1) / kBlockKV;
  };
  const int n_blocks = max(tile_blocks(0), tile_blocks(C::kTiles - 1));

  if (warp == 0) {
    if (elect_one()) {
      prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
      mbar_arrive_expect_tx(q_full, C::kTiles * C::kQBytes);
#pragma unroll
      for (int t = 0; t < C::kTiles; ++t)
#pragma unroll
        for (int s = 0; s < D / 64; ++s)  // a tile past the end of the sequence reads rows that nobody uses
          tma_load_2d(q_smem + t * C::kQBytes + s * 16384, &tmap_q, q_full, tile_head(t) * D + 64 * s, seq_start + tile_q0(t));
      bool ok = true;
      for (int j = 0; j < n_blocks && ok; ++j) {
        const int st = j % C::kStages;
        const uint32_t ph = (j / C::kStages) & 1;
        const uint32_t k_dst = kv_smem + st * C::kStageBytes, v_dst = k_dst + C::kKBytes;
        const int row = seq_start + j * kBlockKV;
        if (!(ok = mbar_wait(k_empty0 + 8 * st, ph ^ 1, wc, 11))) break;
        mbar_arrive_expect_tx(k_full0 + 8 * st, C::kKBytes);
#pragma unroll
        for (int s = 0; s < D / 64; ++s) tma_load_2d(k_dst + s * 16384, &tmap_k, k_full0 + 8 * st, kv_head * D + 64 * s, row);
        if (!(ok = mbar_wait(v_empty0 + 8 * st, ph ^ 1, wc, 10))) break;
        mbar_arrive_expect_tx(v_full0 + 8 * st, C::kKBytes);
#pragma unroll
        for (int s = 0; s < D / 64; ++s) tma_load_2d(v_dst + s * 16384, &tmap_v, v_full0 + 8 * st, kv_head * D + 64 * s, row);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(kBlockQ, kBlockKV, false, false);
      const uint32_t idesc_o = make_idesc_bf16(kBlockQ, D, false, true);
      bool ok = mbar_wait(q_full, 0, wc, 12);
      auto issue_s = [&](int t, int j) -> bool {
        const int st = j % C::kStages;
        if (!mbar_wait(k_full0 + 8 * st, (j / C::kStages) & 1, wc, 13)) return false;
        tc_fence_after();
        const uint64_t qd = make_smem_desc(q_smem + t * C::kQBytes, 16, 1024);
        const uint64_t kd = make_smem_desc(kv_smem + st * C::kStageBytes, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = ((k >> 2) * 16384 + (k & 3) * 32) >> 4;
          umma_f16(tmem_base + t * 128, qd + off, kd + off, idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full0 + 8 * t);
        return true;
      };
      int nb[C::kTiles];
#pragma unroll
      for (int t = 0; t < C::kTiles; ++t) {
        nb[t] = tile_blocks(t);
        if (ok && nb[t] > 0) ok = issue_s(t, 0);
      }
      if (ok) umma_commit(k_empty0);
      for (int j = 0; j < n_blocks && ok; ++j) {
        const int st = j % C::kStages;
        const uint64_t vd = make_smem_desc(kv_smem + st * C::kStageBytes + C::kKBytes, 16384, 1024);
#pragma unroll
        for (int t = 0; t < C::kTiles; ++t) {
          if (ok && C::kPrivateP && j + 1 < nb[t]) {
            ok = mbar_wait(s_empty0 + 8 * t, j & 1, wc, 15);
            if (ok) ok = issue_s(t, j + 1);
          }
          if (ok && j < nb[t]) {
            ok = mbar_wait(v_full0 + 8 * st, (j / C::kStages) & 1, wc, 14);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
              if (!(ok = ok && mbar_wait(p_full0 + 16 * t + 8 * part, j & 1, wc, 16))) break;
              tc_fence_after();
#pragma unroll
              for (int k = 4 * part; k < 4 * part + 4; ++k)
                umma_f16_ts(tmem_base + C::kOCol + t * D, tmem_base + C::p_col(t, part) + (k & 3) * 8,
                            vd + ((k * 2048) >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
            }
            if (ok) umma_commit(o_ready0 + 8 * t);
          }
          if (t == C::kTiles - 1) umma_commit(v_empty0 + 8 * st);
          if (ok && !C::kPrivateP && j + 1 < nb[t]) ok = issue_s(t, j + 1);
        }
        if (ok && j + 1 < n_blocks) umma_commit(k_empty0 + 8 * ((j + 1) % C::kStages));
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax / epilogue
    const int quad = warp & 3;
    const int t = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1;
    const int row = quad * 32 + lane;            // query row within the tile
    const int head = tile_head(t), q0 = tile_q0(t), nb = tile_blocks(t);
    const int q_rel = q0 + row;                  // position inside the sequence
    const bool row_valid = q_rel < seq_len;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t t_s = lanes + t * 128 + 64 * half, t_p = lanes + C::p_col(t, half);
    const uint32_t t_o = lanes + C::kOCol + t * D + half * (D / 2);
    const int pair_bar = 1 + t * 4 + quad;       // the two warps that share the quad's rows
    float* xch = reinterpret_cast<float*>(smem + C::kTiles * C::kQBytes + C::kStages * C::kStageBytes + C::kBarBytes) + t * 512;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nb; ++j) {               // a warp that gives up keeps walking the pair's barriers
      ok = ok && mbar_wait(s_full0 + 8 * t, j & 1, wc, 17);
      tc_fence_after();
      const int kv0 = j * kBlockKV + 64 * half;
      const bool need_mask = (kv0 + 64 > seq_len) || (p.causal && kv0 + 64 > q0);
      uint32_t sr[64];
      tmem_ld_32x32(t_s, sr);
      tmem_ld_32x32(t_s + 32, sr + 32);
      tmem_ld_wait();
      if (C::kPrivateP) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty0 + 8 * t);
      }
      if (need_mask) {
        // keys [kv0, kv_hi) are visible to this row; everything from kv_hi on is masked
        const int kv_hi = min(seq_len, p.causal ? q_rel + 1 : seq_len) - kv0;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i >= kv_hi) sr[i] = 0xff800000u;  // -inf
      }
      // independent chains: a single running value would put 64 dependent operations on the critical path
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 2)
        mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(sr[i]), __uint_as_float(sr[i + 1]));
      float mx = max3(fmaxf(mx4[0], mx4[1]), mx4[2], mx4[3]);
      xch[(j & 1) * 256 + half * 128 + row] = mx;
      named_barrier_sync(pair_bar, 64);
      mx = fmaxf(mx, xch[(j & 1) * 256 + (half ^ 1) * 128 + row]);
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      // lazy rescale of the running output (exact: P and l keep using m_used until it is bumped)
      const bool bump = (m_new - m_used > kRescaleThreshold) || (m_used == -INFINITY && m_new > -INFINITY);
      if (j == 0) {
        m_used = m_new;
      } else if (__any_sync(0xffffffffu, bump)) {
        ok = ok && mbar_wait(o_ready0 + 8 * t, (j - 1) & 1, wc, 19);  // P V(j-1) is complete: O may be rescaled
        tc_fence_after();
        const float alpha = (m_new == -INFINITY) ? 1.f : exp2f(m_used - m_new);
#pragma unroll 1
        for (int c = 0; c < D / 2; c += 16) {
          uint32_t r[16];
          tmem_ld_32x16(t_o + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st_32x16(t_o + c, r);
        }
        l *= alpha;
        m_used = m_new;
        // P of the first 64 keys alone starts a product into all columns of O, so the half 0 warp may say that it is there
        // only when the half 1 warp has scaled its columns too.  Both hold the same rows and maxima: both come here.
        tmem_st_wait();
        tc_fence_before();
        named_barrier_sync(pair_bar, 64);
        tc_fence_after();
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), sub2 = make_float2(-m_sub, -m_sub);
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int e = 32 * v + 2 * i;
          float2 f = fma2(make_float2(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), scale2, sub2);
          if ((i + 1) * C::kPolyPairs / 16 > i * C::kPolyPairs / 16) {
            f = exp2_poly(f);
          } else {
            f.x = exp2f(f.x);
            f.y = exp2f(f.y);
          }
          sum2[i & 1] = add2(sum2[i & 1], f);
          pk[i] = pack2(f.x, f.y);
        }
        // P V(j-1) is complete: P may be overwritten (without columns of its own P lies in the scores, which come after it)
        if (v == 0 && C::kPrivateP && j > 0) ok = ok && mbar_wait(o_ready0 + 8 * t, (j - 1) & 1, wc, 18);
        tmem_st_32x16(t_p + 16 * v, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full0 + 16 * t + 8 * half);
      l += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
    }
    // epilogue: O / l -> bf16, log-sum-exp; the slot that the last step did not use takes the row sums
    if (nb > 0) {
      xch[(nb & 1) * 256 + half * 128 + row] = l;
      named_barrier_sync(pair_bar, 64);
      l += xch[(nb & 1) * 256 + (half ^ 1) * 128 + row];
      ok = ok && mbar_wait(o_ready0 + 8 * t, (nb - 1) & 1, wc, 20);
    }
    if (ok && nb > 0) {
      tc_fence_after();
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      __nv_bfloat16* orow = p.o + static_cast<long long>(seq_start + q_rel) * p.o_stride + head * D + half * (D / 2);
#pragma unroll 1
      for (int c = 0; c < D / 64; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(t_o + c * 32, r);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 o;
            o.x = pack2(__uint_as_float(r[8 * v]) * inv, __uint_as_float(r[8 * v + 1]) * inv);
            o.y = pack2(__uint_as_float(r[8 * v + 2]) * inv, __uint_as_float(r[8 * v + 3]) * inv);
            o.z = pack2(__uint_as_float(r[8 * v + 4]) * inv, __uint_as_float(r[8 * v + 5]) * inv);
            o.w = pack2(__uint_as_float(r[8 * v + 6]) * inv, __uint_as_float(r[8 * v + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + v * 8) = o;
          }
        }
      }
      if (row_valid && half == 0)
        p.lse[static_cast<long long>(head) * p.total_tokens + seq_start + q_rel] =
            (l > 0.f) ? (m_used + log2f(l)) * kLn2 : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}


// =================================================================================== backward
struct BwdParams {
  const int* cu_seqlens;
  int num_seqs;
  int n_q, n_kv;
  const float* lse;    // [n_q, total_tokens]
  const float* delta;  // [n_q, total_tokens]
  float* dq_acc;       // [total_tokens, n_q, D] fp32, zero-initialised
  __nv_bfloat16* dk;   // rows of n_kv * D values, dkv_stride elements apart
  __nv_bfloat16* dv;
  long long dkv_stride;
  int parts;           // CTAs that share the query heads of one (key tile, kv head); each takes n_q / n_kv / parts of them
  float* kv_parts;     // parts > 1: [parts][dK, dV][total_tokens, n_kv, D] fp32, summed by the post-pass
  int total_tokens;
  float scale, scale_log2;
  float lse_scale;     // log-sum-exp -> what to add to a score
  int causal;
  int* status;
};

// One CTA owns (128 keys, kv head) and walks the query tiles of all heads of the group.  Scores are formed transposed
// (S^T = K Q^T, keys in the TMEM lanes), so P^T is written back to tensor memory as the A operand of dV += P^T dO and
// dS^T goes to shared memory once, where dK reads it K-major and dQ reads the same bytes MN-major.
//   warp 0       TMA producer of Q / dO, and the log-sum-exp and delta of the tile's queries into shared memory
//   warp 1       MMA issuer
//   warps 2-9    P and dS: two warpgroups, each takes 64 of the 128 query columns
//   warps 10-13  dQ tile from tensor memory -> fp32 staging -> TMA reduce-add
// Every product of one tile runs under another step of the pipeline: S(i+1) is issued as soon as P(i) exists, dK(i) runs
// while dQ(i) is read out, the exponentials of tile i+1 run under dQ(i), dK(i) and dP(i+1).  With one chain per tile
// (scores -> P, dS -> dK, dV, dQ -> read-out) the tensor cores sat idle through every element-wise step: 32768 tokens,
// 40 query and 8 key/value heads, D = 128: forward + backward 54.3 ms then, 42.4 ms with this pipeline.
// Bound: shared memory.  At D = 128 the four products with both operands there read 256 KiB per tile at 128 B/clk, which
// is also the tensor cores' time for them; staging and loads add 256 KiB.  At D = 64 there is room to take traffic out:
//   - Every thread needs the log-sum-exp and delta of all its queries: 581 of 3550 clocks per tile went to reading them.  They
//     are 16-byte rows of an operand instead, each value in three bf16 terms (its 24 bits), and one more K step of S and dP with
//     a selector of ones adds them to the whole tile.  Each has rows of its own: beside a selector of zeros in one row, a NaN or
//     infinite delta would reach the scores as well.
//   - dS^T is also written over dP^T in tensor memory, where dK reads it; from shared memory only dQ does.
// 16321 tokens, lengths up to 8192, 32/8 heads: 1.27 ms, with the rows 1.23, with both 1.16; 8192 tokens in one sequence:
// 0.95, 0.91, 0.83 ms.
template <int D>
struct BwdCfg {
  static constexpr int kQStages = 2;                       // Q(i+1) feeds S(i+1) while dK(i) still reads Q(i)
  static constexpr int kDoStages = (D == 64) ? 2 : 1;      // shared memory is full at D = 128
  static constexpr int kTile = 128 * D * 2;                // one [128][D] bf16 operand
  static constexpr int kDsBytes = 128 * 128 * 2;
  static constexpr int kStageBytes = 2 * 16384;            // two [128][32] fp32 boxes of the dQ reduction
  // Log-sum-exp and delta of the tile's queries.  D = 64: as rows of an operand (below), with the row selector;
  // D = 128: two stages of plain values that every thread reads (as rows they would have to wait for dP of the tile before,
  // which is late there: 32768 tokens, 40/8 heads 27.4 ms, with rows 27.9)
  static constexpr bool kRows = (D == 64);
  static constexpr int kStatBytes = kRows ? 2 * 2048 + 256 : kQStages * 2 * 128 * 4;
  static constexpr int kBarBytes = 256;
  // the dynamic window starts 1024-byte aligned in practice; the kernel checks and reports otherwise
  static constexpr int kAlignSlack = 768;
  static constexpr int kSmem =
      (2 + kQStages + kDoStages) * kTile + kDsBytes + kStageBytes + kStatBytes + kBarBytes + kAlignSlack;
  // tensor memory columns.  D = 64 has room for P and dQ of their own; D = 128 fills all 512: P takes over the score
  // columns it came from and dQ the columns of the consumed dP
  static constexpr int kS = 0, kDp = 128, kDv = 256, kDk = 256 + D;
  static constexpr bool kPrivate = (D == 64);
  static constexpr int kDq = kPrivate ? 384 : kDp;
  __host__ __device__ static constexpr int p_col(int half) { return kPrivate ? 448 + 32 * half : kS + 64 * half; }
};
static_assert(BwdCfg<128>::kSmem <= 232448, "shared memory of one CTA");

constexpr int kBwdThreads = 32 * (2 + 8 + 4);

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const __grid_constant__ CUtensorMap tmap_dq, const BwdParams p) {
  using C = BwdCfg<D>;
  int seq_start, seq_len, work;
  if (!locate_tile(p.cu_seqlens, p.num_seqs, blockIdx.x / (p.n_kv * p.parts), 128, &seq_start, &seq_len, &work)) return;
  const int kv_head = blockIdx.x / p.parts % p.n_kv, part = blockIdx.x % p.parts;
  const int rep = p.n_q / p.n_kv / p.parts;                     // query heads of this CTA
  const int first_head = (kv_head * p.parts + part) * rep;
  const int n_qblocks = (seq_len + 127) / 128;
  const int kv0 = (n_qblocks - work) * 128;
  const int i_first = p.causal ? kv0 / 128 : 0;
  const int iters_per_head = n_qblocks - i_first;
  const int total_iters = iters_per_head * rep;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  if (base - raw > static_cast<uint32_t>(C::kAlignSlack)) {  // cannot happen with a 1024-aligned window
    if (threadIdx.x == 0) report(p.status, kErrBounds, 41, static_cast<int>(base - raw));
    return;
  }
  constexpr int kQOff = 2 * C::kTile, kDoOff = kQOff + C::kQStages * C::kTile, kDsOff = kDoOff + C::kDoStages * C::kTile;
  constexpr int kStageOff = kDsOff + C::kDsBytes, kStatOff = kStageOff + C::kStageBytes, kBarOff = kStatOff + C::kStatBytes;
  const uint32_t k_smem = base, v_smem = base + C::kTile, ds_smem = base + kDsOff;
  uint4* rows_smem = reinterpret_cast<uint4*>(smem + kStatOff);  // kRows: [lse, delta][128] queries, the selector, [2][8]
  float* stats = reinterpret_cast<float*>(smem + kStatOff);      // else [stage][-log2(e) * lse, delta][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBarOff);
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t kv_full = bar0;
  const uint32_t q_full0 = bar0 + 8, q_empty0 = bar0 + 24, do_full0 = bar0 + 40, do_empty0 = bar0 + 56, stat_full0 = bar0 + 72;
  const uint32_t s_full = bar0 + 88;    // S^T of this tile is complete
  const uint32_t p_full = bar0 + 96;    // P^T is in tensor memory, the scores have been read
  const uint32_t dp_full = bar0 + 104;  // dP^T is complete
  const uint32_t ds_full = bar0 + 112;  // dS^T is in shared memory, dP^T has been read
  const uint32_t ds_empty = bar0 + 120; // dK and dQ have read dS^T
  const uint32_t dq_full = bar0 + 128, dq_read = bar0 + 136, dkv_full = bar0 + 144;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitCtx wc{abort_flag, p.status, kWaitBudgetNs};

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(q_full0 + 8 * s, 1);
      mbar_init(q_empty0 + 8 * s, 1);
      mbar_init(do_full0 + 8 * s, 1);
      mbar_init(do_empty0 + 8 * s, 1);
      mbar_init(stat_full0 + 8 * s, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(ds_empty, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, 4);
    mbar_init(dkv_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (C::kRows && warp == 2) {  // ones in the three places of a query's row
    if (lane < 16) rows_smem[256 + lane] = lane < 8 ? make_uint4(0x3f803f80u, 0x00003f80u, 0, 0) : make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    const bool leader = elect_one();
    if (leader) {
      prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v); prefetch_tmap(&tmap_do);
      prefetch_tmap(&tmap_dq);
      mbar_arrive_expect_tx(kv_full, 2 * C::kTile);
#pragma unroll
      for (int s = 0; s < D / 64; ++s) {
        tma_load_2d(k_smem + s * 16384, &tmap_k, kv_full, kv_head * D + 64 * s, seq_start + kv0);
        tma_load_2d(v_smem + s * 16384, &tmap_v, kv_full, kv_head * D + 64 * s, seq_start + kv0);
      }
    }
    int head = first_head, i = i_first;
    auto load_q = [&](int stage, int row) {
      const uint32_t bar = q_full0 + 8 * stage, dst = base + kQOff + stage * C::kTile;
      mbar_arrive_expect_tx(bar, C::kTile);
#pragma unroll
      for (int s = 0; s < D / 64; ++s) tma_load_2d(dst + s * 16384, &tmap_q, bar, head * D + 64 * s, row);
    };
    if (leader) load_q(0, seq_start + i * 128);   // not after the loads of log-sum-exp and delta below
    for (int it = 0; it < total_iters; ++it) {
      const int qs = it % C::kQStages, os = it % C::kDoStages;
      const int row = seq_start + i * 128;
      float nl[4], dl[4];
      const long long first = static_cast<long long>(head) * p.total_tokens + row;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = lane + 32 * e;
        const bool in = i * 128 + c < seq_len;
        nl[e] = in ? p.lse_scale * p.lse[first + c] : 0.f;
        dl[e] = in ? (C::kRows ? -p.delta[first + c] : p.delta[first + c]) : 0.f;
      }
      if (it > 0) {
        if (!__all_sync(0xffffffffu, mbar_wait(q_empty0 + 8 * qs, ((it / C::kQStages) & 1) ^ 1, wc, 31))) break;
        if (leader) load_q(qs, row);
      }
      if constexpr (C::kRows) {
        // dP(it-1) has read the rows of the tile before
        if (it > 0 && !__all_sync(0xffffffffu, mbar_wait(dp_full, (it - 1) & 1, wc, 25))) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // three bf16 terms hold the 24 bits of each value
          float rest[2] = {nl[e], dl[e]};
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint32_t h[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const __nv_bfloat16 t = __float2bfloat16(rest[r]);
              rest[r] -= __bfloat162float(t);
              h[k] = __bfloat16_as_ushort(t);
            }
            rows_smem[128 * r + lane + 32 * e] = make_uint4(h[0] | h[1] << 16, h[2], 0, 0);
          }
        }
        fence_proxy_async();
      } else {
        // a free Q stage also means that this slot's values have been read: dS was made from them
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          stats[qs * 256 + lane + 32 * e] = nl[e];
          stats[qs * 256 + 128 + lane + 32 * e] = dl[e];
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(stat_full0 + 8 * (C::kRows ? 0 : qs));
      if (!__all_sync(0xffffffffu, mbar_wait(do_empty0 + 8 * os, ((it / C::kDoStages) & 1) ^ 1, wc, 30))) break;
      if (leader) {
        const uint32_t bar = do_full0 + 8 * os, dst = base + kDoOff + os * C::kTile;
        mbar_arrive_expect_tx(bar, C::kTile);
#pragma unroll
        for (int s = 0; s < D / 64; ++s) tma_load_2d(dst + s * 16384, &tmap_do, bar, head * D + 64 * s, row);
      }
      if (++i == n_qblocks) { i = i_first; ++head; }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);  // S^T, dP^T: both operands K-major
      const uint32_t idesc_kn = make_idesc_bf16(128, D, false, true);    // dV (A in tensor memory), dK: K-major x MN-major
      const uint32_t idesc_nn = make_idesc_bf16(128, D, true, true);     // dQ: dS^T read MN-major x MN-major
      const uint64_t ds_k = make_smem_desc(ds_smem, 16, 1024), ds_mn = make_smem_desc(ds_smem, 16384, 1024);
      const uint64_t k_mn = make_smem_desc(k_smem, 16384, 1024);
      auto scores = [&](uint32_t d_col, uint32_t a_smem, uint32_t b_smem) {
        const uint64_t ad = make_smem_desc(a_smem, 16, 1024), bd = make_smem_desc(b_smem, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = ((k >> 2) * 16384 + (k & 3) * 32) >> 4;
          umma_f16(tmem_base + d_col, ad + off, bd + off, idesc_s, k > 0 ? 1u : 0u);
        }
      };
      // rows of 16 bytes without swizzle: both halves of K read the same eight values, all keys the same eight selector rows
      const uint64_t lse_rows = make_plain_desc(base + kStatOff, 0, 128), delta_rows = make_plain_desc(base + kStatOff + 2048, 0, 128);
      const uint64_t sel = make_plain_desc(base + kStatOff + 4096, 128, 0);
      auto issue_s = [&](int it) -> bool {
        if (!mbar_wait(q_full0 + 8 * (it % C::kQStages), (it / C::kQStages) & 1, wc, 33)) return false;
        tc_fence_after();
        scores(C::kS, k_smem, base + kQOff + (it % C::kQStages) * C::kTile);
        if constexpr (C::kRows) {
          if (!mbar_wait(stat_full0, it & 1, wc, 26)) return false;
          umma_f16(tmem_base + C::kS, sel, lse_rows, idesc_s, 1u);      // - log-sum-exp of the query
        }
        umma_commit(s_full);
        return true;
      };
      auto issue_dp = [&](int it) -> bool {
        if (!mbar_wait(do_full0 + 8 * (it % C::kDoStages), (it / C::kDoStages) & 1, wc, 29)) return false;
        tc_fence_after();
        scores(C::kDp, v_smem, base + kDoOff + (it % C::kDoStages) * C::kTile);
        if constexpr (C::kRows) umma_f16(tmem_base + C::kDp, sel, delta_rows, idesc_s, 1u);    // - delta of the query
        umma_commit(dp_full);
        return true;
      };
      auto issue_dk = [&](int it) {  // dK += dS^T Q, over the 128 query rows, 16 at a time
        const uint64_t qd = make_smem_desc(base + kQOff + (it % C::kQStages) * C::kTile, 16384, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if constexpr (C::kPrivate)
            umma_f16_ts(tmem_base + C::kDk, tmem_base + C::kDp + 64 * (k >> 2) + (k & 3) * 8, qd + ((k * 2048) >> 4), idesc_kn,
                        (it > 0 || k > 0) ? 1u : 0u);
          else
            umma_f16(tmem_base + C::kDk, ds_k + (((k >> 2) * 16384 + (k & 3) * 32) >> 4), qd + ((k * 2048) >> 4), idesc_kn,
                     (it > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(q_empty0 + 8 * (it % C::kQStages));
      };
      auto issue_dq = [&]() {  // dQ = dS K, over the 128 keys
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16(tmem_base + C::kDq, ds_mn + ((k * 2048) >> 4), k_mn + ((k * 2048) >> 4), idesc_nn, k > 0 ? 1u : 0u);
        umma_commit(dq_full);
      };
      bool ok = mbar_wait(kv_full, 0, wc, 32) && issue_s(0) && issue_dp(0);
      for (int it = 0; it < total_iters && ok; ++it) {
        const bool more = it + 1 < total_iters;
        if (!(ok = mbar_wait(p_full, it & 1, wc, 35))) break;
        tc_fence_after();
        if (C::kPrivate && more && !(ok = issue_s(it + 1))) break;
        const uint64_t dod = make_smem_desc(base + kDoOff + (it % C::kDoStages) * C::kTile, 16384, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k)  // dV += P^T dO
          umma_f16_ts(tmem_base + C::kDv, tmem_base + C::p_col(k >> 2) + (k & 3) * 8, dod + ((k * 2048) >> 4), idesc_kn,
                      (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(do_empty0 + 8 * (it % C::kDoStages));
        if (!C::kPrivate && more) {
          // P lies in the score columns: they are free once dV(it) is complete
          if (!(ok = mbar_wait(do_empty0 + 8 * (it % C::kDoStages), (it / C::kDoStages) & 1, wc, 28))) break;
          if (!(ok = issue_s(it + 1))) break;
        }
        if (!(ok = mbar_wait(ds_full, it & 1, wc, 27))) break;
        tc_fence_after();
        if (C::kPrivate) {
          issue_dk(it);   // reads dS^T from the columns that dP(it+1) takes
          if (more && !(ok = issue_dp(it + 1))) break;
          if (it > 0 && !(ok = mbar_wait(dq_read, (it - 1) & 1, wc, 34))) break;
          tc_fence_after();
          issue_dq();
          umma_commit(ds_empty);
        } else {
          issue_dq();
          issue_dk(it);
          umma_commit(ds_empty);
          if (more) {  // dP(it+1) takes the columns that dQ(it) is read from
            if (!(ok = mbar_wait(dq_read, it & 1, wc, 34))) break;
            if (!(ok = issue_dp(it + 1))) break;
          }
        }
      }
      if (ok) umma_commit(dkv_full);
    }
  } else if (warp < 10) {
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;            // which 64 of the 128 query columns this warpgroup handles
    const int row = quad * 32 + lane;            // key within the tile
    const int kv = kv0 + row;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    bool ok = true;
    int i = i_first;
    for (int it = 0; it < total_iters; ++it) {
      const float4* nl = reinterpret_cast<const float4*>(stats + (it % C::kQStages) * 256 + half * 64);
      if (!C::kRows && !(ok = mbar_wait(stat_full0 + 8 * (it % C::kQStages), (it / C::kQStages) & 1, wc, 26))) break;
      if (!(ok = mbar_wait(s_full, it & 1, wc, 36))) break;
      tc_fence_after();
      float pr[64];
      {
        uint32_t* r = reinterpret_cast<uint32_t*>(pr);
        tmem_ld_32x32(lanes + C::kS + half * 64, r);
        tmem_ld_32x32(lanes + C::kS + half * 64 + 32, r + 32);
        tmem_ld_wait();
      }
      if constexpr (C::kRows) {  // the log-sum-exp is in the score
#pragma unroll
        for (int v = 0; v < 64; ++v) pr[v] = exp2f(pr[v] * p.scale_log2);
      } else {
#pragma unroll
        for (int v = 0; v < 16; ++v) {
          const float4 l4 = nl[v];
          pr[4 * v] = exp2f(fmaf(pr[4 * v], p.scale_log2, l4.x));
          pr[4 * v + 1] = exp2f(fmaf(pr[4 * v + 1], p.scale_log2, l4.y));
          pr[4 * v + 2] = exp2f(fmaf(pr[4 * v + 2], p.scale_log2, l4.z));
          pr[4 * v + 3] = exp2f(fmaf(pr[4 * v + 3], p.scale_log2, l4.w));
        }
      }
      const int q0 = i * 128;
      if (q0 + 128 > seq_len || kv0 + 128 > seq_len || (p.causal && i * 128 < kv0 + 128)) {
        // queries [lo, hi) of this warpgroup's columns see the key
        const int lo = (p.causal ? kv - q0 : 0) - half * 64, hi = (kv < seq_len ? seq_len - q0 : 0) - half * 64;
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (c < lo || c >= hi) pr[c] = 0.f;
      }
      // S(it) may be complete before dV(it-1), which reads the previous P from its own columns
      if (C::kPrivate && it > 0 &&
          !(ok = mbar_wait(do_empty0 + 8 * ((it - 1) % C::kDoStages), ((it - 1) / C::kDoStages) & 1, wc, 24)))
        break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) pk[c] = pack2(pr[32 * h + 2 * c], pr[32 * h + 2 * c + 1]);
        tmem_st_32x16(lanes + C::p_col(half) + 16 * h, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (!(ok = mbar_wait(dp_full, it & 1, wc, 37))) break;
      tc_fence_after();
      if (it > 0 && !(ok = mbar_wait(ds_empty, (it - 1) & 1, wc, 39))) break;
      // dS without the score scale: dK takes it in its epilogue and dQ where it is narrowed to bf16
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tmem_ld_32x32(lanes + C::kDp + half * 64 + 32 * h, r);
        tmem_ld_wait();
        uint32_t pk[16];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const float* pv = pr + 32 * h + 8 * v;
          const uint32_t* rv = r + 8 * v;
          float dl[8] = {};
          if constexpr (!C::kRows) {
            const float4 a = nl[32 + 8 * h + 2 * v], b = nl[32 + 8 * h + 2 * v + 1];
            dl[0] = a.x; dl[1] = a.y; dl[2] = a.z; dl[3] = a.w; dl[4] = b.x; dl[5] = b.y; dl[6] = b.z; dl[7] = b.w;
          }
          auto two = [&](int c) {
            return pack2(pv[c] * (__uint_as_float(rv[c]) - dl[c]), pv[c + 1] * (__uint_as_float(rv[c + 1]) - dl[c + 1]));
          };
          const uint4 o = make_uint4(two(0), two(2), two(4), two(6));
          *reinterpret_cast<uint4*>(smem + kDsOff + swz_chunk_offset(row, half * 8 + 4 * h + v)) = o;
          pk[4 * v] = o.x; pk[4 * v + 1] = o.y; pk[4 * v + 2] = o.z; pk[4 * v + 3] = o.w;
        }
        if constexpr (C::kPrivate) tmem_st_32x16(lanes + C::kDp + half * 64 + 16 * h, pk);
      }
      if constexpr (C::kPrivate) tmem_st_wait();
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      if (++i == n_qblocks) i = i_first;
    }
    // dK / dV of this key tile: one warpgroup writes dV, the other dK
    if (ok) ok = mbar_wait(dkv_full, 0, wc, 38);
    if (ok) {
      tc_fence_after();
      const long long off = static_cast<long long>(seq_start + kv) * p.dkv_stride + kv_head * D;
      __nv_bfloat16* dst = (half == 0 ? p.dv : p.dk) + off;
      const uint32_t src = lanes + (half == 0 ? C::kDv : C::kDk);
      const float f = half == 0 ? 1.f : p.scale;
      float* sum = p.kv_parts + ((static_cast<long long>(2 * part + 1 - half) * p.total_tokens + seq_start + kv) * p.n_kv + kv_head) * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(src + c * 32, r);
        tmem_ld_wait();
        if (kv < seq_len && p.parts > 1) {
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<uint4*>(sum + c * 32 + v * 4) = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
        } else if (kv < seq_len) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 o;
            o.x = pack2(__uint_as_float(r[8 * v]) * f, __uint_as_float(r[8 * v + 1]) * f);
            o.y = pack2(__uint_as_float(r[8 * v + 2]) * f, __uint_as_float(r[8 * v + 3]) * f);
            o.z = pack2(__uint_as_float(r[8 * v + 4]) * f, __uint_as_float(r[8 * v + 5]) * f);
            o.w = pack2(__uint_as_float(r[8 * v + 6]) * f, __uint_as_float(r[8 * v + 7]) * f);
            *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = o;
          }
        }
      }
    }
  } else {
    // dQ tile -> fp32 staging, 32 columns at a time in two alternating boxes -> TMA reduce-add into the global accumulator;
    // rows past the end of the sequence are staged as zeros.  A warp that gives up keeps walking the named barriers.
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t src = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + C::kDq;
    const bool issuer = warp == 10 && lane == 0;
    bool ok = true;
    int head = first_head, i = i_first;
    for (int it = 0; it < total_iters; ++it) {
      ok = ok && mbar_wait(dq_full, it & 1, wc, 40);
      tc_fence_after();
      const bool q_valid = i * 128 + row < seq_len;
#pragma unroll 1
      for (int c = 0; c < D / 32; c += 2) {
        uint32_t r[64];
        tmem_ld_32x32(src + c * 32, r);
        tmem_ld_32x32(src + c * 32 + 32, r + 32);
        tmem_ld_wait();
        if (c + 2 == D / 32) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_read);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if (issuer) bulk_wait_group_read1();  // the box two steps back has been read
          named_barrier_sync(1, 128);
          uint8_t* box = smem + kStageOff + b * 16384 + row * 128;
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const uint32_t* x = r + 32 * b + 4 * v;
            *reinterpret_cast<uint4*>(box + ((v ^ (row & 7)) << 4)) =
                q_valid ? make_uint4(x[0], x[1], x[2], x[3]) : make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async();
          named_barrier_sync(1, 128);
          if (issuer && ok) {
            tma_reduce_add_2d(&tmap_dq, base + kStageOff + b * 16384, head * D + 32 * (c + b), seq_start + i * 128);
            bulk_commit_group();
          }
        }
      }
      if (++i == n_qblocks) { i = i_first; ++head; }
    }
    if (issuer) bulk_wait_group0();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d].  A thread takes 16 bytes of both tensors; the D/8 threads of one
// (token, head) pair are neighbours in a warp and combine with shuffles.  A CTA covers 256 / (D/8) consecutive tokens of
// kDeltaHeads heads, all of them loaded at once, so the loads of a warp are whole 128-byte rows and the stores of one head
// form one contiguous run of tokens.  (One CTA walking all heads, one load at a time: 765 tokens, 12 heads, D = 128,
// 11.0 us, now 4.3; 16321 tokens, 32 heads, D = 64, 31.9 us, now 22.1.)
constexpr int kDeltaHeads = 4;
template <int D>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ o, float* __restrict__ delta,
                  float* __restrict__ dq_acc, int total_tokens, int n_q, long long do_stride, long long o_stride) {
  constexpr int kLanes = D / 8;               // threads per (token, head)
  constexpr int kTokens = 256 / kLanes;       // tokens per CTA
  const int part = threadIdx.x % kLanes;
  const int t = blockIdx.x * kTokens + threadIdx.x / kLanes;
  const int h0 = blockIdx.y * kDeltaHeads;
  const bool live = t < total_tokens;
  const __nv_bfloat16* a = dout + static_cast<long long>(live ? t : 0) * do_stride + part * 8;
  const __nv_bfloat16* b = o + static_cast<long long>(live ? t : 0) * o_stride + part * 8;
  uint4 x[kDeltaHeads], y[kDeltaHeads];
#pragma unroll
  for (int k = 0; k < kDeltaHeads; ++k) {
    const int h = min(h0 + k, n_q - 1);
    x[k] = *reinterpret_cast<const uint4*>(a + h * D);
    y[k] = *reinterpret_cast<const uint4*>(b + h * D);
  }
#pragma unroll
  for (int k = 0; k < kDeltaHeads; ++k) {
    const uint32_t xs[4] = {x[k].x, x[k].y, x[k].z, x[k].w}, ys[4] = {y[k].x, y[k].y, y[k].z, y[k].w};
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s += __uint_as_float(xs[i] << 16) * __uint_as_float(ys[i] << 16);
      s += __uint_as_float(xs[i] & 0xffff0000u) * __uint_as_float(ys[i] & 0xffff0000u);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (live && h0 + k < n_q) {
      if (part == 0) delta[static_cast<long long>(h0 + k) * total_tokens + t] = s;
      float4* acc = reinterpret_cast<float4*>(dq_acc + (static_cast<long long>(t) * n_q + h0 + k) * D + part * 8);
      acc[0] = acc[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// dq = bf16(acc * scale); acc is dense [tokens, width] fp32; dq rows are dq_stride elements apart.  With parts > 1 also
// dk = bf16(scale * sum over parts) and dv = bf16(sum over parts), in order, from dense [parts][2][tokens, kv width] fp32.
__global__ void __launch_bounds__(256)
narrow_grads_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long long n8, int width8, long long dq_stride,
                    float scale, const float* __restrict__ kv_parts, int parts, __nv_bfloat16* __restrict__ dk,
                    __nv_bfloat16* __restrict__ dv, long long kv_n8, int kv_width8, long long dkv_stride) {
  const long long total = n8 + (parts > 1 ? 2 * kv_n8 : 0);
  for (long long v = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; v < total;
       v += static_cast<long long>(gridDim.x) * blockDim.x) {
    const bool is_q = v < n8, is_v = v >= n8 + kv_n8;
    const long long i = is_q ? v : v - n8 - (is_v ? kv_n8 : 0);
    const float* src = is_q ? acc + v * 8 : kv_parts + (v - n8) * 8;
    float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    if (!is_q) {
      for (int s = 1; s < parts; ++s) {
        src += 16 * kv_n8;
        const float4 c = *reinterpret_cast<const float4*>(src), d = *reinterpret_cast<const float4*>(src + 4);
        a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
        b.x += d.x; b.y += d.y; b.z += d.z; b.w += d.w;
      }
    }
    const int w8 = is_q ? width8 : kv_width8;
    const long long row = i / w8;
    const int col = static_cast<int>(i % w8) * 8;
    __nv_bfloat16* dst = is_q ? dq + row * dq_stride : (is_v ? dv : dk) + row * dkv_stride;
    const float f = is_v ? 1.f : scale;
    *reinterpret_cast<uint4*>(dst + col) =
        make_uint4(pack2(a.x * f, a.y * f), pack2(a.z * f, a.w * f), pack2(b.x * f, b.y * f), pack2(b.z * f, b.w * f));
  }
}

// The same for queries and keys that were rotated by their positions after the projection: the gradients are rotated back on the
// way, rounded before as the pass over them finds them, and v's are left alone.  Bound by memory: fp32 dQ read once, dQ written and dK read
// and written once, instead of a pass that narrows dQ and one over the whole of dqkv (16321 tokens, 32/8 heads of 64: 35 + 43 us).
// 128 threads for two tokens: 16321 tokens, 32/8 heads of 64, 40.3 us; 256 for four 41.9, for two 48.5, 128 for one 45.2; 1000 tokens,
// 12/2 heads of 128, 6.1, 7.2, 6.0, 5.6.
constexpr int kFinishTokens = 2, kFinishThreads = 128;
template <int D>
__global__ void __launch_bounds__(kFinishThreads)
finish_rope_grads_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk,
                         __nv_bfloat16* __restrict__ dv, int total_tokens, int n_q, int n_kv, long long dq_stride, long long dkv_stride,
                         float scale, const float* __restrict__ kv_parts, int parts, const long long* __restrict__ pos, float log2_theta) {
  constexpr int kHalf = D / 2, kVecs = kHalf / 8;
  __shared__ float cs[kFinishTokens][2][kHalf];   // cosine and sine of the rotation back
  const int t0 = blockIdx.x * kFinishTokens, tokens = min(kFinishTokens, total_tokens - t0);
  for (int i = threadIdx.x; i < tokens * kHalf; i += blockDim.x) {
    const int f = i % kHalf;
    float sn, c;
    sincosf(static_cast<float>(pos[t0 + i / kHalf]) * exp2f(-log2_theta * (2.0f * f) / D), &sn, &c);
    cs[i / kHalf][0][f] = c;
    cs[i / kHalf][1][f] = -sn;
  }
  __syncthreads();
  const long long part_stride = 2ll * total_tokens * n_kv * D;
  auto load8 = [&](const float* src, float* x, int n_parts) {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = 0.f;
    for (int s = 0; s < n_parts; ++s, src += part_stride) {
      const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
      x[0] += a.x; x[1] += a.y; x[2] += a.z; x[3] += a.w;
      x[4] += b.x; x[5] += b.y; x[6] += b.z; x[7] += b.w;
    }
  };
  auto load8_bf16 = [&](const __nv_bfloat16* src, float* x) {
    const uint4 u = *reinterpret_cast<const uint4*>(src);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = __uint_as_float(w[i] << 16);
      x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  };
  auto store8 = [&](__nv_bfloat16* dst, const float* x) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack2(x[0], x[1]), pack2(x[2], x[3]), pack2(x[4], x[5]), pack2(x[6], x[7]));
  };
  const int per_token = (n_q + n_kv) * kVecs;
  for (int i = threadIdx.x; i < tokens * per_token; i += blockDim.x) {
    const int tok = i / per_token, it = i - tok * per_token, head = it / kVecs, j = it % kVecs * 8;
    const long long t = t0 + tok;
    float x1[8], x2[8], o1[8], o2[8];
    __nv_bfloat16* dst;
    float f = scale;
    if (head < n_q) {
      const float* src = acc + (t * n_q + head) * D + j;
      load8(src, x1, 1);
      load8(src + kHalf, x2, 1);
      dst = dq + t * dq_stride + head * D + j;
    } else {
      dst = dk + t * dkv_stride + (head - n_q) * D + j;
      if (parts > 1) {
        const float* src = kv_parts + (t * n_kv + head - n_q) * D + j;
        load8(src, x1, parts);
        load8(src + kHalf, x2, parts);
      } else {   // scaled and rounded by the kernel that formed it
        load8_bf16(dst, x1);
        load8_bf16(dst + kHalf, x2);
        f = 1.f;
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float a = __bfloat162float(__float2bfloat16(x1[e] * f)), b = __bfloat162float(__float2bfloat16(x2[e] * f));
      rotate_pair(a, b, cs[tok][0][j + e], cs[tok][1][j + e], &o1[e], &o2[e]);
    }
    store8(dst, o1);
    store8(dst + kHalf, o2);
  }
  if (parts > 1) {
    const int v_per_token = n_kv * D / 8;
    for (int i = threadIdx.x; i < tokens * v_per_token; i += blockDim.x) {
      const int tok = i / v_per_token, col = (i - tok * v_per_token) * 8;
      const long long t = t0 + tok;
      float x[8];
      load8(kv_parts + (static_cast<long long>(total_tokens) + t) * n_kv * D + col, x, parts);
      store8(dv + t * dkv_stride + col, x);
    }
  }
}

}  // namespace

// D = 128: whether a CTA takes a pair of query tiles, which share its K and V loads and hide each other's softmax, or one, of
// which twice as many spread over the SMs.  Estimated time in us: as long as the longest tile or as an even share of all key
// blocks, 1.3 us a key block for one tile and 1.7 for a pair, plus 1.5 us per wave of CTAs.  The host knows the number of
// sequences and the longest; unless they are all about as long, each counts as half a tile more than it fills, and with
// the key blocks of the longest.  (max_seqlen is the caller's word; a wrong one costs time only.)  Several waves of pairs
// of one head that mostly lack their second tile are not worth it either.  Fitted to the times of 500 shapes, 100 to
// 32000 tokens in 1 to 300 sequences, 1 to 40 heads: never slower than pairs throughout.  1000 tokens in one sequence,
// 12/2 heads: pairs 24.6 us, single 15.3; 8000 tokens, 1 head: 138 and 82; 8000 tokens, 12/2 heads: 220 and 232; 12
// sequences of 300 tokens, 14/2 heads: 36.5 and 31.1.
bool attn_fwd_pairs(int total_tokens, int num_seqs, int max_seqlen, int n_q, int n_kv, bool causal, int sm_count) {
  const double longest = std::min(std::max(max_seqlen, 1), total_tokens);
  const double key_blocks = std::ceil(longest / kBlockKV);
  const double per_tile = causal ? (key_blocks + 1) / 2 : key_blocks;
  auto ctas = [&](double rows) {  // per head
    return num_seqs * longest <= 1.1 * total_tokens ? num_seqs * std::ceil(longest / rows) : total_tokens / rows + num_seqs / 2.0;
  };
  const double tiles = n_q * ctas(kBlockQ);
  const double pairs = (n_q / n_kv) % 2 == 0 ? tiles / 2 : n_q * ctas(2 * kBlockQ);
  auto cost = [&](double n, double block_us) {
    return block_us * std::max(key_blocks, n * per_tile / sm_count) + 1.5 * std::ceil(n / sm_count);
  };
  if (2 * pairs > 1.3 * tiles && pairs > sm_count) return false;
  return cost(pairs, 1.7) <= cost(tiles, 1.3);
}

cudaError_t attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int* cu_seqlens,
                     int num_seqs, int total_tokens, int max_seqlen, int n_q, int n_kv, int head_dim,
                     long long q_stride, long long kv_stride, long long o_stride, float scale, bool causal,
                     int* status, int sm_count, cudaStream_t stream) {
  if (total_tokens == 0 || num_seqs == 0) return cudaSuccess;
  if (head_dim != 64 && head_dim != 128) return cudaErrorInvalidValue;
  if (n_q % n_kv != 0) return cudaErrorInvalidValue;
  if ((q_stride % 8) || (kv_stride % 8) || (o_stride % 8)) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o)) & 15)
    return cudaErrorMisalignedAddress;
  CUtensorMap tq, tk, tv;
  if (!encode_tile_map_2d(&tq, q, static_cast<uint64_t>(n_q) * head_dim, total_tokens, q_stride * 2, 64, kBlockQ) ||
      !encode_tile_map_2d(&tk, k, static_cast<uint64_t>(n_kv) * head_dim, total_tokens, kv_stride * 2, 64, kBlockKV) ||
      !encode_tile_map_2d(&tv, v, static_cast<uint64_t>(n_kv) * head_dim, total_tokens, kv_stride * 2, 64, kBlockKV))
    return cudaErrorInvalidValue;
  FwdParams p;
  p.cu_seqlens = cu_seqlens; p.num_seqs = num_seqs; p.n_q = n_q; p.n_kv = n_kv;
  p.o = static_cast<__nv_bfloat16*>(o); p.o_stride = o_stride; p.lse = lse; p.total_tokens = total_tokens;
  p.scale_log2 = scale * kLog2e; p.causal = causal ? 1 : 0; p.status = status;
  const bool pairs = head_dim == 128 && attn_fwd_pairs(total_tokens, num_seqs, max_seqlen, n_q, n_kv, causal, sm_count);
  // a pair takes two heads of a key/value group: both tiles then see the same keys, and a short sequence fills both.  An
  // odd group is walked two query tiles at a time instead.
  const int tiles = pairs ? 2 : 1;
  p.heads_per_cta = (n_q / n_kv) % tiles == 0 ? tiles : 1;
  const int rows = kBlockQ * tiles / p.heads_per_cta;
  const unsigned int grid = ((total_tokens + rows - 1) / rows + num_seqs) * (n_q / p.heads_per_cta);
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    auto allow = [](auto kernel, int smem) {
      if (attr_err == cudaSuccess) attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    };
    allow(attn_fwd_kernel<64, 1>, FwdCfg<64, 1>::kSmem);
    allow(attn_fwd_kernel<128, 1>, FwdCfg<128, 1>::kSmem);
    allow(attn_fwd_kernel<128, 2>, FwdCfg<128, 2>::kSmem);
  });
  if (attr_err != cudaSuccess) return attr_err;
  if (head_dim == 64)
    launch(attn_fwd_kernel<64, 1>, grid, FwdCfg<64, 1>::kThreads, FwdCfg<64, 1>::kSmem, stream, tq, tk, tv, p);
  else if (!pairs)
    launch(attn_fwd_kernel<128, 1>, grid, FwdCfg<128, 1>::kThreads, FwdCfg<128, 1>::kSmem, stream, tq, tk, tv, p);
  else
    launch(attn_fwd_kernel<128, 2>, grid, FwdCfg<128, 2>::kThreads, FwdCfg<128, 2>::kSmem, stream, tq, tk, tv, p);
  return cudaGetLastError();
}

}  // namespace odc

namespace odc {

// Into how many CTAs the query heads of one (key tile, kv head) are divided: a divisor of the group.  Estimated time in us:
// as long as the longest tile with its heads or as an even share of all products of tiles, 3 us each, plus 5 us per wave of
// CTAs and, divided, 0.25 us per MB of the fp32 partial dK and dV; a finer division has to be 15 % better.  The host knows
// the number of sequences and the longest, so the others count as half a tile more than they fill, and as long.  Fitted to
// 514 timings (100 to 20000 tokens in 1 to 300 sequences, 2 to 40 heads, both head sizes): 0.3 % above the best division on
// average.  D = 128, 12/2 heads: 765 tokens 93 us whole, 45 divided by six; 2048 tokens 275 and 79.  Dividing whenever there
// were fewer tiles than SMs cost short sequences the partial sums for nothing: 300 sequences of 20 tokens, 14/2 heads,
// 160 us whole, 356 divided by seven.
int attn_bwd_parts(int total_tokens, int num_seqs, int max_seqlen, int n_q, int n_kv, int head_dim, bool causal, int sm_count) {
  const int rep = n_q / n_kv;
  const double longest = (std::min(std::max(max_seqlen, 1), total_tokens) + 127) / 128;
  const double tiles = n_kv * (total_tokens / 128.0 + num_seqs / 2.0);
  const double even = tiles * rep * (causal ? (longest + 1) / 2 : longest) / sm_count;
  const double partial_mb = 8e-6 * total_tokens * n_kv * head_dim;
  auto cost = [&](int parts) {
    return 3.0 * std::max(longest * rep / parts, even) + 5.0 * std::ceil(tiles * parts / sm_count) +
           (parts > 1 ? 0.25 * parts * partial_mb : 0.0);
  };
  int best = 1;
  for (int parts = 2; parts <= rep; ++parts)
    if (rep % parts == 0 && cost(parts) < 0.85 * cost(best)) best = parts;
  return best;
}

cudaError_t attn_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse,
                     void* dq, void* dk, void* dv, float* delta, float* dq_acc, float* kv_parts, int parts,
                     const int* cu_seqlens, int num_seqs,
                     int total_tokens, int max_seqlen, int n_q, int n_kv, int head_dim, long long q_stride,
                     long long kv_stride, long long o_stride, long long dq_stride, long long dkv_stride, float scale,
                     bool causal, int* status, int sm_count, cudaStream_t stream, const long long* rope_pos, float rope_theta) {
  (void)max_seqlen;
  if (total_tokens == 0 || num_seqs == 0) return cudaSuccess;
  if (head_dim != 64 && head_dim != 128) return cudaErrorInvalidValue;
  if (n_q % n_kv != 0 || parts < 1 || n_q / n_kv % parts != 0 || (parts > 1 && kv_parts == nullptr))
    return cudaErrorInvalidValue;
  if ((q_stride % 8) || (kv_stride % 8) || (o_stride % 8) || (dq_stride % 8) || (dkv_stride % 8))
    return cudaErrorInvalidValue;
  // dout is contiguous [T, n_q, D]; dq / dk / dv rows may be strided (views of one fused qkv gradient)
  const long long do_stride = static_cast<long long>(n_q) * head_dim;
  const unsigned int delta_y = (n_q + kDeltaHeads - 1) / kDeltaHeads;
  if (head_dim == 64) {
    launch(attn_delta_kernel<64>, dim3((total_tokens + 31) / 32, delta_y), 256, 0, stream,
        static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(o), delta, dq_acc, total_tokens, n_q,
        do_stride, o_stride);
  } else {
    launch(attn_delta_kernel<128>, dim3((total_tokens + 15) / 16, delta_y), 256, 0, stream,
        static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(o), delta, dq_acc, total_tokens, n_q,
        do_stride, o_stride);
  }
  CUtensorMap tq, tk, tv, tdo, tdq;
  if (!encode_tile_map_2d_f32(&tdq, dq_acc, static_cast<uint64_t>(n_q) * head_dim, total_tokens,
                              static_cast<uint64_t>(n_q) * head_dim * 4, 32, 128))
    return cudaErrorInvalidValue;
  if (!encode_tile_map_2d(&tq, q, static_cast<uint64_t>(n_q) * head_dim, total_tokens, q_stride * 2, 64, 128) ||
      !encode_tile_map_2d(&tk, k, static_cast<uint64_t>(n_kv) * head_dim, total_tokens, kv_stride * 2, 64, 128) ||
      !encode_tile_map_2d(&tv, v, static_cast<uint64_t>(n_kv) * head_dim, total_tokens, kv_stride * 2, 64, 128) ||
      !encode_tile_map_2d(&tdo, dout, static_cast<uint64_t>(n_q) * head_dim, total_tokens, do_stride * 2, 64, 128))
    return cudaErrorInvalidValue;
  BwdParams p;
  p.cu_seqlens = cu_seqlens; p.num_seqs = num_seqs; p.n_q = n_q; p.n_kv = n_kv; p.lse = lse; p.delta = delta;
  p.dq_acc = dq_acc; p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  p.total_tokens = total_tokens; p.scale = scale; p.causal = causal ? 1 : 0;
  if (head_dim == 64) {
    // The log-sum-exp joins the scores before they are scaled, divided by the scale.  A scale of zero (all keys alike), or one
    // whose quotient could leave fp32, counts as 2^-100 here: no score below 2^76 shows beside a log-sum-exp then.
    const float score_scale = std::fabs(scale) < 0x1p-100f ? 0x1p-100f : scale;
    p.scale_log2 = score_scale * kLog2e;
    p.lse_scale = -1.f / score_scale;
  } else {
    p.scale_log2 = scale * kLog2e;
    p.lse_scale = -kLog2e;
  }
  p.status = status; p.dkv_stride = dkv_stride;
  p.parts = parts;
  p.kv_parts = kv_parts;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(attn_bwd_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdCfg<64>::kSmem);
    if (attr_err == cudaSuccess)
      attr_err = cudaFuncSetAttribute(attn_bwd_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      BwdCfg<128>::kSmem);
  });
  if (attr_err != cudaSuccess) return attr_err;
  const unsigned int grid = ((total_tokens + 127) / 128 + num_seqs) * n_kv * p.parts;
  if (head_dim == 64)
    launch(attn_bwd_kernel<64>, grid, kBwdThreads, BwdCfg<64>::kSmem, stream, tq, tk, tv, tdo, tdq, p);
  else
    launch(attn_bwd_kernel<128>, grid, kBwdThreads, BwdCfg<128>::kSmem, stream, tq, tk, tv, tdo, tdq, p);
  if (rope_pos != nullptr) {
    const auto kernel = head_dim == 64 ? finish_rope_grads_kernel<64> : finish_rope_grads_kernel<128>;
    launch(kernel, (total_tokens + kFinishTokens - 1) / kFinishTokens, kFinishThreads, 0, stream, static_cast<const float*>(dq_acc),
           static_cast<__nv_bfloat16*>(dq), static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), total_tokens, n_q, n_kv,
           dq_stride, dkv_stride, scale, static_cast<const float*>(kv_parts), p.parts, rope_pos, log2f(rope_theta));
    return cudaGetLastError();
  }
  const long long n8 = static_cast<long long>(total_tokens) * n_q * head_dim / 8;
  const long long kv_n8 = static_cast<long long>(total_tokens) * n_kv * head_dim / 8;
  long long g = (n8 + (p.parts > 1 ? 2 * kv_n8 : 0) + 255) / 256;
  if (g > sm_count * 16) g = sm_count * 16;
  launch(narrow_grads_kernel, static_cast<int>(g), 256, 0, stream,
      dq_acc, static_cast<__nv_bfloat16*>(dq), n8, n_q * head_dim / 8, dq_stride, scale, kv_parts, p.parts,
      static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), kv_n8, n_kv * head_dim / 8, dkv_stride);
  return cudaGetLastError();
}

cudaError_t launch_exp2_poly(const float* x, float* y, long long n, cudaStream_t stream) {
  if (n % 2 != 0) return cudaErrorInvalidValue;
  if (n == 0) return cudaSuccess;
  launch(exp2_poly_kernel, static_cast<unsigned int>((n / 2 + 255) / 256), 256, 0, stream, reinterpret_cast<const float2*>(x),
      reinterpret_cast<float2*>(y), n / 2);
  return cudaGetLastError();
}

}  // namespace odc
