// Host-callable launchers of every kernel in this package.  Plain pointers + stream: no PyTorch
// headers, so kernel files compile in seconds; the binding layer converts tensors.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace odc {

enum DType : int { kF32 = 0, kBF16 = 1, kF16 = 2 };

// ---- communication -------------------------------------------------------------------------
// Debug launches (ODC_DEBUG_BOUNDS=1): `check` / a non-zero `src_region_elems` / `acc_len` make the kernel verify,
// before it touches anything, that the rotation start names a member of the group, that no table entry is null or
// misaligned, and that the elements it is about to read (gather) or add (scatter) fit the DECLARED length of the
// registered region.  A refused launch sets kErrBounds / kErrPeerIndex in the status word and returns normally.
cudaError_t launch_gather(const long long* peers, void* out, size_t n, int src_elem_size, int dst_elem_size,
                          bool src_is_f32_dst_is_bf16, int nranks, int start, bool check, int* status,
                          int sm_count, cudaStream_t stream, size_t src_region_elems = 0);
cudaError_t launch_scatter_accumulate(const void* inp, int in_kind, const long long* accs, int acc_kind,
                                      const long long* ctrs, size_t n, int nranks, int start, float scale,
                                      unsigned int* done_slot, int sm_count, cudaStream_t stream,
                                      int* status_for_bulk = nullptr, long long acc_len = 0,
                                      const float* scale_ptr = nullptr /* device factor on top of scale, fp32 accumulators */);
// row t of dx (bf16 [tokens, width]) times scale is added to row ids[t] of a matrix whose rows are spread over nranks
// fp32 accumulators, rows_per_rank each; ids outside [0, vocab) are skipped; then one arrival per owner
cudaError_t launch_embedding_scatter(const long long* ids, const void* dx, int tokens, int width, const long long* accs,
                                     const long long* ctrs, long long rows_per_rank, long long vocab, int nranks, float scale,
                                     unsigned int* done_slot, int sm_count, cudaStream_t stream);
// scatter_accumulate taken straight from up to kMaxScatterSegments contiguous gradient tensors (fp32 accumulators
// only).  The caller fills count/src/chunk/total/dst; the launcher derives tile_prefix and vec.
constexpr int kMaxScatterSegments = 32;
struct ScatterSegments {
  int count;
  const void* src[kMaxScatterSegments];       // contiguous gradient tensor
  long long chunk[kMaxScatterSegments];       // elements per owner (dim-0 chunk of the padded tensor)
  long long total[kMaxScatterSegments];       // elements that exist (owners past the end get fewer or none)
  long long dst[kMaxScatterSegments];         // element offset inside every owner's accumulator
  long long tile_prefix[kMaxScatterSegments + 1];
  int vec[kMaxScatterSegments];
};
cudaError_t launch_scatter_accumulate_segments(ScatterSegments segs, int in_kind, const long long* accs,
                                               const long long* ctrs, int nranks, int start, float scale,
                                               unsigned int* done_slot, int sm_count, cudaStream_t stream,
                                               long long acc_len = 0, int* status = nullptr);
cudaError_t launch_wait_counter(const void* ctr, unsigned long long expected, unsigned long long budget_ns,
                                int* status, cudaStream_t stream);
// One-sided exchange of the dispatch counts (what `sync` needs to know how many arrivals to wait for).
// post: value[i] = (synchronisation number << 32) | contributions sent so far to owner i, stored with a system-scope
// release at slot_addr[i] (this producer's slot on owner i).  wait: collect nprod postings of `epoch` from the
// local slots, then wait until the arrival counter reaches their sum; bounded, reports through `status`.
constexpr int kMaxPostedCounts = 72;
struct PostedCounts {
  int n;
  long long slot_addr[kMaxPostedCounts];
  unsigned long long value[kMaxPostedCounts];
};
cudaError_t launch_post_counts(const PostedCounts& pc, cudaStream_t stream);
cudaError_t launch_wait_posted(const void* slots, int nprod, unsigned long long epoch, const void* ctr,
                               unsigned long long budget_ns, int* status, unsigned long long* expected_out,
                               cudaStream_t stream);
// Both in one launch: post to every owner, then wait; then (epoch << 8) | status code is written to host_word (the device address of
// pinned host memory), where the caller finds it without a copy or a synchronisation.
cudaError_t launch_post_and_wait(const PostedCounts& pc, const void* slots, int nprod, unsigned long long epoch, const void* ctr,
                                 unsigned long long budget_ns, int* status, unsigned long long* host_word, cudaStream_t stream);

// ---- single-primitive test kernels (device_prims.cu) ---------------------------------------------
cudaError_t launch_put_block(void* remote_dst, const void* local_src, size_t bytes, cudaStream_t s);
cudaError_t launch_get_block(void* local_dst, const void* remote_src, size_t bytes, cudaStream_t s);
cudaError_t launch_scalar_put_get(int* remote_word, int value, int* readback, cudaStream_t s);
cudaError_t launch_atomic_test(int* word, int* cas_seen, int* swap_seen, int ctas, int expected_old, int cas_new,
                               int swap_new, cudaStream_t s);
cudaError_t launch_grid_barrier_test(unsigned int* counter, int* slots, int* out, int ctas,
                                     unsigned long long budget_ns, int* status, cudaStream_t s);

// ---- elementwise / normalisation (bf16 activations, fp32 math) -----------------------------
cudaError_t launch_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows, int cols, float eps,
                               int sm_count, cudaStream_t stream);
// partial: [grid, cols] fp32 scratch (nullptr: in-kernel atomics into dw), dw: [cols] fp32; dres: optional bf16
// [rows, cols] gradient that reached x through a residual connection, added to dx in the same pass
cudaError_t launch_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                               float* partial, float* dw, int rows, int cols, int grid, cudaStream_t stream,
                               const void* dres = nullptr, bool add = false /* dw += instead of dw = */);
int rmsnorm_bwd_grid(int rows, int sm_count);
cudaError_t launch_rope_qkv(const void* in, void* out, const long long* pos, int tokens, int n_q, int n_kv,
                            int head_dim, float theta, bool inverse, cudaStream_t stream);
cudaError_t launch_swiglu_fwd(const void* gate_up, void* out, long long rows, int f, int sm_count,
                              cudaStream_t stream);
cudaError_t launch_swiglu_bwd(const void* dy, const void* gate_up, void* dgate_up, long long rows, int f,
                              int sm_count, cudaStream_t stream);
// logits [rows, vocab] bf16 are overwritten by scale * (softmax - onehot); loss += sum scale * nll
cudaError_t launch_ce_fwd_bwd(void* logits, const long long* labels, const float* loss_scale, float* loss,
                              int rows, int vocab, long long ignore_index, cudaStream_t stream, float inv_temp = 1.f);
// per_token[row] = log_softmax(logits[row] * inv_temp)[labels[row]] (0 where the label is ignore_index); logits are only read
cudaError_t launch_token_logprobs(const void* logits, const long long* labels, float* per_token, int rows, int vocab,
                                  long long ignore_index, cudaStream_t stream, float inv_temp = 1.f);
cudaError_t launch_adamw(float* p, const void* g, int g_kind, float* m, float* v, void* p_lowp, size_t n, float lr,
                         float beta1, float beta2, float eps, float wd, float bc1, float bc2, float grad_scale,
                         cudaStream_t stream);
// column sums of a bf16 [rows, cols] matrix, fp32 inside: rounded into out (bf16) or added to sink (fp32); cols % 8 == 0
cudaError_t launch_column_sum(const void* x, void* out, float* sink, long long rows, int cols, cudaStream_t stream);
// a, b (bf16 [n]) = the halves of in (fp32 [2, n])
cudaError_t launch_narrow_pair(const float* in, void* a, void* b, int n, cudaStream_t stream);
// out (bf16) = in (fp32 or bf16) * *scale
cudaError_t launch_scale_to_bf16(const void* in, int in_kind, void* out, const float* scale, size_t n, int sm_count,
                                 cudaStream_t stream);
cudaError_t launch_cast_f32_to_bf16(const float* in, void* out, size_t n, int sm_count, cudaStream_t stream);
cudaError_t launch_sumsq(const void* x, int kind, size_t n, float* out, int sm_count, cudaStream_t stream);

// ---- tcgen05 GEMM ----------------------------------------------------------------------------
// layout: 0 = "nt" C[M,N] = A[M,K] B[N,K]^T ; 1 = "nn" C = A[M,K] B[K,N] ; 2 = "tn" C = A[K,M]^T B[K,N]
// All operands row-major bf16; C is bf16 or fp32; bias (bf16, length N) optional; accumulate adds into C.
cudaError_t gemm_bf16(const void* a, const void* b, void* c, int c_kind, const void* bias, int M, int N, int K,
                      int layout, bool accumulate, long long lda, long long ldb, long long ldc, int* status,
                      int sm_count, cudaStream_t stream, const void* residual = nullptr, long long ldr = 0,
                      int pair_mode = -1 /* -1: ODC_GEMM_PAIR decides, 0: single-CTA kernel, 1: CTA-pair kernel */,
                      float* split_ws = nullptr);
bool gemm_pairs_enabled();   // ODC_GEMM_PAIR=0 (read once) keeps every product on the single-CTA kernel
// How the CTA-pair kernel takes a product that it is given scratch for (split_ws): the first `whole` of its 256 x 256 tiles as
// they are, the reduction of every other in `parts`.  No scratch bytes: nothing is divided.
struct GemmPlan {
  int tiles, whole, parts;
  size_t scratch_bytes;
};
GemmPlan gemm_plan(int M, int N, int K, int c_kind, int sm_count);
// the same of a weight gradient that is added into its owners' accumulators (no scratch) and may be divided
GemmPlan scatter_plan(int n_out, int k_in, int tokens, int nranks, int sm_count);

// Same contract on CTA pairs (tcgen05 cta_group::2, 256 x 256 tiles).  Returns cudaErrorNotSupported for shapes it
// does not take (N below 256, M below 256 without split_ws, bf16 accumulation); gemm_bf16 tries it first unless ODC_GEMM_PAIR=0.
cudaError_t gemm_bf16_pair(const void* a, const void* b, void* c, int c_kind, const void* bias, int M, int N, int K,
                           int layout, bool accumulate, long long lda, long long ldb, long long ldc, int* status,
                           int sm_count, cudaStream_t stream, const void* residual = nullptr, long long ldr = 0,
                           float* split_ws = nullptr);

// Up to three products of one layout each, none of which reads what another writes, as one launch on CTA pairs.  C is bf16 or fp32,
// times scale and, unless scale_ptr is null, the value there; an fp32 result is added to C if accumulate, and to a bf16
// one an fp32 matrix may be added.  ctr_ptrs: device table whose first entry is an arrival counter that receives
// `arrivals` once everything is in memory (0: none).  scratch: the plan's scratch_bytes.  words: kGroupLaunchWords zeros that are
// this launch's alone while it runs, left zero by it unless a wait runs out: gemm_group_words() of its stream (null: no more of
// them), but not for a captured launch, which may run on another stream.  gemm_group_new_words(): a launch on this device has given up.
// cudaErrorNotSupported: one by one.
constexpr int kMaxGroupProducts = 3;
constexpr int kMaxGroupDivided = 512;   // divided tiles of a launch: those of two rounds of pairs for each product, at most
constexpr int kGroupLaunchWords = 2 + 2 * kMaxGroupDivided;
struct GemmProduct {
  const void *a, *b;
  void* c;
  int c_kind, M, N, K, layout;
  bool accumulate, whole;   // whole: the sum is not divided, as a bf16 product by itself or one that is added in any order may be
  long long lda, ldb, ldc;
  float scale;
  const float* scale_ptr;
  const float* addend;   // bf16 C: fp32 [M, N], joins the sum before scale and rounding
};
struct GemmGroupPlan {
  bool taken;
  int parts[kMaxGroupProducts];     // of every tile (1 where some are whole); 0: not taken as a group
  int columns[kMaxGroupProducts];   // of a tile
  GemmPlan tiles[kMaxGroupProducts];
  int kb_split[kMaxGroupProducts];  // k-blocks of a part
  int order[kMaxGroupProducts];     // longest items first
  size_t scratch_bytes;
};
GemmGroupPlan gemm_group_plan(const GemmProduct* g, int n, int sm_count);
bool gemm_group_takes(const GemmProduct* g, int n, int sm_count);   // what gemm_group answers with cudaErrorNotSupported is false
unsigned int* gemm_group_words(cudaStream_t stream);
void gemm_group_new_words();
cudaError_t gemm_group(const GemmProduct* g, int n, const GemmGroupPlan& plan, float* scratch, unsigned int* words,
                       const long long* ctr_ptrs, int arrivals, int* status, int sm_count, cudaStream_t stream);

// act[M, F] = silu(x Wg^T) * (x Wu^T), w = [Wg; Wu]; gate_up [M, 2F] optional.  cudaErrorNotSupported: use the plain product.
cudaError_t gemm_swiglu_pair(const void* x, const void* w, void* gate_up, void* act, int M, int F, int K, long long ldx,
                             long long ldw, int* status, int sm_count, cudaStream_t stream);
// out[M, N] = x w^T + bias with the heads of the columns below rot_cols rotated by pos[row], as launch_rope_qkv does.
// cudaErrorNotSupported: use the plain product and that.
cudaError_t gemm_rope_pair(const void* x, const void* w, const void* bias, void* out, const long long* pos, int M, int N, int K,
                           long long ldx, long long ldw, int rot_cols, int head_dim, float theta, int* status, int sm_count,
                           cudaStream_t stream);
cudaError_t gemm_wgrad_scatter_pair(const void* dy, const void* x, int tokens, int n_out, int k_in, long long ld_dy,
                                    long long ld_x, const long long* acc_addrs_host, const long long* ctr_ptrs,
                                    long long acc_offset, int rows_per_rank, int nranks, float scale,
                                    unsigned int* done_slot, int* status, int sm_count, cudaStream_t stream,
                                    int start_rank = 0, bool fixed_order = false);
cudaError_t gemm_swiglu_bwd_pair(const void* dy, const void* w, const void* gate_up, void* dgate_up, int M, int F, int K,
                                 long long lddy, long long ldw, int* status, int sm_count, cudaStream_t stream);
// logits[M, N] = h w^T in bf16 (not written if null) on CTA pairs, with the softmax statistics of logits * inv_temp that the two
// launches below take: row_stats [logits_stat_tiles(N), M, 2], label_logits [M].  cudaErrorNotSupported where a pair does not
// take the product.
int logits_stat_tiles(int N);
bool logits_stats_pay(int M, int N, int K, bool store_logits, int sm_count);   // else the passes over plain logits
cudaError_t gemm_logits_pair(const void* h, const void* w, void* logits, const long long* labels, float* row_stats,
                             float* label_logits, int M, int N, int K, long long ldh, long long ldw, long long ldl, float inv_temp,
                             int* status, int sm_count, cudaStream_t stream);
// as launch_ce_fwd_bwd / launch_token_logprobs
cudaError_t launch_ce_from_stats(void* logits, const long long* labels, const float* loss_scale, const float* row_stats,
                                 const float* label_logits, float* loss, int rows, int vocab, int tiles, long long ignore_index,
                                 cudaStream_t stream, float inv_temp);
cudaError_t launch_logprobs_from_stats(const long long* labels, const float* row_stats, const float* label_logits, float* per_token,
                                       int rows, int tiles, long long ignore_index, cudaStream_t stream, float inv_temp);
cudaError_t gemm_gather_pair(bool dgrad, const void* a, const long long* shard_ptrs, void* w_local, void* out,
                             const void* bias, int M, int w_rows, int w_cols, long long lda, long long ldo,
                             int rows_per_rank, int nranks, unsigned int* group_flags, int* status, int sm_count,
                             cudaStream_t stream, const void* residual = nullptr, long long ldr = 0, int start_rank = 0);

// ---- GEMMs fused with the on-demand primitives ---------------------------------------------------
// dW[n_out, k_in] = dY[tokens, n_out]^T X[tokens, k_in]; row r of dW is added (x scale) into
// accumulator acc_ptrs[r / rows_per_rank] at element acc_offset + (r % rows_per_rank) * k_in.
cudaError_t gemm_wgrad_scatter(const void* dy, const void* x, int tokens, int n_out, int k_in, long long ld_dy,
                               long long ld_x, const long long* acc_ptrs, const long long* ctr_ptrs,
                               long long acc_offset, int rows_per_rank, int nranks, float scale,
                               unsigned int* done_slot, int* status, int sm_count, cudaStream_t stream);
// Same contract, but output boxes go through shared memory and TMA bulk reduce-add into the owners' accumulators.
// acc_addrs_host: HOST array of the accumulators' addresses (tensor maps are built on the host).  Returns
// cudaErrorNotSupported when rows_per_rank is not a multiple of 128 or there are more than 8 owners.
cudaError_t gemm_wgrad_scatter_tma(const void* dy, const void* x, int tokens, int n_out, int k_in, long long ld_dy,
                                   long long ld_x, const long long* acc_addrs_host, const long long* ctr_ptrs,
                                   long long acc_offset, int rows_per_rank, int nranks, float scale,
                                   unsigned int* done_slot, int* status, int sm_count, cudaStream_t stream,
                                   int start_rank = 0, bool fixed_order = false);
// Y[M, N] = X[M, K] W[N, K]^T with rank r holding rows [r * rows_per_rank, ...) of W at shard_ptrs[r];
// w_local [N, K] receives the gathered weight; panel_flags needs ceil(N / 256) words.
cudaError_t gemm_gather_nt(const void* x, const long long* shard_ptrs, void* w_local, void* y, const void* bias,
                           int M, int N, int K, long long ldx, long long ldy, int rows_per_rank, int nranks,
                           int start_rank, unsigned int* panel_flags, int* status, int sm_count,
                           cudaStream_t stream, const void* residual = nullptr, long long ldr = 0);
// dX[M, k_in] = dY[M, n_out] W[n_out, k_in] with W row-sharded as above: the gathered rows are the reduction
// dimension, so the k-loop of every output tile follows the arrival of the 256-row groups (first tile of a CTA)
// and later tiles find the whole weight in w_local.  group_flags needs ceil(n_out / 256) words.
cudaError_t gemm_gather_nn(const void* dy, const long long* shard_ptrs, void* w_local, void* dx, int M, int n_out,
                           int k_in, long long lddy, long long lddx, int rows_per_rank, int nranks,
                           unsigned int* group_flags, int* status, int sm_count, cudaStream_t stream,
                           int start_rank = 0);

// ---- varlen attention ------------------------------------------------------------------------
cudaError_t attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int* cu_seqlens,
                     int num_seqs, int total_tokens, int max_seqlen, int n_q, int n_kv, int head_dim,
                     long long q_stride, long long kv_stride, long long o_stride, float scale, bool causal,
                     int* status, int sm_count, cudaStream_t stream);
// head_dim 128: the forward takes query tiles in pairs, else (and with head_dim 64) one per CTA
bool attn_fwd_pairs(int total_tokens, int num_seqs, int max_seqlen, int n_q, int n_kv, bool causal, int sm_count);
// 2^x as the forward computes it on the FMA pipe, for tests; n is even, both 8-byte aligned
cudaError_t launch_exp2_poly(const float* x, float* y, long long n, cudaStream_t stream);
// CTAs per (key tile, kv head) of the backward; above 1 it needs kv_parts, [parts][2][tokens, n_kv, head_dim] fp32 scratch
int attn_bwd_parts(int total_tokens, int num_seqs, int max_seqlen, int n_q, int n_kv, int head_dim, bool causal, int sm_count);
cudaError_t attn_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse,
                     void* dq, void* dk, void* dv, float* delta, float* dq_acc, float* kv_parts, int parts, const int* cu_seqlens, int num_seqs,
                     int total_tokens, int max_seqlen, int n_q, int n_kv, int head_dim, long long q_stride,
                     long long kv_stride, long long o_stride, long long dq_stride, long long dkv_stride, float scale,
                     bool causal, int* status, int sm_count, cudaStream_t stream,
                     // positions [tokens] by which q and k were rotated (rotary base rope_theta): their gradients are rotated back
                     const long long* rope_pos = nullptr, float rope_theta = 0.f);

}  // namespace odc
