// The decoder's ops: raw kernel entry points, and their differentiable forms as native autograd functions.
//
// A training step of a small model is bound by the host: a Python autograd function costs 15-25 us per direction, the
// kernels behind it 3-10 us.  The native functions cost 3-5 us per direction and run their backward without the
// interpreter lock.
#include "ops.h"

#include <torch/csrc/autograd/custom_function.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace odc_bind {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

constexpr const char* kLayoutNames[3] = {"nt", "nn", "tn"};

// kernels of this package launched by the ops so far (benchmark accounting)
std::atomic<long long> g_launches{0};
void count(int n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

std::tuple<Tensor, Tensor> rmsnorm_fwd(Tensor x, Tensor w, double eps) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.scalar_type() == at::kBFloat16, "rmsnorm: x must be [T,H] bf16");
  TORCH_CHECK(w.scalar_type() == at::kBFloat16 && w.is_contiguous(), "rmsnorm: weight must be bf16");
  auto y = at::empty_like(x);
  auto rstd = at::empty({x.size(0)}, x.options().dtype(at::kFloat));
  check(odc::launch_rmsnorm_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(),
                                static_cast<int>(x.size(0)), static_cast<int>(x.size(1)), static_cast<float>(eps),
                                sm_count(), cur_stream()),
        "rmsnorm_fwd");
  return {y, rstd};
}

// sink (fp32 [H], not with fixed_order): dw is added there and an undefined tensor comes back in its place
std::tuple<Tensor, Tensor> rmsnorm_bwd(Tensor dy, Tensor x, Tensor w, Tensor rstd, bool fixed_order,
                                       c10::optional<Tensor> dres, c10::optional<Tensor> sink) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(dy.is_contiguous() && x.is_contiguous() && dy.sizes() == x.sizes(), "rmsnorm_bwd: contiguous dy, x [T,H]");
  const int rows = static_cast<int>(x.size(0)), cols = static_cast<int>(x.size(1));
  auto dx = at::empty_like(x);
  const int grid = odc::rmsnorm_bwd_grid(rows, sm_count());
  const bool add = sink.has_value();
  if (add)
    TORCH_CHECK(!fixed_order && sink->scalar_type() == at::kFloat && sink->numel() == cols && sink->is_contiguous(),
                "rmsnorm_bwd: sink is fp32 [H]");
  auto dw = add ? *sink : at::empty({cols}, x.options().dtype(at::kFloat));
  Tensor partial;
  float* partial_ptr = nullptr;
  if (fixed_order) {  // per-CTA column sums added up in a fixed order by a second pass (bitwise reproducible)
    partial = at::empty({grid, cols}, x.options().dtype(at::kFloat));
    partial_ptr = partial.data_ptr<float>();
  }
  const void* dres_ptr = nullptr;
  if (dres.has_value()) {
    TORCH_CHECK(dres->is_contiguous() && dres->sizes() == x.sizes() && dres->scalar_type() == at::kBFloat16,
                "rmsnorm_bwd: residual gradient must be contiguous bf16 of x's shape");
    dres_ptr = dres->data_ptr();
  }
  check(odc::launch_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(), dx.data_ptr(),
                                partial_ptr, dw.data_ptr<float>(), rows, cols, grid, cur_stream(), dres_ptr, add),
        "rmsnorm_bwd");
  return {dx, add ? Tensor() : dw};
}

Tensor rope_qkv(Tensor qkv, Tensor pos, int n_q, int n_kv, int head_dim, double theta, bool inverse) {
  c10::cuda::CUDAGuard g(qkv.device());
  odc::bind_device(qkv.get_device());
  pos = pos.contiguous();
  TORCH_CHECK(qkv.dim() == 2 && qkv.is_contiguous() && qkv.scalar_type() == at::kBFloat16, "rope: qkv [T,W] bf16");
  TORCH_CHECK(qkv.size(1) == int64_t(n_q + 2 * n_kv) * head_dim, "rope: width mismatch");
  TORCH_CHECK(pos.scalar_type() == at::kLong && pos.numel() == qkv.size(0), "rope: position_ids int64 [T]");
  TORCH_CHECK(pos.device() == qkv.device(), "rope: position_ids on ", pos.device(), ", qkv on ", qkv.device());
  auto out = at::empty_like(qkv);
  check(odc::launch_rope_qkv(qkv.data_ptr(), out.data_ptr(), reinterpret_cast<const long long*>(pos.data_ptr<int64_t>()),
                             static_cast<int>(qkv.size(0)), n_q, n_kv, head_dim, static_cast<float>(theta), inverse,
                             cur_stream()),
        "rope_qkv");
  return out;
}

Tensor swiglu_fwd(Tensor gu) {
  c10::cuda::CUDAGuard g(gu.device());
  odc::bind_device(gu.get_device());
  TORCH_CHECK(gu.is_contiguous() && gu.scalar_type() == at::kBFloat16, "swiglu: bf16 contiguous");
  const int f = static_cast<int>(gu.size(-1) / 2);
  auto sizes = gu.sizes().vec();
  sizes.back() = f;
  auto out = at::empty(sizes, gu.options());
  check(odc::launch_swiglu_fwd(gu.data_ptr(), out.data_ptr(), gu.numel() / (2 * f), f, sm_count(), cur_stream()),
        "swiglu_fwd");
  return out;
}

Tensor swiglu_bwd(Tensor dy, Tensor gu) {
  c10::cuda::CUDAGuard g(gu.device());
  odc::bind_device(gu.get_device());
  const int f = static_cast<int>(gu.size(-1) / 2);
  auto out = at::empty_like(gu);
  check(odc::launch_swiglu_bwd(dy.data_ptr(), gu.data_ptr(), out.data_ptr(), gu.numel() / (2 * f), f, sm_count(),
                               cur_stream()),
        "swiglu_bwd");
  return out;
}

void ce_fwd_bwd(Tensor logits, Tensor labels, c10::optional<Tensor> loss_scale, Tensor loss, int64_t ignore_index,
                double inv_temp) {
  c10::cuda::CUDAGuard g(logits.device());
  odc::bind_device(logits.get_device());
  TORCH_CHECK(logits.dim() == 2 && logits.is_contiguous() && logits.scalar_type() == at::kBFloat16, "ce: logits bf16");
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous(), "ce: labels int64");
  const float* ls = nullptr;
  if (loss_scale.has_value()) {
    TORCH_CHECK(loss_scale->scalar_type() == at::kFloat && loss_scale->is_contiguous(), "ce: loss_scale fp32");
    ls = loss_scale->data_ptr<float>();
  }
  check(odc::launch_ce_fwd_bwd(logits.data_ptr(), reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()), ls,
                               loss.data_ptr<float>(), static_cast<int>(logits.size(0)),
                               static_cast<int>(logits.size(1)), ignore_index, cur_stream(), static_cast<float>(inv_temp)),
        "ce_fwd_bwd");
}

void token_logprobs(Tensor logits, Tensor labels, Tensor out, int64_t ignore_index, double inv_temp) {
  c10::cuda::CUDAGuard g(logits.device());
  odc::bind_device(logits.get_device());
  TORCH_CHECK(logits.dim() == 2 && logits.is_contiguous() && logits.scalar_type() == at::kBFloat16, "token_logprobs: logits bf16");
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == logits.size(0),
              "token_logprobs: one int64 label per row");
  TORCH_CHECK(out.scalar_type() == at::kFloat && out.is_contiguous() && out.numel() == logits.size(0) && out.is_cuda(),
              "token_logprobs: one fp32 output per row");
  check(odc::launch_token_logprobs(logits.data_ptr(), reinterpret_cast<const long long*>(labels.data_ptr<int64_t>()),
                                   out.data_ptr<float>(), static_cast<int>(logits.size(0)),
                                   static_cast<int>(logits.size(1)), ignore_index, cur_stream(), static_cast<float>(inv_temp)),
        "token_logprobs");
}

void adamw_step(Tensor p, Tensor g, Tensor m, Tensor v, c10::optional<Tensor> p_lowp, double lr, double beta1,
                double beta2, double eps, double wd, int64_t step, double grad_scale) {
  c10::cuda::CUDAGuard guard(p.device());
  odc::bind_device(p.get_device());
  TORCH_CHECK(p.scalar_type() == at::kFloat && m.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat,
              "adamw: fp32 master state");
  TORCH_CHECK(p.is_contiguous() && g.is_contiguous() && m.is_contiguous() && v.is_contiguous(), "adamw: contiguous");
  void* lp = nullptr;
  if (p_lowp.has_value()) {
    TORCH_CHECK(p_lowp->scalar_type() == at::kBFloat16 && p_lowp->numel() == p.numel(), "adamw: bf16 replica");
    lp = p_lowp->data_ptr();
  }
  const float bc1 = 1.f - std::pow(static_cast<float>(beta1), static_cast<float>(step));
  const float bc2 = 1.f - std::pow(static_cast<float>(beta2), static_cast<float>(step));
  check(odc::launch_adamw(p.data_ptr<float>(), g.data_ptr(), kind_of(g.scalar_type()), m.data_ptr<float>(),
                          v.data_ptr<float>(), lp, static_cast<size_t>(p.numel()), static_cast<float>(lr),
                          static_cast<float>(beta1), static_cast<float>(beta2), static_cast<float>(eps),
                          static_cast<float>(wd), bc1, bc2, static_cast<float>(grad_scale), cur_stream()),
        "adamw");
}

void cast_f32_to_bf16(Tensor in, Tensor out) {
  c10::cuda::CUDAGuard g(in.device());
  odc::bind_device(in.get_device());
  TORCH_CHECK(in.scalar_type() == at::kFloat && out.scalar_type() == at::kBFloat16 && in.numel() == out.numel() &&
                  in.is_contiguous() && out.is_contiguous(), "cast: fp32 -> bf16, same numel, contiguous");
  check(odc::launch_cast_f32_to_bf16(in.data_ptr<float>(), out.data_ptr(), static_cast<size_t>(in.numel()), sm_count(),
                                     cur_stream()),
        "cast");
}

void sumsq(Tensor x, Tensor out) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.is_contiguous() && out.scalar_type() == at::kFloat, "sumsq: contiguous input, fp32 output");
  check(odc::launch_sumsq(x.data_ptr(), kind_of(x.scalar_type()), static_cast<size_t>(x.numel()), out.data_ptr<float>(),
                          sm_count(), cur_stream()),
        "sumsq");
}

Tensor kernel_status() {
  int dev = 0;
  cudaGetDevice(&dev);
  return device_status(dev);
}

// The host read an error there.  A launch that gave up may have left the counters of its stream's groups half way: the next ones get
// others; nothing waits for what other streams have in flight.
void clear_kernel_status() {
  kernel_status().zero_();
  odc::gemm_group_new_words();
}

bool capturing() {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  check(cudaStreamIsCapturing(cur_stream(), &capture), "capture");
  return capture != cudaStreamCaptureStatusNone;
}

// the counters of the current stream's groups, or null where a launch has to bring its own
unsigned int* group_words() { return capturing() ? nullptr : odc::gemm_group_words(cur_stream()); }

// ODC_GEMM=cublas: library products, to measure the hand-written kernels against (read at every call)
bool library_gemm() {
  const char* e = std::getenv("ODC_GEMM");
  return e != nullptr && std::strcmp(e, "cublas") == 0;
}

enum Layout : int { kNT = 0, kNN = 1, kTN = 2 };  // C = A B^T (forward), A B (input gradient), A^T B (weight gradient)

void gemm_into(const Tensor& a, const Tensor& b, const Tensor& c, int lay, const Tensor& bias = {}, bool accumulate = false,
               const Tensor& residual = {}, int pair = -1) {
  c10::cuda::CUDAGuard g(a.device());
  odc::bind_device(a.get_device());
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && c.dim() == 2, "gemm: 2-D operands");
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "gemm: bf16 inputs");
  TORCH_CHECK(a.stride(1) == 1 && b.stride(1) == 1 && c.stride(1) == 1, "gemm: innermost stride must be 1");
  const int K = lay == kTN ? a.size(0) : a.size(1), M = lay == kTN ? a.size(1) : a.size(0);
  const int N = lay == kNT ? b.size(0) : b.size(1);
  TORCH_CHECK((lay == kNT ? b.size(1) : b.size(0)) == K, "gemm ", kLayoutNames[lay], ": K mismatch");
  TORCH_CHECK(c.size(0) == M && c.size(1) == N, "gemm: output shape mismatch");
  const void* bias_ptr = nullptr;
  if (bias.defined()) {
    TORCH_CHECK(bias.scalar_type() == at::kBFloat16 && bias.numel() == N && bias.is_contiguous(), "gemm: bias bf16 [N]");
    bias_ptr = bias.data_ptr();
  }
  const void* res_ptr = nullptr;
  long long ldr = 0;
  if (residual.defined()) {
    TORCH_CHECK(residual.scalar_type() == at::kBFloat16 && residual.dim() == 2 && residual.size(0) == M &&
                    residual.size(1) == N && residual.stride(1) == 1, "gemm: residual bf16 [M,N]");
    res_ptr = residual.data_ptr();
    ldr = residual.stride(0);
  }
  Tensor parts;  // few tiles and a long reduction: scratch for the partial products
  if (pair < 0 && !accumulate && odc::gemm_pairs_enabled()) {
    const size_t bytes = odc::gemm_plan(M, N, K, kind_of(c.scalar_type()), sm_count()).scratch_bytes;
    if (bytes > 0) {
      parts = at::empty({static_cast<int64_t>(bytes / sizeof(float))}, a.options().dtype(at::kFloat));
      count();
    }
  }
  cudaError_t e = odc::gemm_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), kind_of(c.scalar_type()), bias_ptr, M, N, K,
                                 lay, accumulate, a.stride(0), b.stride(0), c.stride(0),
                                 device_status(a.get_device()).data_ptr<int>(), sm_count(), cur_stream(), res_ptr, ldr,
                                 pair, parts.defined() ? parts.data_ptr<float>() : nullptr);
  TORCH_CHECK(e == cudaSuccess, "gemm(", kLayoutNames[lay], ") M=", M, " N=", N, " K=", K, " lda=", a.stride(0), " ldb=",
              b.stride(0), " ldc=", c.stride(0), " align(a,b,c)=", reinterpret_cast<uintptr_t>(a.data_ptr()) % 16, ",",
              reinterpret_cast<uintptr_t>(b.data_ptr()) % 16, ",", reinterpret_cast<uintptr_t>(c.data_ptr()) % 16, ": ",
              cudaGetErrorString(e));
}

void gemm(Tensor a, Tensor b, Tensor c, const std::string& layout, c10::optional<Tensor> bias, bool accumulate,
          c10::optional<Tensor> residual, int pair) {
  int lay = 0;
  while (lay < 3 && layout != kLayoutNames[lay]) ++lay;
  TORCH_CHECK(lay < 3, "gemm: unknown layout ", layout);
  gemm_into(a, b, c, lay, bias.value_or(Tensor()), accumulate, residual.value_or(Tensor()), pair);
}

// the product the ops use: own kernel, or the library when asked for
void product_into(const Tensor& a, const Tensor& b, const Tensor& c, int lay, const Tensor& bias = {}, bool accumulate = false,
                  const Tensor& residual = {}) {
  if (library_gemm()) {
    Tensor r = at::matmul(lay == kTN ? a.t() : a, lay == kNT ? b.t() : b);
    if (bias.defined()) r = r + bias;
    if (residual.defined()) r = r + residual;
    if (accumulate) c.add_(r.to(c.scalar_type())); else c.copy_(r);
    return;
  }
  gemm_into(a, b, c, lay, bias, accumulate, residual);
  count();
}
Tensor product(const Tensor& a, const Tensor& b, int lay, const Tensor& bias = {}, const Tensor& residual = {},
               c10::optional<at::ScalarType> dtype = c10::nullopt) {
  auto c = at::empty({lay == kTN ? a.size(1) : a.size(0), lay == kNT ? b.size(0) : b.size(1)},
                     dtype ? a.options().dtype(*dtype) : a.options());
  product_into(a, b, c, lay, bias, false, residual);
  return c;
}

// Products none of which reads what another writes: one launch where the kernel takes them together, else one by one.
struct Product {
  Tensor a, b, c;
  int lay;
  bool accumulate = false;
  double scale = 1.0;    // group_into only: of the result
  Tensor times;          // group_into only: a further factor, one fp32 value on the device
  Tensor addend;         // group_into only: contiguous fp32 that joins a bf16 result before it is rounded
  bool any_order = false;   // group_into only: an accumulating product may add its parts in any order
  bool whole = false;       // group_into only: a bf16 product is one sum
};
bool fixed_order_asked() {
  const char* e = std::getenv("ODC_DETERMINISTIC");
  return at::globalContext().deterministicAlgorithms() ||
         (e != nullptr && *e != 0 && std::strcmp(e, "0") != 0 && std::strcmp(e, "false") != 0);
}
// arrivals > 0: that many are reported to the counter behind ctr_table (one entry) when the results are in memory
bool group_into(const std::vector<Product>& products, const Tensor& ctr_table = {}, int arrivals = 0) {
  const int n = static_cast<int>(products.size());
  if (n < 1 || n > odc::kMaxGroupProducts || library_gemm() || !odc::gemm_pairs_enabled()) return false;
  odc::GemmProduct g[odc::kMaxGroupProducts];
  const bool fixed = fixed_order_asked();
  for (int i = 0; i < n; ++i) {
    const auto& [a, b, c, lay, accumulate, scale, times, addend, any_order, whole] = products[i];
    if (a.dim() != 2 || b.dim() != 2 || c.dim() != 2 || a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16 ||
        (c.scalar_type() != at::kBFloat16 && c.scalar_type() != at::kFloat) || a.stride(1) != 1 || b.stride(1) != 1 || c.stride(1) != 1)
      return false;
    const int64_t K = lay == kTN ? a.size(0) : a.size(1), M = lay == kTN ? a.size(1) : a.size(0), N = lay == kNT ? b.size(0) : b.size(1);
    if ((lay == kNT ? b.size(1) : b.size(0)) != K || c.size(0) != M || c.size(1) != N) return false;
    g[i] = odc::GemmProduct{a.data_ptr(), b.data_ptr(), c.data_ptr(), kind_of(c.scalar_type()), static_cast<int>(M), static_cast<int>(N),
                            static_cast<int>(K), lay, accumulate,
                            c.scalar_type() == at::kFloat ? fixed || !any_order : whole, a.stride(0), b.stride(0), c.stride(0), static_cast<float>(scale),
                            times.defined() ? times.data_ptr<float>() : nullptr, addend.defined() ? addend.data_ptr<float>() : nullptr};
  }
  const Tensor& a = products[0].a;
  c10::cuda::CUDAGuard guard(a.device());
  odc::bind_device(a.get_device());
  const odc::GemmGroupPlan plan = odc::gemm_group_plan(g, n, sm_count());
  if (!plan.taken) return false;
  Tensor scratch;
  if (plan.scratch_bytes > 0)
    scratch = at::empty({static_cast<int64_t>(plan.scratch_bytes / sizeof(float))}, a.options().dtype(at::kFloat));
  unsigned int* words = group_words();
  Tensor own;
  if (words == nullptr) {   // a graph's are cleared at each replay
    own = at::zeros({odc::kGroupLaunchWords}, a.options().dtype(at::kInt));
    words = reinterpret_cast<unsigned int*>(own.data_ptr<int>());
  }
  const cudaError_t e = odc::gemm_group(g, n, plan, scratch.defined() ? scratch.data_ptr<float>() : nullptr, words,
                                        ctr_table.defined() ? reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()) : nullptr,
                                        arrivals, device_status(a.get_device()).data_ptr<int>(), sm_count(), cur_stream());
  if (e == cudaErrorNotSupported) return false;
  check(e, "group of products");
  count();
  return true;
}
void products_into(const std::vector<Product>& products) {
  if (group_into(products)) return;
  for (const auto& p : products) product_into(p.a, p.b, p.c, p.lay, {}, p.accumulate);
}
Tensor product_out(const Tensor& a, const Tensor& b, int lay, c10::optional<at::ScalarType> dtype = c10::nullopt) {
  return at::empty({lay == kTN ? a.size(1) : a.size(0), lay == kNT ? b.size(0) : b.size(1)}, dtype ? a.options().dtype(*dtype) : a.options());
}
// the input gradient and the weight gradient of y = x w^T, what is wanted of them
std::tuple<Tensor, Tensor> linear_grads(const Tensor& dy2, const Tensor& x2, const Tensor& w, bool need_dx, bool need_dw) {
  Tensor dx, dw;
  std::vector<Product> todo;
  if (need_dx) todo.push_back({dy2, w, dx = product_out(dy2, w, kNN), kNN});
  if (need_dw) todo.push_back({dy2, x2, dw = product_out(dy2, x2, kTN, w.scalar_type()), kTN});
  products_into(todo);
  return {dx, dw};
}

std::tuple<Tensor, Tensor> attn_fwd(Tensor q, Tensor k, Tensor v, Tensor cu_seqlens, int max_seqlen, bool causal,
                                    double scale) {
  c10::cuda::CUDAGuard g(q.device());
  odc::bind_device(q.get_device());
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, "attention: q/k/v are [T, H, D]");
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16,
              "attention: bf16 inputs");
  const int T = q.size(0), hq = q.size(1), d = q.size(2), hkv = k.size(1);
  TORCH_CHECK(q.stride(2) == 1 && q.stride(1) == d && k.stride(2) == 1 && k.stride(1) == d && v.stride(2) == 1 &&
                  v.stride(1) == d, "attention: heads must be packed within a token");
  TORCH_CHECK(k.stride(0) == v.stride(0), "attention: k and v must share a row stride");
  TORCH_CHECK(cu_seqlens.scalar_type() == at::kInt && cu_seqlens.is_contiguous(), "attention: cu_seqlens int32");
  TORCH_CHECK(cu_seqlens.device() == q.device(), "attention: cu_seqlens on ", cu_seqlens.device(), ", q on ", q.device());
  auto o = at::empty({T, hq, d}, q.options());
  auto lse = at::empty({hq, T}, q.options().dtype(at::kFloat));
  check(odc::attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr<float>(),
                      cu_seqlens.data_ptr<int>(), static_cast<int>(cu_seqlens.numel() - 1), T, max_seqlen, hq, hkv, d,
                      q.stride(0), k.stride(0), o.stride(0), static_cast<float>(scale), causal,
                      device_status(q.get_device()).data_ptr<int>(), sm_count(), cur_stream()),
        "attn_fwd");
  return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> attn_bwd(Tensor dout, Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse,
                                                    Tensor cu_seqlens, int max_seqlen, bool causal, double scale,
                                                    bool fused_qkv, const Tensor& rope_pos = {}, double rope_theta = 0) {
  c10::cuda::CUDAGuard g(q.device());
  odc::bind_device(q.get_device());
  const int T = q.size(0), hq = q.size(1), d = q.size(2), hkv = k.size(1);
  TORCH_CHECK(dout.is_contiguous() && dout.scalar_type() == at::kBFloat16, "attention bwd: dout contiguous bf16");
  TORCH_CHECK(o.stride(2) == 1 && o.stride(1) == d, "attention bwd: o heads packed");
  TORCH_CHECK(q.stride(2) == 1 && q.stride(1) == d && k.stride(2) == 1 && k.stride(1) == d && v.stride(2) == 1 &&
                  v.stride(1) == d && k.stride(0) == v.stride(0), "attention bwd: q/k/v layout");
  Tensor dq, dk, dv, dqkv;
  if (fused_qkv) {
    // one [T, (hq + 2 hkv) d] gradient; dq/dk/dv are column views of it, so slicing costs nothing in autograd
    dqkv = at::empty({T, int64_t(hq + 2 * hkv) * d}, q.options());
    dq = dqkv.narrow(1, 0, int64_t(hq) * d).view({T, hq, d});
    dk = dqkv.narrow(1, int64_t(hq) * d, int64_t(hkv) * d).view({T, hkv, d});
    dv = dqkv.narrow(1, int64_t(hq + hkv) * d, int64_t(hkv) * d).view({T, hkv, d});
  } else {
    dq = at::empty({T, hq, d}, q.options());
    dk = at::empty({T, hkv, d}, q.options());
    dv = at::empty({T, hkv, d}, q.options());
  }
  auto delta = at::empty({hq, T}, q.options().dtype(at::kFloat));
  auto dq_acc = at::empty({T, hq, d}, q.options().dtype(at::kFloat));
  const int n_seqs = static_cast<int>(cu_seqlens.numel() - 1);
  const int n_parts = hkv > 0 && hq % hkv == 0 ? odc::attn_bwd_parts(T, n_seqs, max_seqlen, hq, hkv, d, causal, sm_count()) : 1;
  Tensor kv_parts;
  if (n_parts > 1) kv_parts = at::empty({n_parts, 2, T, hkv, d}, q.options().dtype(at::kFloat));
  check(odc::attn_bwd(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr<float>(),
                      dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), delta.data_ptr<float>(), dq_acc.data_ptr<float>(),
                      n_parts > 1 ? kv_parts.data_ptr<float>() : nullptr, n_parts, cu_seqlens.data_ptr<int>(), n_seqs, T, max_seqlen, hq, hkv, d,
                      q.stride(0), k.stride(0), o.stride(0), dq.stride(0), dk.stride(0), static_cast<float>(scale),
                      causal, device_status(q.get_device()).data_ptr<int>(), sm_count(), cur_stream(),
                      rope_pos.defined() ? reinterpret_cast<const long long*>(rope_pos.data_ptr<int64_t>()) : nullptr,
                      static_cast<float>(rope_theta)),
        "attn_bwd");
  return {dq, dk, dv, fused_qkv ? dqkv : dq};  // 4th: the fused gradient when requested
}

Tensor exp2_poly(Tensor x) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.is_contiguous() && x.numel() % 2 == 0 &&
                  reinterpret_cast<uintptr_t>(x.data_ptr()) % 8 == 0, "exp2_poly: pairs of fp32 values, contiguous");
  auto y = at::empty_like(x);
  check(odc::launch_exp2_poly(x.data_ptr<float>(), y.data_ptr<float>(), x.numel(), cur_stream()), "exp2_poly");
  return y;
}

// ------------------------------------------------------------------------------------------------ differentiable ops
bool env_on(const char* name) {
  const char* e = std::getenv(name);
  return e != nullptr && *e != 0 && std::strcmp(e, "0") != 0 && std::strcmp(e, "false") != 0;
}
bool wants_grad(const Tensor& t) { return at::GradMode::is_enabled() && t.defined() && t.requires_grad(); }
// sum over the rows of a gradient (the bias gradient), fp32 inside
Tensor column_sum(const Tensor& x) {
  c10::cuda::CUDAGuard g(x.device());
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous(), "column_sum: contiguous [T,N]");
  // the kernel reads bf16, 16 bytes at a time; gradients of library products come in other types and widths too
  if (x.scalar_type() != at::kBFloat16 || x.size(1) % 8 != 0 || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0)
    return x.sum(0, false, at::kFloat).to(x.scalar_type());
  auto out = at::empty({x.size(1)}, x.options());
  check(odc::launch_column_sum(x.data_ptr(), out.data_ptr(), nullptr, x.size(0), static_cast<int>(x.size(1)), cur_stream()),
        "column_sum");
  count();
  return out;
}

// bf16(in * *scale) for a one-element scale on the device; in is fp32 or bf16
Tensor scale_to_bf16(Tensor in, Tensor scale) {
  c10::cuda::CUDAGuard g(in.device());
  TORCH_CHECK(in.is_contiguous() && scale.numel() == 1 && scale.is_cuda(), "scale_to_bf16: contiguous input, one device value");
  scale = scale.to(at::kFloat);
  auto out = at::empty(in.sizes(), in.options().dtype(at::kBFloat16));
  check(odc::launch_scale_to_bf16(in.data_ptr(), kind_of(in.scalar_type()), out.data_ptr(), scale.data_ptr<float>(),
                                  static_cast<size_t>(in.numel()), sm_count(), cur_stream()),
        "scale_to_bf16");
  count();
  return out;
}

Tensor rows2d(const Tensor& x) { return x.dim() == 2 ? x : x.reshape({-1, x.size(-1)}); }
Tensor like(const Tensor& y2, const Tensor& x, int64_t last) {
  if (x.dim() == 2) return y2;
  auto sizes = x.sizes().vec();
  sizes.back() = last;
  return y2.view(sizes);
}

struct LinearFn : Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w, c10::optional<Tensor> bias, c10::optional<Tensor> residual,
                        bool need_dx, bool need_dw, bool need_db, bool need_dres) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["need"] = static_cast<int64_t>(need_dx | need_dw << 1 | need_db << 2 | need_dres << 3);
    Tensor res;
    if (residual.has_value()) res = rows2d(*residual);  // added in the GEMM epilogue
    return like(product(rows2d(x), w, kNT, bias.value_or(Tensor()), res), x, w.size(0));
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &dy = grads[0];
    const int64_t need = ctx->saved_data["need"].toInt();
    const Tensor dy2 = rows2d(dy).contiguous();
    Tensor db;
    auto [dx, dw] = linear_grads(dy2, rows2d(x), w, need & 1, need & 2);
    if (dx.defined()) dx = dx.view(x.sizes());
    if (need & 4) db = column_sum(dy2);
    return {dx, dw, db, (need & 8) ? dy : Tensor(), {}, {}, {}, {}};
  }
};

Tensor linear(Tensor x, Tensor w, c10::optional<Tensor> bias, c10::optional<Tensor> residual) {
  const bool db = bias.has_value() && wants_grad(*bias), dres = residual.has_value() && wants_grad(*residual);
  return LinearFn::apply(x, w, bias, residual, wants_grad(x), wants_grad(w), db, dres);
}

// RMSNorm; with_residual also returns x, and backward forms d(norm) + d(residual) in one pass over the activation
// instead of leaving a separate addition to autograd.  `sink` (fp32 [H]): the weight's gradient is added there by the
// kernel and the weight itself gets none (engines that keep all small parameters in one flat accumulator).
//
// dx, and the weight's gradient unless it went to the sink
std::tuple<Tensor, Tensor> norm_grads(const Tensor& dy2, const Tensor& x2, const Tensor& w, const Tensor& rstd,
                                      const c10::optional<Tensor>& dres, const c10::optional<Tensor>& sink) {
  const bool fixed = env_on("ODC_DETERMINISTIC");  // fixed-order column sums instead of in-kernel atomics
  auto [dx, dw] = rmsnorm_bwd(dy2, x2, w, rstd, fixed, dres, fixed ? c10::nullopt : sink);
  count(fixed ? 2 : 1);
  if (sink.has_value()) {
    if (fixed) sink->add_(dw);
    dw = Tensor();
  } else if (dw.scalar_type() != w.scalar_type()) {
    dw = dw.to(w.scalar_type());
  }
  return {dx, dw};
}

struct RMSNormFn : Function<RMSNormFn> {
  static variable_list forward(AutogradContext* ctx, Tensor x, Tensor w, double eps, bool with_residual,
                               c10::optional<Tensor> sink) {
    const Tensor x2 = rows2d(x);
    auto [y, rstd] = rmsnorm_fwd(x2, w, eps);
    count();
    ctx->save_for_backward({x2, w, rstd});
    if (sink.has_value()) ctx->saved_data["sink"] = *sink;
    ctx->saved_data["residual"] = with_residual;
    ctx->saved_data["sizes"] = x.sizes().vec();
    if (x.dim() != 2) y = y.view(x.sizes());
    if (!with_residual) return {y};
    return {y, x.view_as(x)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1], &rstd = saved[2];
    const Tensor dy2 = rows2d(grads[0]).contiguous();
    c10::optional<Tensor> dres;
    if (ctx->saved_data["residual"].toBool() && grads[1].defined()) dres = rows2d(grads[1]).contiguous();
    auto it = ctx->saved_data.find("sink");
    c10::optional<Tensor> sink;
    if (it != ctx->saved_data.end()) sink = it->second.toTensor();
    auto [dx, dw] = norm_grads(dy2, x2, w, rstd, dres, sink);
    return {dx.view(ctx->saved_data["sizes"].toIntVector()), dw, {}, {}, {}};
  }
};

Tensor rms_norm(Tensor x, Tensor w, double eps, c10::optional<Tensor> sink) {
  return RMSNormFn::apply(x.contiguous(), w, eps, false, sink)[0];
}
std::tuple<Tensor, Tensor> rms_norm_residual(Tensor x, Tensor w, double eps, c10::optional<Tensor> sink) {
  auto out = RMSNormFn::apply(x.contiguous(), w, eps, true, sink);
  return {out[0], out[1]};
}

// rotary embedding of the q and k heads of a fused [T, (Hq+2Hkv)*D] projection; v passes through
struct RopeFn : Function<RopeFn> {
  static Tensor forward(AutogradContext* ctx, Tensor qkv, Tensor pos, int64_t n_q, int64_t n_kv, int64_t d, double theta) {
    ctx->save_for_backward({pos});
    ctx->saved_data["cfg"] = std::vector<int64_t>{n_q, n_kv, d};
    ctx->saved_data["theta"] = theta;
    auto out = rope_qkv(qkv, pos, n_q, n_kv, d, theta, false);
    count();
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor pos = ctx->get_saved_variables()[0];
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    auto d = rope_qkv(grads[0].contiguous(), pos, cfg[0], cfg[1], cfg[2], ctx->saved_data["theta"].toDouble(), true);
    count();
    return {d, {}, {}, {}, {}, {}};
  }
};
Tensor rope(Tensor qkv, Tensor pos, int64_t n_q, int64_t n_kv, int64_t d, double theta) {
  return RopeFn::apply(qkv, pos, n_q, n_kv, d, theta);
}

struct SwiGLUFn : Function<SwiGLUFn> {
  static Tensor forward(AutogradContext* ctx, Tensor gate_up) {
    ctx->save_for_backward({gate_up});
    count();
    return swiglu_fwd(gate_up);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor gate_up = ctx->get_saved_variables()[0];
    count();
    return {swiglu_bwd(grads[0].contiguous(), gate_up)};
  }
};
Tensor swiglu(Tensor gate_up) { return SwiGLUFn::apply(gate_up.contiguous()); }

// rope(x w^T + bias): rotated in the epilogue of the product where that kernel takes the shape
Tensor linear_rope(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& pos, int64_t n_q, int64_t n_kv, int64_t d,
                   double theta) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && w.size(0) == (n_q + 2 * n_kv) * d, "linear_rope: x [T,K], w [(Hq+2Hkv)*D,K]");
  TORCH_CHECK(pos.scalar_type() == at::kLong && pos.is_contiguous() && pos.numel() == x.size(0), "linear_rope: position_ids int64 [T]");
  TORCH_CHECK(!bias.defined() || bias.numel() == w.size(0), "linear_rope: bias [(Hq+2Hkv)*D]");
  TORCH_CHECK(pos.device() == x.device(), "linear_rope: position_ids on ", pos.device(), ", x on ", x.device());
  if (odc::gemm_pairs_enabled() && !library_gemm() && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
      x.stride(1) == 1 && w.stride(1) == 1 && (!bias.defined() || (bias.scalar_type() == at::kBFloat16 && bias.is_contiguous()))) {
    auto out = at::empty({x.size(0), w.size(0)}, x.options());
    const cudaError_t e = odc::gemm_rope_pair(
        x.data_ptr(), w.data_ptr(), bias.defined() ? bias.data_ptr() : nullptr, out.data_ptr(),
        reinterpret_cast<const long long*>(pos.data_ptr<int64_t>()), static_cast<int>(x.size(0)), static_cast<int>(w.size(0)),
        static_cast<int>(x.size(1)), x.stride(0), w.stride(0), static_cast<int>((n_q + n_kv) * d), static_cast<int>(d),
        static_cast<float>(theta), device_status(x.get_device()).data_ptr<int>(), sm_count(), cur_stream());
    if (e != cudaErrorNotSupported) {
      check(e, "linear_rope");
      count();
      return out;
    }
  }
  const Tensor qkv = product(x, w, kNT, bias);
  count();
  return rope_qkv(qkv, pos, n_q, n_kv, d, theta, false);
}

// swiglu(x w^T) for w = [gate; up]: the activation is formed in the epilogue of the product where that kernel takes the
// shape.  gate_up is only written when a gradient will need it.
std::tuple<Tensor, Tensor> linear_swiglu_fwd(const Tensor& x, const Tensor& w, bool need_gate_up) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && w.size(0) % 2 == 0, "linear_swiglu: x [T,K], w [2F,K]");
  TORCH_CHECK(x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16, "linear_swiglu: bf16 inputs");
  TORCH_CHECK(x.stride(1) == 1 && w.stride(1) == 1, "linear_swiglu: innermost stride must be 1");
  const int64_t T = x.size(0), F = w.size(0) / 2;
  if (odc::gemm_pairs_enabled() && !library_gemm()) {
    Tensor gate_up;
    if (need_gate_up) gate_up = at::empty({T, 2 * F}, x.options());
    auto act = at::empty({T, F}, x.options());
    const cudaError_t e = odc::gemm_swiglu_pair(x.data_ptr(), w.data_ptr(), need_gate_up ? gate_up.data_ptr() : nullptr,
                                                act.data_ptr(), static_cast<int>(T), static_cast<int>(F),
                                                static_cast<int>(x.size(1)), x.stride(0), w.stride(0),
                                                device_status(x.get_device()).data_ptr<int>(), sm_count(), cur_stream());
    if (e != cudaErrorNotSupported) {
      check(e, "linear_swiglu");
      count();
      return {act, gate_up};
    }
  }
  const Tensor gate_up = product(x, w, kNT);
  count();
  return {swiglu_fwd(gate_up), gate_up};
}

struct LinearSwigluFn : Function<LinearSwigluFn> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w, bool need_dx, bool need_dw) {
    auto [act, gate_up] = linear_swiglu_fwd(rows2d(x), w, need_dx || need_dw);
    ctx->saved_data["need"] = static_cast<int64_t>(need_dx | need_dw << 1);
    if (need_dx || need_dw) ctx->save_for_backward({x, w, gate_up});
    return like(act, x, w.size(0) / 2);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const int64_t need = ctx->saved_data["need"].toInt();
    const Tensor d = swiglu_bwd(rows2d(grads[0]).contiguous(), saved[2]);
    count();
    auto [dx, dw] = linear_grads(d, rows2d(x), w, need & 1, need & 2);
    if (dx.defined()) dx = dx.view(x.sizes());
    return {dx, dw, {}, {}};
  }
};
Tensor linear_swiglu(Tensor x, Tensor w) { return LinearSwigluFn::apply(x, w, wants_grad(x), wants_grad(w)); }

// gradient of gate_up [T, 2F] for y = swiglu(gate_up) w^T, w [H, F]: formed in the epilogue of the product dy w where that
// kernel takes the shape
Tensor swiglu_product_bwd(const Tensor& dy, const Tensor& w, const Tensor& gate_up) {
  c10::cuda::CUDAGuard g(dy.device());
  odc::bind_device(dy.get_device());
  TORCH_CHECK(dy.dim() == 2 && w.dim() == 2 && gate_up.dim() == 2 && dy.size(1) == w.size(0) && gate_up.size(0) == dy.size(0) &&
                  gate_up.size(1) == 2 * w.size(1), "swiglu_product_bwd: dy [T,H], w [H,F], gate_up [T,2F]");
  if (odc::gemm_pairs_enabled() && !library_gemm() && dy.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
      gate_up.scalar_type() == at::kBFloat16 && gate_up.is_contiguous() && dy.stride(1) == 1 && w.stride(1) == 1) {
    auto out = at::empty_like(gate_up);
    const cudaError_t e = odc::gemm_swiglu_bwd_pair(dy.data_ptr(), w.data_ptr(), gate_up.data_ptr(), out.data_ptr(),
                                                    static_cast<int>(dy.size(0)), static_cast<int>(w.size(1)),
                                                    static_cast<int>(dy.size(1)), dy.stride(0), w.stride(0),
                                                    device_status(dy.get_device()).data_ptr<int>(), sm_count(), cur_stream());
    if (e != cudaErrorNotSupported) {
      check(e, "swiglu_product_bwd");
      count();
      return out;
    }
  }
  const Tensor d = product(dy, w, kNN);
  count();
  return swiglu_bwd(d, gate_up);
}

// swiglu(x w_gate_up^T) w_down^T + residual as one function, so that the activations' gradient stays inside a product
struct MlpFn : Function<MlpFn> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w_gate_up, Tensor w_down, c10::optional<Tensor> residual, bool need_dx,
                        bool need_dgu, bool need_dd, bool need_dres) {
    const Tensor x2 = rows2d(x);
    auto [act, gate_up] = linear_swiglu_fwd(x2, w_gate_up, need_dx || need_dgu);
    Tensor res;
    if (residual.has_value()) res = rows2d(*residual);
    const Tensor y = product(act, w_down, kNT, {}, res);
    ctx->saved_data["need"] = static_cast<int64_t>(need_dx | need_dgu << 1 | need_dd << 2 | need_dres << 3);
    if (!(need_dx || need_dgu)) gate_up = Tensor();
    if (!need_dd) act = Tensor();
    ctx->save_for_backward({x, w_gate_up, w_down, gate_up, act});
    return like(y, x, w_down.size(0));
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &w_gate_up = s[1], &w_down = s[2];
    const int64_t need = ctx->saved_data["need"].toInt();
    const Tensor dy2 = rows2d(grads[0]).contiguous();
    Tensor d, dx, dgu, dd;
    if (need & 3) d = swiglu_product_bwd(dy2, w_down, s[3]);
    std::vector<Product> todo;
    if (need & 1) todo.push_back({d, w_gate_up, dx = product_out(d, w_gate_up, kNN), kNN});
    if (need & 2) todo.push_back({d, rows2d(x), dgu = product_out(d, rows2d(x), kTN, w_gate_up.scalar_type()), kTN});
    if (need & 4) todo.push_back({dy2, s[4], dd = product_out(dy2, s[4], kTN, w_down.scalar_type()), kTN});
    products_into(todo);
    if (dx.defined()) dx = dx.view(x.sizes());
    return {dx, dgu, dd, (need & 8) ? grads[0] : Tensor(), {}, {}, {}, {}};
  }
};
Tensor mlp(Tensor x, Tensor w_gate_up, Tensor w_down, c10::optional<Tensor> residual) {
  return MlpFn::apply(x, w_gate_up, w_down, residual, wants_grad(x), wants_grad(w_gate_up), wants_grad(w_down),
                      residual.has_value() && wants_grad(*residual));
}

struct AttentionFn : Function<AttentionFn> {
  static Tensor forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, Tensor cu, int64_t max_seqlen, bool causal,
                        double scale) {
    auto [o, lse] = attn_fwd(q, k, v, cu, max_seqlen, causal, scale);
    count();
    ctx->save_for_backward({q, k, v, o, lse, cu});
    ctx->saved_data["max"] = max_seqlen;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv, all] = attn_bwd(grads[0].contiguous(), s[0], s[1], s[2], s[3], s[4], s[5], ctx->saved_data["max"].toInt(),
                                      ctx->saved_data["causal"].toBool(), ctx->saved_data["scale"].toDouble(), false);
    count(3);
    return {dq, dk, dv, {}, {}, {}, {}};
  }
};
Tensor attention(Tensor q, Tensor k, Tensor v, Tensor cu, int64_t max_seqlen, bool causal, double scale) {
  return AttentionFn::apply(q, k, v, cu, max_seqlen, causal, scale);
}

// Attention straight on a fused projection: q/k/v are column views in forward, and the backward kernels write dq/dk/dv
// into column views of ONE gradient tensor, so autograd never materialises zero-padded slices.
struct AttentionQKVFn : Function<AttentionQKVFn> {
  static std::array<Tensor, 3> parts(const Tensor& qkv, int64_t n_q, int64_t n_kv, int64_t d) {
    const int64_t T = qkv.size(0), ld = qkv.stride(0);
    auto view = [&](int64_t first, int64_t heads) {
      return qkv.as_strided({T, heads, d}, {ld, d, 1}, qkv.storage_offset() + first * d);
    };
    return {view(0, n_q), view(n_q, n_kv), view(n_q + n_kv, n_kv)};
  }
  static Tensor forward(AutogradContext* ctx, Tensor qkv, int64_t n_q, int64_t n_kv, int64_t d, Tensor cu, int64_t max_seqlen,
                        bool causal, double scale) {
    TORCH_CHECK(qkv.dim() == 2 && qkv.size(1) == (n_q + 2 * n_kv) * d && qkv.stride(1) == 1, "attention: qkv [T,(Hq+2Hkv)*D]");
    const auto [q, k, v] = parts(qkv, n_q, n_kv, d);
    auto [o, lse] = attn_fwd(q, k, v, cu, max_seqlen, causal, scale);
    count();
    ctx->save_for_backward({qkv, o, lse, cu});
    ctx->saved_data["cfg"] = std::vector<int64_t>{n_q, n_kv, d, max_seqlen, causal};
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const auto [q, k, v] = parts(s[0], cfg[0], cfg[1], cfg[2]);
    auto [dq, dk, dv, dqkv] = attn_bwd(grads[0].contiguous(), q, k, v, s[1], s[2], s[3], cfg[3], cfg[4] != 0,
                                       ctx->saved_data["scale"].toDouble(), true);
    count(3);
    return {dqkv, {}, {}, {}, {}, {}, {}, {}};
  }
};
Tensor attention_qkv(Tensor qkv, int64_t n_q, int64_t n_kv, int64_t d, Tensor cu, int64_t max_seqlen, bool causal, double scale) {
  return AttentionQKVFn::apply(qkv, n_q, n_kv, d, cu, max_seqlen, causal, scale);
}

// ---- LM head ---------------------------------------------------------------------------------------------------------
void check_chunk(int64_t chunk) {
  if (chunk == 0) throw py::value_error("chunk must not be zero");   // the walk over the tokens would not end
  TORCH_CHECK(chunk > 0, "chunk must be positive");
}
// bf16 logits of one chunk of tokens, whatever type a library product of the head is in
Tensor chunk_logits(const Tensor& h, int64_t vocab, int64_t chunk) {
  check_chunk(chunk);
  return at::empty({std::min(chunk, h.size(0)), vocab}, h.options().dtype(at::kBFloat16));
}

// One chunk of the head: logits = h w^T, then either the log-probability of every label (`per_token`; `logits` is scratch that the
// first chunk to need it brings) or the logits turned in place into loss_scale * (softmax - onehot), with the summed loss added
// to `loss`.  Where the kernel takes the product its epilogue leaves the softmax statistics, and one pass over the logits, or
// both, is saved.
void head_chunk(const Tensor& h, const Tensor& w, Tensor& logits, const Tensor& labels, const c10::optional<Tensor>& loss_scale,
                const Tensor& loss, const Tensor& per_token, int64_t ignore_index, double inv_temp) {
  const int64_t n = h.size(0), V = w.size(0);
  if (!library_gemm() && odc::gemm_pairs_enabled() && h.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
      labels.scalar_type() == at::kLong && labels.is_contiguous() && h.stride(1) == 1 && w.stride(1) == 1 && w.size(1) == h.size(1) &&
      odc::logits_stats_pay(static_cast<int>(n), static_cast<int>(V), static_cast<int>(h.size(1)), !per_token.defined(), sm_count())) {
    c10::cuda::CUDAGuard g(h.device());
    odc::bind_device(h.get_device());
    const int tiles = odc::logits_stat_tiles(static_cast<int>(V));
    const auto f32 = h.options().dtype(at::kFloat);
    auto stats = at::empty({tiles, n, 2}, f32), at_label = at::empty({n}, f32);
    const auto* ids = reinterpret_cast<const long long*>(labels.data_ptr<int64_t>());
    const float t = static_cast<float>(inv_temp);
    const bool forward = per_token.defined();
    const cudaError_t e = odc::gemm_logits_pair(h.data_ptr(), w.data_ptr(), forward ? nullptr : logits.data_ptr(), ids,
                                                stats.data_ptr<float>(), at_label.data_ptr<float>(), static_cast<int>(n),
                                                static_cast<int>(V), static_cast<int>(h.size(1)), h.stride(0), w.stride(0),
                                                forward ? 8 : logits.stride(0), t, device_status(h.get_device()).data_ptr<int>(),
                                                sm_count(), cur_stream());
    if (e != cudaErrorNotSupported) {
      check(e, "head product");
      if (forward) {
        check(odc::launch_logprobs_from_stats(ids, stats.data_ptr<float>(), at_label.data_ptr<float>(), per_token.data_ptr<float>(),
                                              static_cast<int>(n), tiles, ignore_index, cur_stream(), t), "logprobs_from_stats");
      } else {
        if (loss_scale.has_value())
          TORCH_CHECK(loss_scale->scalar_type() == at::kFloat && loss_scale->is_contiguous(), "ce: loss_scale fp32");
        check(odc::launch_ce_from_stats(logits.data_ptr(), ids, loss_scale.has_value() ? loss_scale->data_ptr<float>() : nullptr,
                                        stats.data_ptr<float>(), at_label.data_ptr<float>(), loss.data_ptr<float>(),
                                        static_cast<int>(n), static_cast<int>(V), tiles, ignore_index, cur_stream(), t),
              "ce_from_stats");
      }
      count(2);
      return;
    }
  }
  if (!logits.defined()) logits = chunk_logits(h, V, n);
  const Tensor lg = logits.narrow(0, 0, n);
  product_into(h, w, lg, kNT);
  if (per_token.defined())
    token_logprobs(lg, labels, per_token, ignore_index, inv_temp);
  else
    ce_fwd_bwd(lg, labels, loss_scale, loss, ignore_index, inv_temp);
  count();
}

// Loss and both gradients (for a loss gradient of one) in one pass over token chunks; [T, vocab] logits never exist.
// Same mathematics as the reference's chunked LM head (examples/llm_training/lm_head.py:7-59), but the gradients are
// formed while the chunk's logits are at hand, so backward is a multiplication by the loss gradient.
std::tuple<Tensor, Tensor, Tensor> lm_head_loss(const Tensor& h, const Tensor& w, const Tensor& labels,
                                                const c10::optional<Tensor>& loss_scale, int64_t ignore_index, int64_t chunk,
                                                bool need_dh, bool need_dw, c10::optional<Tensor> dw_out) {
  const int64_t T = h.size(0), V = w.size(0), H = h.size(1);
  auto loss = at::zeros({}, h.options().dtype(at::kFloat));
  auto logits = chunk_logits(h, V, chunk);
  Tensor dh, dw;
  if (need_dh) dh = at::empty_like(h);
  if (need_dw) dw = dw_out.has_value() ? *dw_out : at::empty({V, H}, h.options().dtype(at::kFloat));
  if (T == 0 && need_dw) dw.zero_();
  for (int64_t s = 0; s < T; s += chunk) {
    const int64_t n = std::min(chunk, T - s);
    const Tensor hs = h.narrow(0, s, n);
    Tensor lg = logits.narrow(0, 0, n);
    head_chunk(hs, w, lg, labels.narrow(0, s, n), loss_scale.has_value() ? c10::optional<Tensor>(loss_scale->narrow(0, s, n)) : c10::nullopt,
               loss, {}, ignore_index, 1.0);
    std::vector<Product> todo;
    if (need_dh) todo.push_back({lg, w, dh.narrow(0, s, n), kNN});
    if (need_dw) todo.push_back({lg, hs, dw, kTN, s > 0});
    products_into(todo);
  }
  return {loss, dh, dw};
}

// Tokens of one chunk: the gradient of their logits is kept for the backward instead of the fp32 gradient of the weight, which is
// then formed with the loss gradient in its epilogue and rounded once.  The fp32 matrix is neither written nor read again by a pass
// that multiplies it (128256 words, 2048 wide: 2.1 of 2.6 GB).  What waits for the backward is no larger than that matrix, or small.
// Loss and gradients of 256 tokens 720 us with the matrix, 452 without, of 1000 1540 and 1255, 4096 wide 1380 and 830; 4096 tokens
// the same.  Smallest training step, whose weight gradient goes straight to the accumulator: 1545 and 1367 us.
// Only where the kernel takes the products that are to gain by it, the weight's gradient alone or, `sharded`, both gradients: else the
// fp32 matrix would be formed after all, next to what has been kept (4000 tokens, 128256 words, 2048 wide: a peak of 3.0 GB instead of 2.0).
bool logit_grads_pay(int64_t T, int64_t V, int64_t H, int64_t chunk, bool sharded, int sms) {
  constexpr int64_t kSmall = 128 << 20;
  const int64_t kept = T * V * 2, instead = V * H * 4;
  if (T < 1 || T > chunk || (kept > instead && kept > kSmall)) return false;
  odc::GemmProduct g[2] = {};
  g[0].M = static_cast<int>(V); g[0].N = static_cast<int>(H); g[0].K = static_cast<int>(T);
  g[0].layout = kTN; g[0].lda = V; g[0].ldb = g[0].ldc = H;
  g[0].c_kind = sharded ? odc::kF32 : odc::kBF16;
  g[1].M = static_cast<int>(T); g[1].N = static_cast<int>(H); g[1].K = static_cast<int>(V);
  g[1].layout = kNN; g[1].lda = V; g[1].ldb = g[1].ldc = H;
  g[1].c_kind = odc::kBF16;
  return odc::gemm_group_takes(g, sharded ? 2 : 1, sms);
}
bool keeps_logit_grads(const Tensor& h, const Tensor& w, int64_t chunk, bool need_dw, bool sharded) {
  return need_dw && h.dim() == 2 && h.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && !library_gemm() &&
         odc::gemm_pairs_enabled() && logit_grads_pay(h.size(0), w.size(0), h.size(1), chunk, sharded, sm_count());
}
std::tuple<Tensor, Tensor> loss_and_logit_grads(const Tensor& h, const Tensor& w, const Tensor& labels, const c10::optional<Tensor>& loss_scale,
                                                int64_t ignore_index) {
  auto loss = at::zeros({}, h.options().dtype(at::kFloat));
  auto logits = chunk_logits(h, w.size(0), h.size(0));
  head_chunk(h, w, logits, labels, loss_scale, loss, {}, ignore_index, 1.0);
  return {loss, logits};
}
// (logits' gradient)^T h * *g, in the type of the weight
Tensor head_weight_grad(const Tensor& dlogits, const Tensor& h, const Tensor& g) {
  const Tensor g32 = g.to(at::kFloat);
  Tensor dw = product_out(dlogits, h, kTN);
  if (group_into({{dlogits, h, dw, kTN, false, 1.0, g32, {}, false, true}})) return dw;   // one sum, as the fp32 matrix is
  return scale_to_bf16(product(dlogits, h, kTN, {}, {}, at::kFloat), g32);
}

struct LinearCrossEntropyFn : Function<LinearCrossEntropyFn> {
  static Tensor forward(AutogradContext* ctx, Tensor h, Tensor w, Tensor labels, c10::optional<Tensor> loss_scale,
                        int64_t ignore_index, int64_t chunk, bool need_dh, bool need_dw) {
    check_chunk(chunk);
    if (keeps_logit_grads(h, w, chunk, need_dw, false)) {
      auto [loss, dlogits] = loss_and_logit_grads(h, w, labels, loss_scale, ignore_index);
      Tensor dh;
      if (need_dh) dh = product(dlogits, w, kNN);
      ctx->save_for_backward({dh, h.clone(), dlogits});   // a copy: the caller may write to h before the backward, as with several chunks
      return loss;
    }
    auto [loss, dh, dw] = lm_head_loss(h, w, labels, loss_scale, ignore_index, chunk, need_dh, need_dw, c10::nullopt);
    ctx->save_for_backward({dh, dw});
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor& g = grads[0];
    Tensor gh, gw;
    if (s[0].defined()) gh = scale_to_bf16(s[0], g);
    if (s.size() == 3) return {gh, head_weight_grad(s[2], s[1], g), {}, {}, {}, {}, {}, {}};
    if (s[1].defined()) gw = scale_to_bf16(s[1], g);
    return {gh, gw, {}, {}, {}, {}, {}, {}};
  }
};
Tensor linear_cross_entropy(Tensor h, Tensor w, Tensor labels, c10::optional<Tensor> loss_scale, int64_t ignore_index,
                            int64_t chunk) {
  if (loss_scale.has_value()) loss_scale = loss_scale->to(at::kFloat);  // FSDP's mixed-precision input cast may have narrowed it
  return LinearCrossEntropyFn::apply(h.contiguous(), w, labels.contiguous(), loss_scale, ignore_index, chunk, wants_grad(h),
                                     wants_grad(w));
}

// Per-token log-probability of `ids` under softmax(h w^T / temperature), in token chunks: the policy-gradient form of the
// chunked LM head (the reference's FusedLinearForPPOFunction, examples/llm_training/lm_head.py:62-190).  The weights of
// the tokens are only known in backward, so backward recomputes each chunk's logits and turns them in place into
// dlogp / temperature * (onehot - softmax).
struct LinearTokenLogProbsFn : Function<LinearTokenLogProbsFn> {
  static Tensor forward(AutogradContext* ctx, Tensor h, Tensor w, Tensor ids, double temperature, int64_t ignore_index,
                        int64_t chunk, bool need_dh, bool need_dw) {
    const int64_t T = h.size(0);
    auto out = at::empty({T}, h.options().dtype(at::kFloat));
    check_chunk(chunk);
    Tensor logits;
    for (int64_t s = 0; s < T; s += chunk) {
      const int64_t n = std::min(chunk, T - s);
      head_chunk(h.narrow(0, s, n), w, logits, ids.narrow(0, s, n), c10::nullopt, {}, out.narrow(0, s, n), ignore_index, 1.0 / temperature);
    }
    ctx->save_for_backward({h, w, ids});
    ctx->saved_data["cfg"] = std::vector<int64_t>{ignore_index, chunk, need_dh, need_dw};
    ctx->saved_data["temperature"] = temperature;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &w = saved[1], &ids = saved[2];
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const double temperature = ctx->saved_data["temperature"].toDouble();
    const int64_t T = h.size(0), chunk = cfg[1];
    Tensor dh, dw;
    if (cfg[2]) dh = at::empty_like(h);
    // Several chunks are summed in fp32, and the product of the last one is rounded once, in its own epilogue, with the sum so far:
    // the sum is read once more instead of read and written, and there is no pass that narrows it (6000 tokens, 151936 words, 1536
    // wide, forward and backward: 8.62 -> 8.44 ms).
    if (cfg[3]) dw = at::empty(w.sizes(), T > chunk ? w.options().dtype(at::kFloat) : w.options());
    if (T == 0 && cfg[3]) dw.zero_();
    const Tensor scale = (grads[0].reshape({-1}).to(at::kFloat) * (-1.0 / temperature)).contiguous();
    auto sink = at::zeros({}, scale.options());  // the kernel's loss output is not used here
    auto logits = chunk_logits(h, w.size(0), chunk);
    for (int64_t s = 0; s < T; s += chunk) {
      const int64_t n = std::min(chunk, T - s);
      const Tensor hs = h.narrow(0, s, n);
      Tensor lg = logits.narrow(0, 0, n);
      head_chunk(hs, w, lg, ids.narrow(0, s, n), scale.narrow(0, s, n), sink, {}, cfg[0], 1.0 / temperature);
      std::vector<Product> todo;
      if (cfg[2]) todo.push_back({lg, w, dh.narrow(0, s, n), kNN});
      if (cfg[3] && s > 0 && s + n == T && w.scalar_type() == at::kBFloat16) {
        const Tensor whole = at::empty(w.sizes(), w.options());
        todo.push_back({lg, hs, whole, kTN, false, 1.0, {}, dw});
        if (group_into(todo)) {
          dw = whole;
          break;
        }
        todo.pop_back();
      }
      if (cfg[3]) todo.push_back({lg, hs, dw, kTN, s > 0});
      products_into(todo);
    }
    return {dh, dw.defined() ? dw.to(w.scalar_type()) : dw, {}, {}, {}, {}, {}, {}};
  }
};
Tensor linear_token_logprobs(Tensor h, Tensor w, Tensor ids, double temperature, int64_t ignore_index, int64_t chunk) {
  return LinearTokenLogProbsFn::apply(h.contiguous(), w, ids.contiguous(), temperature, ignore_index, chunk, wants_grad(h),
                                      wants_grad(w));
}

// ---- linear layer of the sharded engine --------------------------------------------------------------------------------
// Contributions sent by native code since the reduction service last asked (it adds them to its own books at `sync`).
struct DispatchCounter : torch::CustomClassHolder {
  std::atomic<int64_t> n{0};
  int64_t take() { return n.exchange(0); }
};

// What one row-sharded matrix needs at every call: its shard, the peers' addresses, its accumulator.
struct ShardedMatrix : torch::CustomClassHolder {
  int64_t id = 0;                       // how the Python side knows it
  Tensor shard;                         // [rows_per_rank, K] bf16, in the symmetric heap
  Tensor table, acc_table, ctr_table;   // device tables of the owners' shards / accumulators / arrival counters
  std::vector<int64_t> acc_addrs;
  int64_t out_features = 0, rows_per_rank = 0, world = 1, index = 0;
  double grad_scale = 1.0;
  bool local_pending = false;           // earlier microbatches left a gradient in the local buffer
  c10::intrusive_ptr<DispatchCounter> dispatched;
  Tensor matrix;                        // [out_features, K]: the shard of one rank without its padding rows
  const Tensor& whole() const { return matrix; }
};

// Start of the last minibatch: an event behind its work, and the stream it ran on.  A pass on that stream is in order as it
// is; any other waits for the event.  (A stream that is being captured cannot wait for work outside of the capture.)
struct MinibatchStart {
  std::mutex mu;
  cudaEvent_t event = nullptr;
  std::atomic<cudaStream_t> stream{nullptr};
  std::atomic<bool> set{false};
} g_start;

void mark_start() {
  std::lock_guard<std::mutex> lock(g_start.mu);
  const cudaStream_t s = cur_stream();
  if (g_start.event == nullptr) check(cudaEventCreateWithFlags(&g_start.event, cudaEventDisableTiming), "mark_start");
  check(cudaEventRecord(g_start.event, s), "mark_start");
  g_start.stream = s;
  g_start.set = true;
}

void after_start() {
  if (!g_start.set) return;
  const cudaStream_t s = cur_stream();
  if (s == g_start.stream) return;
  if (capturing()) return;
  std::lock_guard<std::mutex> lock(g_start.mu);
  check(cudaStreamWaitEvent(s, g_start.event, 0), "after_start");
}

std::atomic<bool> g_sync_grads{true};   // false: weight gradients are accumulated on the producing rank
// Python, by matrix: a gradient (id, dy2, x2) that is not pushed straight away; the local buffer, which has something to push from
// here on; push it
py::object *g_deferred = nullptr, *g_local_buffer = nullptr, *g_push_local = nullptr;

// dy2^T x2 into the owners' accumulators, or, where pushes are off, into the local buffer
void push_weight_grad(ShardedMatrix* m, const Tensor& dy2, const Tensor& x2) {
  if (!g_sync_grads || m->local_pending) {
    py::gil_scoped_acquire gil;
    (*g_deferred)(m->id, dy2, x2);
    return;
  }
  // whole 128-row tiles per owner and at most 8 owners: output boxes added by the TMA unit; else per-thread reductions
  if (!gemm_wgrad_scatter_tma(dy2, x2, m->acc_addrs, m->ctr_table, 0, m->rows_per_rank, m->grad_scale, m->index))
    gemm_wgrad_scatter(dy2, x2, m->acc_table, m->ctr_table, 0, m->rows_per_rank, m->grad_scale);
  count();
  m->dispatched->n.fetch_add(1);
}

// What one backward forms from dy2: dx = dy2 w, and the gradients dy^T x of one or two matrices.  With one rank that is one launch:
// the weight gradients are added to the accumulators, or to the local buffers where pushes are off, so that dx is summed in the
// same order either way.
struct WeightGrad {
  ShardedMatrix* m;
  Tensor dy2, x2;
};
Tensor sharded_grads(const Tensor& dy2, const ShardedMatrix* m, const std::vector<WeightGrad>& weights) {
  const Tensor dx = product_out(dy2, m->whole(), kNN);
  const bool pushes = g_sync_grads;
  std::vector<Product> todo{{dy2, m->whole(), dx, kNN}};
  for (const auto& w : weights) {
    if (w.m->world != 1 || w.m->ctr_table.data_ptr() != m->ctr_table.data_ptr()) break;
    Tensor to;
    if (pushes) {
      to = at::from_blob(reinterpret_cast<void*>(w.m->acc_addrs[0]), {w.m->out_features, w.m->shard.size(1)}, w.m->shard.options().dtype(at::kFloat));
    } else {
      py::gil_scoped_acquire gil;
      to = (*g_local_buffer)(w.m->id).cast<Tensor>().narrow(0, 0, w.m->out_features);
    }
    // several parts meet in the accumulator as they do in a launch of its own; the local buffer is a sum in one order
    todo.push_back({w.dy2, w.x2, to, kTN, true, pushes ? w.m->grad_scale : 1.0, {}, {}, pushes});
  }
  if (todo.size() == weights.size() + 1 && group_into(todo, m->ctr_table, pushes ? static_cast<int>(weights.size()) : 0)) {
    for (const auto& w : weights) {
      if (!pushes) continue;
      w.m->dispatched->n.fetch_add(1);
      if (w.m->local_pending) {   // what earlier microbatches accumulated locally follows
        py::gil_scoped_acquire gil;
        (*g_push_local)(w.m->id);
      }
    }
    return dx;
  }
  product_into(dy2, m->whole(), dx, kNN);
  for (const auto& w : weights) push_weight_grad(w.m, w.dy2, w.x2);
  return dx;
}

// Backward of the sharded engine's loss over tokens of one chunk: dh = dlogits w * *g, and dlogits^T h * scale * *g into the
// accumulator of one rank (reported as an arrival), or added to `local`, or written to it without the factors.
Tensor sharded_head_grads(const Tensor& dlogits, const Tensor& h, const Tensor& w, const Tensor& g, const c10::intrusive_ptr<ShardedMatrix>& m,
                          c10::optional<Tensor> local, bool add) {
  const Tensor g32 = g.to(at::kFloat);
  const bool direct = !local.has_value();
  TORCH_CHECK(!direct || m->world == 1, "sharded_head_grads: the accumulator of one rank");
  const Tensor dw = direct ? at::from_blob(reinterpret_cast<void*>(m->acc_addrs[0]), {m->out_features, h.size(1)}, h.options().dtype(at::kFloat))
                           : *local;
  const Tensor dh = product_out(dlogits, w, kNN);
  std::vector<Product> todo{{dlogits, w, dh, kNN, false, 1.0, g32},
                            {dlogits, h, dw, kTN, direct || add, direct ? m->grad_scale : 1.0, direct || add ? g32 : Tensor()}};
  if (group_into(todo, direct ? m->ctr_table : Tensor(), direct ? 1 : 0)) {
    if (direct) m->dispatched->n.fetch_add(1);
    return dh;
  }
  // one by one: dh rounded once more; the weight's gradient by way of a matrix of its own
  product_into(dlogits, w, dh, kNN);
  if (direct || add) {
    const Tensor dw32 = product(dlogits, h, kTN, {}, {}, at::kFloat);
    if (direct) {
      check(odc::launch_scatter_accumulate(dw32.data_ptr(), odc::kF32, reinterpret_cast<const long long*>(m->acc_table.data_ptr<int64_t>()),
                                           odc::kF32, reinterpret_cast<const long long*>(m->ctr_table.data_ptr<int64_t>()),
                                           static_cast<size_t>(dw32.numel()), 1, 0, static_cast<float>(m->grad_scale),
                                           next_done_slot(h.get_device()), sm_count(), cur_stream(),
                                           device_status(h.get_device()).data_ptr<int>(), 0, g32.data_ptr<float>()), "head gradient");
      count();
      m->dispatched->n.fetch_add(1);
    } else {
      dw.addcmul_(dw32, g32);
    }
  } else {
    product_into(dlogits, h, dw, kTN);
  }
  return scale_to_bf16(dh, g32);
}

// Forward is the plain product for one rank, else the product that pulls the owners' rows inside the kernel; the weight
// gradient is added into its owners from the epilogue of its product.  The weight is no autograd input.
struct ShardedLinearFn : Function<ShardedLinearFn> {
  static Tensor forward(AutogradContext* ctx, Tensor x, c10::optional<Tensor> bias, c10::optional<Tensor> residual,
                        c10::intrusive_ptr<ShardedMatrix> m, c10::optional<Tensor> bias_sink, bool keep_weight, bool need_dx,
                        bool need_db, bool need_dres) {
    const Tensor x2 = rows2d(x);
    c10::optional<Tensor> res;
    if (residual.has_value()) res = rows2d(*residual);
    Tensor y, w_full;
    if (m->world == 1) {
      y = product(x2, m->whole(), kNT, bias.value_or(Tensor()), res.value_or(Tensor()));
    } else {
      w_full = at::empty({m->out_features, m->shard.size(1)}, m->shard.options());
      y = gemm_gather(x2, m->table, w_full, bias, m->rows_per_rank, m->index, res);
      count();
    }
    if (!keep_weight) w_full = Tensor();  // dropped: backward pulls the shards again
    ctx->save_for_backward({x, w_full});
    ctx->saved_data["need"] = static_cast<int64_t>(need_dx | need_db << 1 | need_dres << 2);
    if (bias_sink.has_value()) ctx->saved_data["sink"] = *bias_sink;
    ctx->saved_data["m"] = c10::IValue::make_capsule(m);
    return like(y, x, m->out_features);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    auto capsule = ctx->saved_data["m"].toCapsule();
    auto* m = static_cast<ShardedMatrix*>(capsule.get());
    const int64_t need = ctx->saved_data["need"].toInt();
    const Tensor dy2 = rows2d(grads[0]).contiguous(), x2 = rows2d(x).contiguous();
    Tensor dx, db;
    if ((need & 1) && m->world == 1) {
      dx = sharded_grads(dy2, m, {{m, dy2, x2}}).view(x.sizes());
    } else if (need & 1) {
      if (saved[1].defined()) {
        dx = product(dy2, saved[1], kNN);
      } else {
        auto w_full = at::empty({m->out_features, m->shard.size(1)}, m->shard.options());
        dx = gemm_gather_dgrad(dy2, m->table, w_full, m->rows_per_rank, m->index);
        count();
      }
      dx = dx.view(x.sizes());
    }
    if (!(need & 1) || m->world != 1) push_weight_grad(m, dy2, x2);
    auto sink = ctx->saved_data.find("sink");
    if (sink != ctx->saved_data.end()) {
      const Tensor s = sink->second.toTensor();
      check(odc::launch_column_sum(dy2.data_ptr(), nullptr, s.data_ptr<float>(), dy2.size(0), static_cast<int>(dy2.size(1)),
                                   cur_stream()), "column_sum");
      count();
    } else if (need & 2) {
      db = column_sum(dy2);
    }
    return {dx, db, (need & 4) ? grads[0] : Tensor(), {}, {}, {}, {}, {}, {}};
  }
};
Tensor sharded_linear(Tensor x, c10::optional<Tensor> bias, c10::optional<Tensor> residual, c10::intrusive_ptr<ShardedMatrix> m,
                      c10::optional<Tensor> bias_sink, bool keep_weight) {
  after_start();
  const bool db = bias.has_value() && wants_grad(*bias), dres = residual.has_value() && wants_grad(*residual);
  return ShardedLinearFn::apply(x, bias, residual, m, bias_sink, keep_weight, wants_grad(x), db, dres);
}

// The two matrices of an MLP on one rank, as MlpFn
struct ShardedMlpFn : Function<ShardedMlpFn> {
  static Tensor forward(AutogradContext* ctx, Tensor x, c10::optional<Tensor> residual, c10::intrusive_ptr<ShardedMatrix> gu,
                        c10::intrusive_ptr<ShardedMatrix> down, bool need_dx, bool need_dres) {
    auto [act, gate_up] = linear_swiglu_fwd(rows2d(x), gu->whole(), need_dx || need_dres);
    Tensor res;
    if (residual.has_value()) res = rows2d(*residual);
    const Tensor y = product(act, down->whole(), kNT, {}, res);
    ctx->save_for_backward({x, gate_up, act});
    ctx->saved_data["need"] = static_cast<int64_t>(need_dx | need_dres << 1);
    ctx->saved_data["gu"] = c10::IValue::make_capsule(gu);
    ctx->saved_data["down"] = c10::IValue::make_capsule(down);
    return like(y, x, down->out_features);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor& x = s[0];
    auto gu_capsule = ctx->saved_data["gu"].toCapsule(), down_capsule = ctx->saved_data["down"].toCapsule();
    auto *gu = static_cast<ShardedMatrix*>(gu_capsule.get()), *down = static_cast<ShardedMatrix*>(down_capsule.get());
    const int64_t need = ctx->saved_data["need"].toInt();
    const Tensor dy2 = rows2d(grads[0]).contiguous(), x2 = rows2d(x).contiguous();
    Tensor dx;
    if (need & 1) {   // as layers one behind the other: without it only the last has anything to do
      const Tensor d = swiglu_product_bwd(dy2, down->whole(), s[1]);
      dx = sharded_grads(d, gu, {{gu, d, x2}, {down, dy2, s[2]}}).view(x.sizes());
    } else {
      push_weight_grad(down, dy2, s[2]);
    }
    return {dx, (need & 2) ? grads[0] : Tensor(), {}, {}, {}, {}};
  }
};
Tensor sharded_mlp(Tensor x, c10::optional<Tensor> residual, c10::intrusive_ptr<ShardedMatrix> gu,
                   c10::intrusive_ptr<ShardedMatrix> down) {
  TORCH_CHECK(gu->world == 1 && down->world == 1, "sharded_mlp: one rank");
  after_start();
  return ShardedMlpFn::apply(x, residual, gu, down, wants_grad(x), residual.has_value() && wants_grad(*residual));
}

// ---- a decoder layer as one function -----------------------------------------------------------------------------------
// norm, projection, rotary embedding, attention, output projection, norm, MLP.  Seven functions one behind the other cost the host
// their interpreter calls, graph nodes and gradient hand-overs, and a small model's step waits for the host all the time.
// Same kernels, same tensors kept for backward.  Two layers, 512 wide, two microbatches: a training step 2123 us in parts, 1685 as
// one function a layer; a layer over 1000 tokens, 1536 wide, 373 and 365.
struct LayerShape {
  int64_t n_q, n_kv, d, max_seqlen;
  double theta, eps1, eps2;
  double scale() const { return 1.0 / std::sqrt(static_cast<double>(d)); }
  std::vector<int64_t> ints() const { return {n_q, n_kv, d, max_seqlen}; }
};
struct LayerWeights {
  Tensor norm1, wqkv, bqkv, wo, norm2, gate_up, down;   // bqkv may be undefined
};
enum LayerKept : int { kX1, kRstd1, kH1, kQkv, kO, kLse, kX2, kRstd2, kH2, kGateUp, kAct, kKept };

// plain bf16 matrices and vectors of one layer; anything else takes the layer's modules one by one, which say what is wrong
bool layer_takes(const Tensor& x, const Tensor& pos, const Tensor& cu, const LayerWeights& w, const LayerShape& c) {
  const auto plain = [&](const Tensor& t, at::ScalarType type) {
    return t.defined() && t.device() == x.device() && t.scalar_type() == type && t.layout() == at::kStrided && t.is_contiguous() &&
           !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                                     c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched}));
  };
  const auto matrix = [&](const Tensor& t, int64_t rows, int64_t cols) {
    return plain(t, at::kBFloat16) && t.dim() == 2 && t.size(0) == rows && t.size(1) == cols;
  };
  const char* attention = std::getenv("ODC_ATTN");
  if (!x.is_cuda() || x.dim() != 2 || !plain(x, at::kBFloat16) || x.size(0) == 0 || library_gemm() ||
      (attention != nullptr && std::strcmp(attention, "native") != 0))
    return false;
  const int64_t T = x.size(0), H = x.size(1), qkv = (c.n_q + 2 * c.n_kv) * c.d;
  return (c.d == 64 || c.d == 128) && c.n_kv > 0 && c.n_q % c.n_kv == 0 && H % 8 == 0 && plain(pos, at::kLong) && pos.numel() == T &&
         plain(cu, at::kInt) && cu.numel() >= 2 && plain(w.norm1, at::kBFloat16) && w.norm1.numel() == H &&
         plain(w.norm2, at::kBFloat16) && w.norm2.numel() == H && matrix(w.wqkv, qkv, H) && matrix(w.wo, H, c.n_q * c.d) &&
         w.down.defined() && w.down.dim() == 2 && matrix(w.down, H, w.down.size(1)) && w.down.size(1) % 8 == 0 &&
         matrix(w.gate_up, 2 * w.down.size(1), H) && (!w.bqkv.defined() || (plain(w.bqkv, at::kBFloat16) && w.bqkv.numel() == qkv));
}

// y, and what a backward needs (empty unless `keep`)
std::tuple<Tensor, variable_list> layer_forward(const Tensor& x, const Tensor& pos, const Tensor& cu, const LayerWeights& w,
                                                const LayerShape& c, bool keep) {
  variable_list kept(keep ? kKept : 0);
  const auto hold = [&](LayerKept i, const Tensor& t) { if (keep) kept[i] = t; };
  Tensor qkv, x2, act;
  {
    auto [h, rstd] = rmsnorm_fwd(x, w.norm1, c.eps1);
    hold(kX1, x); hold(kRstd1, rstd); hold(kH1, h);
    qkv = linear_rope(h, w.wqkv, w.bqkv, pos, c.n_q, c.n_kv, c.d, c.theta);
  }
  hold(kQkv, qkv);
  {
    const auto [q, k, v] = AttentionQKVFn::parts(qkv, c.n_q, c.n_kv, c.d);
    auto [o, lse] = attn_fwd(q, k, v, cu, c.max_seqlen, true, c.scale());
    hold(kO, o); hold(kLse, lse);
    qkv = Tensor();
    x2 = product(o.view({x.size(0), c.n_q * c.d}), w.wo, kNT, {}, x);
  }
  hold(kX2, x2);
  {
    auto [h, rstd] = rmsnorm_fwd(x2, w.norm2, c.eps2);
    hold(kRstd2, rstd); hold(kH2, h);
    auto [a, gate_up] = linear_swiglu_fwd(h, w.gate_up, keep);
    hold(kGateUp, gate_up); hold(kAct, a);
    act = a;
  }
  count(3);
  return {product(act, w.down, kNT, {}, x2), kept};
}

// dx; `sink` takes the gradients of the weights:
//   linear(0: projection, 1: output projection; dy2, x2) -> dx;  mlp(d, x2, dy2, act) -> d gate_up;  norm(which, ...) -> dx;  bias(dqkv)
template <typename Sink>
Tensor layer_backward(const variable_list& kept, const Tensor& pos, const Tensor& cu, const LayerWeights& w, const LayerShape& c,
                      const Tensor& dy, Sink& sink) {
  const int64_t T = dy.size(0);
  const Tensor d = swiglu_product_bwd(dy, w.down, kept[kGateUp]);
  const Tensor dh2 = sink.mlp(d, kept[kH2], dy, kept[kAct]);
  const Tensor dx2 = sink.norm(1, dh2, kept[kX2], w.norm2, kept[kRstd2], dy);
  const Tensor o = kept[kO];
  const Tensor dout = sink.linear(1, dx2, o.view({T, c.n_q * c.d})).view({T, c.n_q, c.d});
  const auto [q, k, v] = AttentionQKVFn::parts(kept[kQkv], c.n_q, c.n_kv, c.d);
  const Tensor dqkv = std::get<3>(attn_bwd(dout, q, k, v, o, kept[kLse], cu, c.max_seqlen, true, c.scale(), true, pos, c.theta));
  count(3);
  const Tensor dh1 = sink.linear(0, dqkv, kept[kH1]);
  sink.bias(dqkv);
  return sink.norm(0, dh1, kept[kX1], w.norm1, kept[kRstd1], dx2);
}

struct LayerFn : Function<LayerFn> {
  struct Sink {
    const LayerWeights& w;
    Tensor norm_grad[2], norm_sums, matrix[2], d_gate_up, d_down, d_bias;
    Tensor linear(int which, const Tensor& dy2, const Tensor& x2) {
      const Tensor& m = which == 0 ? w.wqkv : w.wo;
      Tensor dx;
      std::tie(dx, matrix[which]) = linear_grads(dy2, x2, m, true, true);
      return dx;
    }
    Tensor mlp(const Tensor& d, const Tensor& x2, const Tensor& dy2, const Tensor& act) {
      const Tensor dx = product_out(d, w.gate_up, kNN);
      d_gate_up = product_out(d, x2, kTN);
      d_down = product_out(dy2, act, kTN);
      products_into({{d, w.gate_up, dx, kNN}, {d, x2, d_gate_up, kTN}, {dy2, act, d_down, kTN}});
      return dx;
    }
    Tensor norm(int which, const Tensor& dh, const Tensor& x, const Tensor& weight, const Tensor& rstd, const Tensor& dres) {
      if (!norm_sums.defined()) norm_sums = at::zeros({2, x.size(1)}, x.options().dtype(at::kFloat));   // of both norms
      return std::get<0>(norm_grads(dh, x, weight, rstd, dres, norm_sums.select(0, which)));
    }
    void narrow_norms() {
      for (int i = 0; i < 2; ++i) norm_grad[i] = at::empty({norm_sums.size(1)}, w.norm1.options());
      check(odc::launch_narrow_pair(norm_sums.data_ptr<float>(), norm_grad[0].data_ptr(), norm_grad[1].data_ptr(),
                                    static_cast<int>(norm_sums.size(1)), cur_stream()), "layer backward");
      count();
    }
    void bias(const Tensor& dqkv) { if (w.bqkv.defined()) d_bias = column_sum(dqkv); }
  };
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor norm1, Tensor wqkv, c10::optional<Tensor> bqkv, Tensor wo, Tensor norm2,
                        Tensor gate_up, Tensor down, Tensor pos, Tensor cu, const LayerShape& c, bool keep) {
    const LayerWeights w{norm1, wqkv, bqkv.value_or(Tensor()), wo, norm2, gate_up, down};
    auto [y, kept] = layer_forward(x, pos, cu, w, c, keep);
    if (keep) {
      for (const Tensor& t : {w.norm1, w.wqkv, w.bqkv, w.wo, w.norm2, w.gate_up, w.down, pos, cu}) kept.push_back(t);
      ctx->save_for_backward(std::move(kept));
      ctx->saved_data["shape"] = c.ints();
      ctx->saved_data["theta"] = c.theta;
    }
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto kept = ctx->get_saved_variables();
    const auto i = ctx->saved_data["shape"].toIntVector();
    const LayerShape c{i[0], i[1], i[2], i[3], ctx->saved_data["theta"].toDouble(), 0, 0};
    const LayerWeights w{kept[kKept], kept[kKept + 1], kept[kKept + 2], kept[kKept + 3], kept[kKept + 4], kept[kKept + 5], kept[kKept + 6]};
    Sink sink{w};
    const Tensor dx = layer_backward(kept, kept[kKept + 7], kept[kKept + 8], w, c, grads[0].contiguous(), sink);
    sink.narrow_norms();
    return {dx, sink.norm_grad[0], sink.matrix[0], sink.d_bias, sink.matrix[1], sink.norm_grad[1], sink.d_gate_up, sink.d_down, {}, {}, {}, {}};
  }
};

// None: not a layer of plain weights that all want a gradient, or none: its modules have to be called
c10::optional<Tensor> decoder_layer(Tensor x, Tensor pos, Tensor cu, int64_t max_seqlen, int64_t n_q, int64_t n_kv, int64_t d, double theta,
                                    double eps1, double eps2, Tensor norm1, Tensor wqkv, c10::optional<Tensor> bqkv, Tensor wo, Tensor norm2,
                                    Tensor gate_up, Tensor down) {
  const LayerShape c{n_q, n_kv, d, max_seqlen, theta, eps1, eps2};
  if (!layer_takes(x, pos, cu, {norm1, wqkv, bqkv.value_or(Tensor()), wo, norm2, gate_up, down}, c)) return c10::nullopt;
  const bool keep = wants_grad(x);
  for (const Tensor& t : {norm1, wqkv, bqkv.value_or(x), wo, norm2, gate_up, down})
    if (wants_grad(t) != keep) return c10::nullopt;
  return LayerFn::apply(x, norm1, wqkv, bqkv, wo, norm2, gate_up, down, pos, cu, c, keep);
}

// The same for the sharded engine on one rank: the weights are no autograd inputs, their gradients go to the accumulators.
struct ShardedLayer : torch::CustomClassHolder {
  c10::intrusive_ptr<ShardedMatrix> wqkv, wo, gate_up, down;
  LayerWeights w;
  Tensor norm_sink[2], bias_sink;
  LayerShape c;
};
struct ShardedLayerFn : Function<ShardedLayerFn> {
  struct Sink {
    const ShardedLayer& s;
    Tensor linear(int which, const Tensor& dy2, const Tensor& x2) {
      ShardedMatrix* m = which == 0 ? s.wqkv.get() : s.wo.get();
      return sharded_grads(dy2, m, {{m, dy2, x2}});
    }
    Tensor mlp(const Tensor& d, const Tensor& x2, const Tensor& dy2, const Tensor& act) {
      return sharded_grads(d, s.gate_up.get(), {{s.gate_up.get(), d, x2}, {s.down.get(), dy2, act}});
    }
    Tensor norm(int which, const Tensor& dh, const Tensor& x, const Tensor& weight, const Tensor& rstd, const Tensor& dres) {
      return std::get<0>(norm_grads(dh, x, weight, rstd, dres, s.norm_sink[which]));
    }
    void bias(const Tensor& dqkv) {
      if (!s.w.bqkv.defined()) return;
      check(odc::launch_column_sum(dqkv.data_ptr(), nullptr, s.bias_sink.data_ptr<float>(), dqkv.size(0), static_cast<int>(dqkv.size(1)),
                                   cur_stream()), "column_sum");
      count();
    }
  };
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor pos, Tensor cu, c10::intrusive_ptr<ShardedLayer> s, bool keep) {
    auto [y, kept] = layer_forward(x, pos, cu, s->w, s->c, keep);
    if (keep) {
      kept.push_back(pos);
      kept.push_back(cu);
      ctx->save_for_backward(std::move(kept));
      ctx->saved_data["layer"] = c10::IValue::make_capsule(s);
    }
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto kept = ctx->get_saved_variables();
    auto capsule = ctx->saved_data["layer"].toCapsule();
    const auto& s = *static_cast<ShardedLayer*>(capsule.get());
    Sink sink{s};
    return {layer_backward(kept, kept[kKept], kept[kKept + 1], s.w, s.c, grads[0].contiguous(), sink), {}, {}, {}, {}};
  }
};
// (view of the gathered vector, fp32 buffer its gradient is added to) for both norms and the bias
using SmallWeight = std::tuple<Tensor, Tensor>;
c10::optional<Tensor> sharded_layer(Tensor x, Tensor pos, Tensor cu, int64_t max_seqlen, int64_t n_q, int64_t n_kv, int64_t d, double theta,
                                    double eps, SmallWeight norm1, c10::intrusive_ptr<ShardedMatrix> wqkv, c10::optional<SmallWeight> bqkv,
                                    c10::intrusive_ptr<ShardedMatrix> wo, SmallWeight norm2, c10::intrusive_ptr<ShardedMatrix> gate_up,
                                    c10::intrusive_ptr<ShardedMatrix> down) {
  for (const auto* m : {wqkv.get(), wo.get(), gate_up.get(), down.get()}) TORCH_CHECK(m->world == 1, "sharded_layer: one rank");
  auto s = c10::make_intrusive<ShardedLayer>();
  s->wqkv = wqkv; s->wo = wo; s->gate_up = gate_up; s->down = down;
  s->w = {std::get<0>(norm1), wqkv->whole(), bqkv.has_value() ? std::get<0>(*bqkv) : Tensor(), wo->whole(), std::get<0>(norm2),
          gate_up->whole(), down->whole()};
  s->norm_sink[0] = std::get<1>(norm1); s->norm_sink[1] = std::get<1>(norm2);
  if (bqkv.has_value()) s->bias_sink = std::get<1>(*bqkv);
  s->c = {n_q, n_kv, d, max_seqlen, theta, eps, eps};
  if (!layer_takes(x, pos, cu, s->w, s->c)) return c10::nullopt;
  after_start();
  return ShardedLayerFn::apply(x, pos, cu, s, wants_grad(x));
}

}  // namespace

void register_ops(py::module_& m) {
  m.def("kernel_launches", [] { return g_launches.load(std::memory_order_relaxed); });
  m.def("count_launches", [](int n) { count(n); });
  m.def("rmsnorm_fwd", &rmsnorm_fwd);
  m.def("rmsnorm_bwd", &rmsnorm_bwd, py::arg("dy"), py::arg("x"), py::arg("w"), py::arg("rstd"),
        py::arg("fixed_order") = false, py::arg("dres") = py::none(), py::arg("sink") = py::none());
  m.def("rope_qkv", &rope_qkv);
  m.def("swiglu_fwd", &swiglu_fwd);
  m.def("swiglu_bwd", &swiglu_bwd);
  m.def("ce_fwd_bwd", &ce_fwd_bwd, py::arg("logits"), py::arg("labels"), py::arg("loss_scale"), py::arg("loss"),
        py::arg("ignore_index"), py::arg("inv_temp") = 1.0);
  m.def("token_logprobs", &token_logprobs, py::arg("logits"), py::arg("labels"), py::arg("out"), py::arg("ignore_index"),
        py::arg("inv_temp") = 1.0);
  m.def("adamw_step", &adamw_step);
  m.def("cast_f32_to_bf16", &cast_f32_to_bf16);
  m.def("sumsq", &sumsq);
  m.def("gemm", &gemm, py::arg("a"), py::arg("b"), py::arg("c"), py::arg("layout"), py::arg("bias"),
        py::arg("accumulate"), py::arg("residual") = py::none(), py::arg("pair") = -1);
  m.def("gemm_plan", [](int M, int N, int K, int sms) {
    const odc::GemmPlan p = odc::gemm_plan(M, N, K, odc::kBF16, sms);
    return std::make_tuple(p.tiles, p.whole, p.parts, p.scratch_bytes);
  }, py::arg("M"), py::arg("N"), py::arg("K"), py::arg("sms"));  // (tiles, whole ones, parts of each other, scratch) in bf16
  m.def("gemm_group", [](std::vector<std::tuple<Tensor, Tensor, Tensor, std::string, bool, double>> products) {
    std::vector<Product> todo;
    for (auto& [a, b, c, layout, accumulate, scale] : products) {
      int lay = 0;
      while (lay < 3 && layout != kLayoutNames[lay]) ++lay;
      TORCH_CHECK(lay < 3, "gemm_group: unknown layout ", layout);
      todo.push_back({a, b, c, lay, accumulate, scale, {}, {}, accumulate});
    }
    return group_into(todo);
  });  // (a, b, c, layout, accumulate, scale) each; False: not taken as a group, nothing done
  m.def("group_words", []() -> c10::optional<Tensor> {
    unsigned int* words = group_words();
    if (words == nullptr) return c10::nullopt;
    return at::from_blob(words, {odc::kGroupLaunchWords}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, at::cuda::current_device()));
  });  // counters of the current stream's groups; None where every launch brings its own
  using Shape = std::tuple<int, int, int, bool, bool>;   // (M, N, K, fp32, accumulate)
  static const auto shapes_of = [](const std::vector<Shape>& products) {
    TORCH_CHECK(products.size() <= odc::kMaxGroupProducts, "group plan: too many products");
    std::vector<odc::GemmProduct> g(products.size());
    for (size_t i = 0; i < g.size(); ++i) {
      const auto& [M, N, K, f32, accumulate] = products[i];
      g[i].M = M; g[i].N = N; g[i].K = K; g[i].c_kind = f32 ? odc::kF32 : odc::kBF16; g[i].accumulate = accumulate; g[i].scale = 1.f;
    }
    return g;
  };
  static const auto group_plan = [](const std::vector<Shape>& products, int sms) {
    const auto g = shapes_of(products);
    return odc::gemm_group_plan(g.data(), static_cast<int>(g.size()), sms);
  };
  m.def("gemm_group_plan", [](std::vector<Shape> products, int sms) {
    const auto plan = group_plan(products, sms);
    return std::vector<int>(plan.parts, plan.parts + products.size());
  }, py::arg("products"), py::arg("sms"));  // parts of every tile of each product
  m.def("gemm_group_columns", [](std::vector<Shape> products, int sms) {
    const auto plan = group_plan(products, sms);
    return std::vector<int>(plan.columns, plan.columns + products.size());
  }, py::arg("products"), py::arg("sms"));  // columns of a tile of each
  m.def("gemm_group_tiles", [](std::vector<Shape> products, int sms) {
    const auto plan = group_plan(products, sms);
    std::vector<std::tuple<int, int, int>> out;
    for (size_t i = 0; i < products.size(); ++i) out.emplace_back(plan.tiles[i].tiles, plan.tiles[i].whole, plan.tiles[i].parts);
    return out;
  }, py::arg("products"), py::arg("sms"));  // (tiles, whole ones, parts of each other) of each
  m.def("scatter_plan", [](int n_out, int k_in, int tokens, int ranks, int sms) {
    const odc::GemmPlan p = odc::scatter_plan(n_out, k_in, tokens, ranks, sms);
    return std::make_tuple(p.tiles, p.whole, p.parts);
  }, py::arg("n_out"), py::arg("k_in"), py::arg("tokens"), py::arg("ranks"), py::arg("sms"));
  m.def("head_plan", [](int rows, int words, int width, bool gradient, int sms) {
    return odc::logits_stats_pay(rows, words, width, gradient, sms);
  }, py::arg("rows"), py::arg("words"), py::arg("width"), py::arg("gradient"), py::arg("sms"));  // statistics in the product
  // scratch of a product of which every tile is divided; 0 for one of which some or all are whole
  m.def("gemm_split_bytes", [](int M, int N, int K) {
    const odc::GemmPlan p = odc::gemm_plan(M, N, K, odc::kBF16, sm_count());
    return p.whole == 0 ? p.scratch_bytes : 0;
  });
  m.def("attn_fwd", &attn_fwd);
  m.def("attn_bwd", [](Tensor dout, Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor cu_seqlens, int max_seqlen, bool causal,
                       double scale, bool fused_qkv, c10::optional<Tensor> rope_pos, double rope_theta) {
    return attn_bwd(dout, q, k, v, o, lse, cu_seqlens, max_seqlen, causal, scale, fused_qkv, rope_pos.value_or(Tensor()), rope_theta);
  }, py::arg("dout"), py::arg("q"), py::arg("k"), py::arg("v"), py::arg("o"), py::arg("lse"), py::arg("cu_seqlens"),
        py::arg("max_seqlen"), py::arg("causal"), py::arg("scale"), py::arg("fused_qkv"), py::arg("rope_pos") = py::none(),
        py::arg("rope_theta") = 0.0);
  m.def("exp2_poly", &exp2_poly);
  m.def("attn_plan", [](int tokens, int seqs, int longest, int n_q, int n_kv, int d, bool causal, int sms) {
    return std::make_tuple(d == 128 && odc::attn_fwd_pairs(tokens, seqs, longest, n_q, n_kv, causal, sms),
                           odc::attn_bwd_parts(tokens, seqs, longest, n_q, n_kv, d, causal, sms));
  }, py::arg("tokens"), py::arg("seqs"), py::arg("longest"), py::arg("n_q"), py::arg("n_kv"), py::arg("head_dim"),
        py::arg("causal"), py::arg("sms"));  // (forward in pairs of tiles, parts of the backward)
  m.def("kernel_status", &kernel_status);
  m.def("clear_kernel_status", &clear_kernel_status);
  m.def("scale_to_bf16", &scale_to_bf16);
  py::class_<DispatchCounter, c10::intrusive_ptr<DispatchCounter>>(m, "DispatchCounter")
      .def(py::init([] { return c10::make_intrusive<DispatchCounter>(); }))
      .def("take", &DispatchCounter::take);
  py::class_<ShardedMatrix, c10::intrusive_ptr<ShardedMatrix>>(m, "ShardedMatrix")
      .def(py::init([](int64_t id, Tensor shard, Tensor table, Tensor acc_table, Tensor ctr_table, std::vector<int64_t> acc_addrs,
                       int64_t out_features, int64_t index, double grad_scale, c10::intrusive_ptr<DispatchCounter> dispatched) {
        auto p = c10::make_intrusive<ShardedMatrix>();
        p->id = id; p->shard = shard; p->table = table; p->acc_table = acc_table; p->ctr_table = ctr_table;
        p->world = static_cast<int64_t>(acc_addrs.size());
        p->acc_addrs = std::move(acc_addrs);
        p->out_features = out_features; p->rows_per_rank = shard.size(0); p->index = index; p->grad_scale = grad_scale;
        p->dispatched = dispatched;
        if (p->world == 1) p->matrix = shard.narrow(0, 0, out_features);
        return p;
      }))
      .def_readwrite("local_pending", &ShardedMatrix::local_pending);
  m.def("mark_start", &mark_start);
  m.def("after_start", &after_start);
  m.def("set_sync_grads", [](bool on) { g_sync_grads = on; });
  m.def("set_deferred_weight_grad", [](py::object deferred, py::object local_buffer, py::object push_local) {
    if (g_deferred == nullptr) {   // never destroyed: backward threads may outlive the module
      g_deferred = new py::object();
      g_local_buffer = new py::object();
      g_push_local = new py::object();
    }
    *g_deferred = deferred;
    *g_local_buffer = local_buffer;
    *g_push_local = push_local;
  });
  // differentiable forms
  m.def("sharded_linear", &sharded_linear, py::arg("x"), py::arg("bias"), py::arg("residual"), py::arg("matrix"),
        py::arg("bias_sink") = py::none(), py::arg("keep_weight") = false);
  m.def("sharded_mlp", &sharded_mlp, py::arg("x"), py::arg("residual"), py::arg("gate_up"), py::arg("down"));
  m.def("decoder_layer", &decoder_layer);
  m.def("sharded_layer", &sharded_layer);
  m.def("linear", &linear, py::arg("x"), py::arg("w"), py::arg("bias") = py::none(), py::arg("residual") = py::none());
  m.def("rms_norm", &rms_norm, py::arg("x"), py::arg("w"), py::arg("eps"), py::arg("sink") = py::none());
  m.def("rms_norm_residual", &rms_norm_residual, py::arg("x"), py::arg("w"), py::arg("eps"), py::arg("sink") = py::none());
  m.def("rope", &rope);
  m.def("linear_rope", [](Tensor x, Tensor w, c10::optional<Tensor> bias, Tensor pos, int64_t n_q, int64_t n_kv, int64_t d, double theta) {
    return linear_rope(x, w, bias.value_or(Tensor()), pos, n_q, n_kv, d, theta);
  });
  m.def("swiglu", &swiglu);
  m.def("linear_swiglu", &linear_swiglu, py::arg("x"), py::arg("w"));
  m.def("swiglu_product_bwd", &swiglu_product_bwd, py::arg("dy"), py::arg("w"), py::arg("gate_up"));
  m.def("mlp", &mlp, py::arg("x"), py::arg("w_gate_up"), py::arg("w_down"), py::arg("residual") = py::none());
  m.def("attention", &attention);
  m.def("attention_qkv", &attention_qkv);
  m.def("linear_cross_entropy", &linear_cross_entropy);
  m.def("linear_token_logprobs", &linear_token_logprobs);
  m.def("head_keeps_logit_grads", &keeps_logit_grads, py::arg("h"), py::arg("w"), py::arg("chunk"), py::arg("need_dw") = true,
        py::arg("sharded") = true);
  m.def("logit_grads_pay", &logit_grads_pay, py::arg("tokens"), py::arg("words"), py::arg("width"), py::arg("chunk"), py::arg("sharded"),
        py::arg("sms"));
  m.def("loss_and_logit_grads", &loss_and_logit_grads);
  m.def("sharded_head_grads", &sharded_head_grads, py::arg("dlogits"), py::arg("h"), py::arg("w"), py::arg("g"), py::arg("matrix"),
        py::arg("local") = py::none(), py::arg("add") = false);
  m.def("lm_head_loss", &lm_head_loss, py::arg("h"), py::arg("w"), py::arg("labels"), py::arg("loss_scale"),
        py::arg("ignore_index"), py::arg("chunk"), py::arg("need_dh"), py::arg("need_dw"), py::arg("dw_out") = py::none());
}

}  // namespace odc_bind
