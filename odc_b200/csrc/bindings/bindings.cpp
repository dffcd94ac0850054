// Python bindings of the heap, the communication primitives and the fused GEMMs: tensors in, raw pointers + current
// stream out to the launchers in kernels/api.h.  The decoder's differentiable ops are in ops.cpp.
#include "ops.h"

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>

#include "../heap/symm_heap.h"

namespace odc_bind {

int sm_count() {
  static int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  return n;
}

// Ring of self-resetting completion counters used by scatter_accumulate launches.  A slot is zero again once the
// last CTA of its launch has finished, so a slot may be handed out again only after that launch has run: with
// kDoneSlots slots this holds while fewer than kDoneSlots such launches are queued or running per device.  CUDA
// itself blocks the launching thread long before that many kernels are pending on a device (its launch queue holds
// on the order of a thousand), which is what bounds the number in flight.
constexpr unsigned long long kDoneSlots = 16384;
unsigned int* next_done_slot(int device) {
  static std::mutex mu;
  static std::unordered_map<int, Tensor> rings;
  static std::unordered_map<int, unsigned long long> seq;
  std::lock_guard<std::mutex> lock(mu);
  auto it = rings.find(device);
  if (it == rings.end()) {
    auto t = torch::zeros({static_cast<int64_t>(kDoneSlots)}, torch::dtype(torch::kInt32).device(torch::kCUDA, device));
    it = rings.emplace(device, t).first;
    seq[device] = 0;
  }
  unsigned long long s = seq[device]++;
  return reinterpret_cast<unsigned int*>(it->second.data_ptr<int>()) + (s % kDoneSlots);
}

Tensor& device_status(int device) {
  static std::mutex mu;
  static std::unordered_map<int, Tensor> st;
  std::lock_guard<std::mutex> lock(mu);
  auto it = st.find(device);
  if (it == st.end()) it = st.emplace(device, torch::zeros({4}, torch::dtype(torch::kInt32).device(torch::kCUDA, device))).first;
  return it->second;
}

// ---------------------------------------------------------------------------------------- GEMMs fused with the primitives
void gemm_wgrad_scatter(Tensor dy, Tensor x, Tensor acc_table, Tensor ctr_table, int64_t acc_offset,
                        int64_t rows_per_rank, double scale) {
  c10::cuda::CUDAGuard g(dy.device());
  odc::bind_device(dy.get_device());
  TORCH_CHECK(dy.dim() == 2 && x.dim() == 2 && dy.size(0) == x.size(0), "wgrad_scatter: dy [T,N], x [T,K]");
  TORCH_CHECK(dy.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16, "wgrad_scatter: bf16 inputs");
  TORCH_CHECK(dy.stride(1) == 1 && x.stride(1) == 1, "wgrad_scatter: innermost stride must be 1");
  check(odc::gemm_wgrad_scatter(dy.data_ptr(), x.data_ptr(), dy.size(0), dy.size(1), x.size(1), dy.stride(0),
                                x.stride(0), reinterpret_cast<const long long*>(acc_table.data_ptr<int64_t>()),
                                reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()), acc_offset,
                                static_cast<int>(rows_per_rank), static_cast<int>(acc_table.numel()),
                                static_cast<float>(scale), next_done_slot(dy.get_device()),
                                device_status(dy.get_device()).data_ptr<int>(), sm_count(), cur_stream()),
        "gemm_wgrad_scatter");
}

bool gemm_wgrad_scatter_tma(Tensor dy, Tensor x, std::vector<int64_t> acc_addrs, Tensor ctr_table, int64_t acc_offset,
                            int64_t rows_per_rank, double scale, int start_rank) {
  c10::cuda::CUDAGuard g(dy.device());
  odc::bind_device(dy.get_device());
  TORCH_CHECK(dy.dim() == 2 && x.dim() == 2 && dy.size(0) == x.size(0), "wgrad_scatter: dy [T,N], x [T,K]");
  TORCH_CHECK(dy.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16, "wgrad_scatter: bf16 inputs");
  TORCH_CHECK(dy.stride(1) == 1 && x.stride(1) == 1, "wgrad_scatter: innermost stride must be 1");
  std::vector<long long> addrs(acc_addrs.begin(), acc_addrs.end());
  // parts of one tile meet in the accumulator in any order
  const char* slots = std::getenv("ODC_DETERMINISTIC");
  const bool fixed_order = at::globalContext().deterministicAlgorithms() ||
                           (slots != nullptr && *slots != 0 && std::strcmp(slots, "0") != 0 && std::strcmp(slots, "false") != 0);
  cudaError_t e = odc::gemm_wgrad_scatter_tma(
      dy.data_ptr(), x.data_ptr(), dy.size(0), dy.size(1), x.size(1), dy.stride(0), x.stride(0), addrs.data(),
      reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()), acc_offset, static_cast<int>(rows_per_rank),
      static_cast<int>(addrs.size()), static_cast<float>(scale), next_done_slot(dy.get_device()),
      device_status(dy.get_device()).data_ptr<int>(), sm_count(), cur_stream(), start_rank, fixed_order);
  if (e == cudaErrorNotSupported) return false;  // shape not eligible: the caller uses the red.add variant
  check(e, "gemm_wgrad_scatter_tma");
  return true;
}

Tensor gemm_gather(Tensor x, Tensor shard_table, Tensor w_local, c10::optional<Tensor> bias, int64_t rows_per_rank,
                   int start_rank, c10::optional<Tensor> residual) {
  c10::cuda::CUDAGuard g(x.device());
  odc::bind_device(x.get_device());
  TORCH_CHECK(x.dim() == 2 && w_local.dim() == 2 && x.size(1) == w_local.size(1), "gemm_gather: x [M,K], w_local [N,K]");
  TORCH_CHECK(x.scalar_type() == at::kBFloat16 && w_local.scalar_type() == at::kBFloat16 && w_local.is_contiguous() &&
                  x.stride(1) == 1, "gemm_gather: bf16, contiguous weight buffer");
  const int M = x.size(0), K = x.size(1), N = w_local.size(0);
  auto y = torch::empty({M, N}, x.options());
  auto flags = torch::empty({(N + 255) / 256}, x.options().dtype(at::kInt));
  const void* bias_ptr = nullptr;
  if (bias.has_value()) {
    TORCH_CHECK(bias->scalar_type() == at::kBFloat16 && bias->numel() == N, "gemm_gather: bias bf16 [N]");
    bias_ptr = bias->data_ptr();
  }
  const void* res_ptr = nullptr;
  long long ldr = 0;
  if (residual.has_value()) {
    TORCH_CHECK(residual->scalar_type() == at::kBFloat16 && residual->dim() == 2 && residual->size(0) == M &&
                    residual->size(1) == N && residual->stride(1) == 1, "gemm_gather: residual bf16 [M,N]");
    res_ptr = residual->data_ptr();
    ldr = residual->stride(0);
  }
  check(odc::gemm_gather_nt(x.data_ptr(), reinterpret_cast<const long long*>(shard_table.data_ptr<int64_t>()),
                            w_local.data_ptr(), y.data_ptr(), bias_ptr, M, N, K, x.stride(0), y.stride(0),
                            static_cast<int>(rows_per_rank), static_cast<int>(shard_table.numel()), start_rank,
                            reinterpret_cast<unsigned int*>(flags.data_ptr<int>()),
                            device_status(x.get_device()).data_ptr<int>(), sm_count(), cur_stream(), res_ptr, ldr),
        "gemm_gather");
  return y;
}

Tensor gemm_gather_dgrad(Tensor dy, Tensor shard_table, Tensor w_local, int64_t rows_per_rank, int start_rank) {
  c10::cuda::CUDAGuard g(dy.device());
  odc::bind_device(dy.get_device());
  TORCH_CHECK(dy.dim() == 2 && w_local.dim() == 2 && dy.size(1) == w_local.size(0),
              "gemm_gather_dgrad: dy [M,N], w_local [N,K]");
  TORCH_CHECK(dy.scalar_type() == at::kBFloat16 && w_local.scalar_type() == at::kBFloat16 && w_local.is_contiguous() &&
                  dy.stride(1) == 1, "gemm_gather_dgrad: bf16, contiguous weight buffer");
  const int M = dy.size(0), N = dy.size(1), K = w_local.size(1);
  auto dx = torch::empty({M, K}, dy.options());
  auto flags = torch::empty({(N + 255) / 256}, dy.options().dtype(at::kInt));
  check(odc::gemm_gather_nn(dy.data_ptr(), reinterpret_cast<const long long*>(shard_table.data_ptr<int64_t>()),
                            w_local.data_ptr(), dx.data_ptr(), M, N, K, dy.stride(0), dx.stride(0),
                            static_cast<int>(rows_per_rank), static_cast<int>(shard_table.numel()),
                            reinterpret_cast<unsigned int*>(flags.data_ptr<int>()),
                            device_status(dy.get_device()).data_ptr<int>(), sm_count(), cur_stream(), start_rank),
        "gemm_gather_dgrad");
  return dx;
}

}  // namespace odc_bind

namespace {

using namespace odc_bind;

// ---------------------------------------------------------------------------------------- heap
uintptr_t heap_create(int rank, int world, int device, size_t bytes, const std::string& mode,
                      const std::string& token) {
  return reinterpret_cast<uintptr_t>(odc::heap_create(rank, world, device, bytes, mode, token));
}
odc::Heap* H(uintptr_t h) { return reinterpret_cast<odc::Heap*>(h); }

Tensor tensor_from_ptr(uintptr_t ptr, int64_t numel, at::ScalarType dtype, int device) {
  auto opts = torch::TensorOptions().dtype(dtype).device(torch::kCUDA, device);
  return torch::from_blob(reinterpret_cast<void*>(ptr), {numel}, [](void*) {}, opts);
}

py::bytes get_ipc_handle(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "get_ipc_handle expects a CUDA tensor");
  c10::cuda::CUDAGuard g(t.device());
  odc::bind_device(t.get_device());
  return py::bytes(odc::ipc_export(t.data_ptr()));
}

Tensor reconstruct_tensor(const std::string& blob, std::vector<int64_t> shape, at::ScalarType dtype) {
  void* p = odc::ipc_import(blob);
  int dev = 0;
  cudaGetDevice(&dev);
  auto opts = torch::TensorOptions().dtype(dtype).device(torch::kCUDA, dev);
  return torch::from_blob(p, shape, [](void*) {}, opts);
}

// ---------------------------------------------------------------------------------------- comm
void gather(Tensor out2d, Tensor table, int64_t n, at::ScalarType src_dtype, int my_index, bool checkb,
            Tensor status, int64_t src_region_elems) {
  c10::cuda::CUDAGuard g(out2d.device());
  odc::bind_device(out2d.get_device());
  const int nranks = static_cast<int>(table.numel());
  TORCH_CHECK(out2d.is_contiguous() && out2d.numel() == n * nranks, "gather: bad output shape");
  const int ssz = static_cast<int>(c10::elementSize(src_dtype));
  const int dsz = static_cast<int>(out2d.element_size());
  const bool narrow = (src_dtype == at::kFloat && out2d.scalar_type() == at::kBFloat16);
  TORCH_CHECK(narrow || src_dtype == out2d.scalar_type(), "gather: only same-dtype or fp32->bf16");
  check(odc::launch_gather(table.data_ptr<int64_t>() ? reinterpret_cast<const long long*>(table.data_ptr<int64_t>()) : nullptr,
                           out2d.data_ptr(), static_cast<size_t>(n), ssz, dsz, narrow, nranks, my_index, checkb,
                           status.data_ptr<int>(), sm_count(), cur_stream(),
                           checkb ? static_cast<size_t>(src_region_elems) : 0),
        "gather launch");
}

void scatter_accumulate(Tensor inp2d, Tensor acc_table, Tensor ctr_table, int64_t n, at::ScalarType acc_dtype,
                        int my_index, double scale, bool checkb, Tensor status, int64_t acc_region_elems,
                        c10::optional<Tensor> scale_tensor) {
  c10::cuda::CUDAGuard g(inp2d.device());
  if (scale_tensor.has_value())
    TORCH_CHECK(scale_tensor->is_cuda() && scale_tensor->scalar_type() == at::kFloat && scale_tensor->numel() == 1 &&
                    acc_dtype == at::kFloat, "scatter_accumulate: the scale tensor is one fp32 value on the device");
  odc::bind_device(inp2d.get_device());
  const int nranks = static_cast<int>(acc_table.numel());
  TORCH_CHECK(inp2d.is_contiguous() && inp2d.numel() == n * nranks, "scatter_accumulate: bad input shape");
  check(odc::launch_scatter_accumulate(inp2d.data_ptr(), kind_of(inp2d.scalar_type()),
                                       reinterpret_cast<const long long*>(acc_table.data_ptr<int64_t>()),
                                       kind_of(acc_dtype),
                                       reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()),
                                       static_cast<size_t>(n), nranks, my_index, static_cast<float>(scale),
                                       next_done_slot(inp2d.get_device()), sm_count(), cur_stream(),
                                       status.data_ptr<int>(), checkb ? acc_region_elems : 0,
                                       scale_tensor.has_value() ? scale_tensor->data_ptr<float>() : nullptr),
        "scatter_accumulate launch");
}

bool scatter_accumulate_segments(std::vector<Tensor> grads, std::vector<int64_t> chunk_numels,
                                 std::vector<int64_t> dst_offsets, Tensor acc_table, Tensor ctr_table,
                                 at::ScalarType acc_dtype, int my_index, double scale, bool checkb,
                                 c10::optional<Tensor> status, int64_t acc_region_elems) {
  // Returns false (nothing launched) when the list does not fit this path; the caller then flattens the gradients.
  if (grads.empty() || grads.size() > static_cast<size_t>(odc::kMaxScatterSegments) || acc_dtype != at::kFloat) return false;
  TORCH_CHECK(grads.size() == chunk_numels.size() && grads.size() == dst_offsets.size(),
              "scatter_accumulate_segments: one chunk size and one offset per gradient");
  const auto dt = grads[0].scalar_type();
  if (dt != at::kFloat && dt != at::kBFloat16) return false;
  odc::ScatterSegments segs{};
  segs.count = static_cast<int>(grads.size());
  for (size_t i = 0; i < grads.size(); ++i) {
    const Tensor& g = grads[i];
    if (!g.is_cuda() || !g.is_contiguous() || g.scalar_type() != dt || g.device() != grads[0].device()) return false;
    segs.src[i] = g.data_ptr();
    segs.chunk[i] = chunk_numels[i];
    segs.total[i] = g.numel();
    segs.dst[i] = dst_offsets[i];
  }
  c10::cuda::CUDAGuard guard(grads[0].device());
  odc::bind_device(grads[0].get_device());
  const int nranks = static_cast<int>(acc_table.numel());
  check(odc::launch_scatter_accumulate_segments(segs, kind_of(dt),
                                                reinterpret_cast<const long long*>(acc_table.data_ptr<int64_t>()),
                                                reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()), nranks,
                                                my_index, static_cast<float>(scale),
                                                next_done_slot(grads[0].get_device()), sm_count(), cur_stream(),
                                                (checkb && status.has_value()) ? acc_region_elems : 0,
                                                status.has_value() ? status->data_ptr<int>() : nullptr),
        "scatter_accumulate_segments launch");
  return true;
}

// rows of a bf16 lookup gradient [T, H] into the fp32 accumulators of the ranks that own the looked-up rows
void embedding_scatter(Tensor ids, Tensor dx, Tensor acc_table, Tensor ctr_table, int64_t rows_per_rank, int64_t vocab,
                       double scale) {
  c10::cuda::CUDAGuard g(dx.device());
  odc::bind_device(dx.get_device());
  TORCH_CHECK(ids.scalar_type() == at::kLong && ids.is_contiguous() && dx.dim() == 2 && dx.is_contiguous() &&
                  dx.scalar_type() == at::kBFloat16 && ids.numel() == dx.size(0) && dx.size(1) % 8 == 0,
              "embedding_scatter: int64 ids [T], contiguous bf16 gradient [T, H], H a multiple of 8");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(dx.data_ptr()) % 16 == 0, "embedding_scatter: the gradient starts on 16 bytes");
  TORCH_CHECK(vocab <= rows_per_rank * acc_table.numel(), "embedding_scatter: more rows than the owners hold");
  check(odc::launch_embedding_scatter(reinterpret_cast<const long long*>(ids.data_ptr<int64_t>()), dx.data_ptr(),
                                      static_cast<int>(dx.size(0)), static_cast<int>(dx.size(1)),
                                      reinterpret_cast<const long long*>(acc_table.data_ptr<int64_t>()),
                                      reinterpret_cast<const long long*>(ctr_table.data_ptr<int64_t>()), rows_per_rank, vocab,
                                      static_cast<int>(acc_table.numel()), static_cast<float>(scale),
                                      next_done_slot(dx.get_device()), sm_count(), cur_stream()),
        "embedding_scatter launch");
}

void wait_counter(Tensor counter, int64_t expected, int64_t timeout_ms, Tensor status) {
  c10::cuda::CUDAGuard g(counter.device());
  odc::bind_device(counter.get_device());
  check(odc::launch_wait_counter(counter.data_ptr(), static_cast<unsigned long long>(expected),
                                 static_cast<unsigned long long>(timeout_ms) * 1000000ull, status.data_ptr<int>(),
                                 cur_stream()),
        "wait_counter launch");
}

odc::PostedCounts posted(const std::vector<int64_t>& slot_addrs, const std::vector<int64_t>& counts, int64_t epoch) {
  TORCH_CHECK(slot_addrs.size() == counts.size() && slot_addrs.size() <= size_t(odc::kMaxPostedCounts),
              "post_counts: at most ", odc::kMaxPostedCounts, " owners");
  odc::PostedCounts pc{};
  pc.n = static_cast<int>(slot_addrs.size());
  for (int i = 0; i < pc.n; ++i) {
    TORCH_CHECK(slot_addrs[i] != 0 && (slot_addrs[i] & 7) == 0, "post_counts: bad slot address");
    TORCH_CHECK(counts[i] >= 0 && counts[i] < (int64_t(1) << 32), "post_counts: count out of range");
    pc.slot_addr[i] = slot_addrs[i];
    pc.value[i] = (static_cast<unsigned long long>(epoch) << 32) | static_cast<unsigned long long>(counts[i]);
  }
  return pc;
}

void post_counts(std::vector<int64_t> slot_addrs, std::vector<int64_t> counts, int64_t epoch, int device) {
  c10::cuda::CUDAGuard g(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)));
  odc::bind_device(device);
  check(odc::launch_post_counts(posted(slot_addrs, counts, epoch), cur_stream()), "post_counts launch");
}

// post_counts + wait_posted in one launch; returns {code, detail, observed} of the device's status word once all that was queued on
// the current stream before, and the waits, are done
std::tuple<int, int, int> post_and_wait(std::vector<int64_t> slot_addrs, std::vector<int64_t> counts, int64_t epoch, Tensor slots,
                                        int64_t nprod, Tensor counter, int64_t timeout_ms, Tensor status, Tensor status_host) {
  c10::cuda::CUDAGuard g(counter.device());
  odc::bind_device(counter.get_device());
  TORCH_CHECK(slots.scalar_type() == at::kLong && slots.numel() >= nprod, "post_and_wait: int64 slots, one per producer");
  TORCH_CHECK(status_host.scalar_type() == at::kInt && status_host.numel() >= 4 && status_host.is_pinned(),
              "post_and_wait: four pinned ints");
  auto* word = reinterpret_cast<volatile unsigned long long*>(status_host.data_ptr<int>());
  unsigned long long* mapped = nullptr;
  check(cudaHostGetDevicePointer(reinterpret_cast<void**>(&mapped), status_host.data_ptr<int>(), 0), "post_and_wait: status buffer");
  const cudaStream_t stream = cur_stream();
  *word = 0;
  check(odc::launch_post_and_wait(posted(slot_addrs, counts, epoch), slots.data_ptr(), static_cast<int>(nprod),
                                  static_cast<unsigned long long>(epoch), counter.data_ptr(),
                                  static_cast<unsigned long long>(timeout_ms) * 1000000ull, status.data_ptr<int>(), mapped, stream),
        "post_and_wait launch");
  const unsigned long long done = static_cast<unsigned long long>(epoch) << 8;
  cudaError_t e = cudaSuccess;
  int seen[4] = {0, 0, 0, 0};
  {
    py::gil_scoped_release nogil;
    // The word is there some microseconds before the launch has retired and a synchronisation has returned.  A longer wait is the
    // driver's, which also notices a stream that failed.
    const auto t0 = std::chrono::steady_clock::now();
    unsigned long long v = *word;
    while (v != done && std::chrono::steady_clock::now() - t0 < std::chrono::microseconds(200)) v = *word;
    if (v != done) {
      e = cudaStreamSynchronize(stream);
      if (e == cudaSuccess && *word != done) {
        e = cudaMemcpyAsync(seen, status.data_ptr<int>(), sizeof(seen), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
      }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
  }
  check(e, "post_and_wait");
  return {seen[0], seen[1], seen[2]};
}

void wait_posted(Tensor slots, int64_t nprod, int64_t epoch, Tensor counter, int64_t timeout_ms, Tensor status,
                 Tensor expected_out) {
  c10::cuda::CUDAGuard g(counter.device());
  odc::bind_device(counter.get_device());
  TORCH_CHECK(slots.scalar_type() == at::kLong && slots.numel() >= nprod && expected_out.scalar_type() == at::kLong,
              "wait_posted: int64 slots (one per producer) and an int64 output word");
  check(odc::launch_wait_posted(slots.data_ptr(), static_cast<int>(nprod), static_cast<unsigned long long>(epoch),
                                counter.data_ptr(), static_cast<unsigned long long>(timeout_ms) * 1000000ull,
                                status.data_ptr<int>(), reinterpret_cast<unsigned long long*>(expected_out.data_ptr()),
                                cur_stream()),
        "wait_posted launch");
}

// --- single-primitive test entry points: addresses are plain integers so peers' mappings can be passed
void put_block(uintptr_t remote_dst, Tensor local_src) {
  c10::cuda::CUDAGuard g(local_src.device());
  odc::bind_device(local_src.get_device());
  check(odc::launch_put_block(reinterpret_cast<void*>(remote_dst), local_src.data_ptr(), local_src.nbytes(), cur_stream()),
        "put_block");
}
void get_block(Tensor local_dst, uintptr_t remote_src) {
  c10::cuda::CUDAGuard g(local_dst.device());
  odc::bind_device(local_dst.get_device());
  check(odc::launch_get_block(local_dst.data_ptr(), reinterpret_cast<const void*>(remote_src), local_dst.nbytes(),
                              cur_stream()), "get_block");
}
void scalar_put_get(uintptr_t remote_word, int value, Tensor readback) {
  c10::cuda::CUDAGuard g(readback.device());
  odc::bind_device(readback.get_device());
  check(odc::launch_scalar_put_get(reinterpret_cast<int*>(remote_word), value, readback.data_ptr<int>(), cur_stream()),
        "scalar_put_get");
}
void atomic_test(Tensor word, Tensor cas_seen, Tensor swap_seen, int expected_old, int cas_new, int swap_new) {
  c10::cuda::CUDAGuard g(word.device());
  odc::bind_device(word.get_device());
  check(odc::launch_atomic_test(word.data_ptr<int>(), cas_seen.data_ptr<int>(), swap_seen.data_ptr<int>(),
                                static_cast<int>(cas_seen.numel()), expected_old, cas_new, swap_new, cur_stream()),
        "atomic_test");
}
void grid_barrier_test(Tensor counter, Tensor slots, Tensor out, int64_t timeout_ms, Tensor status) {
  c10::cuda::CUDAGuard g(out.device());
  odc::bind_device(out.get_device());
  TORCH_CHECK(out.numel() <= sm_count(), "grid barrier needs co-resident CTAs: at most one per SM");
  check(odc::launch_grid_barrier_test(reinterpret_cast<unsigned int*>(counter.data_ptr<int>()), slots.data_ptr<int>(),
                                      out.data_ptr<int>(), static_cast<int>(out.numel()),
                                      static_cast<unsigned long long>(timeout_ms) * 1000000ull, status.data_ptr<int>(),
                                      cur_stream()), "grid_barrier_test");
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("heap_create", &heap_create);
  m.def("heap_grow", [](uintptr_t h, size_t n) { odc::heap_grow(H(h), n); }, py::call_guard<py::gil_scoped_release>());
  m.def("heap_ipc_handle", [](uintptr_t h) { return py::bytes(odc::heap_ipc_handle(H(h))); });
  m.def("heap_ipc_open", [](uintptr_t h, int r, const std::string& b) { odc::heap_ipc_open(H(h), r, b); });
  m.def("heap_base", [](uintptr_t h, int r) { return odc::heap_base(H(h), r); });
  m.def("heap_mapped", [](uintptr_t h) { return odc::heap_mapped(H(h)); });
  m.def("heap_destroy", [](uintptr_t h) { odc::heap_destroy(H(h)); });
  m.def("tensor_from_ptr", &tensor_from_ptr);
  m.def("get_ipc_handle", &get_ipc_handle);
  m.def("reconstruct_tensor", &reconstruct_tensor);
  // the trailing *_region_elems arguments are the DECLARED lengths the debug checks (check = true) hold the launch to
  m.def("gather", &gather, py::arg("out2d"), py::arg("table"), py::arg("n"), py::arg("src_dtype"), py::arg("my_index"),
        py::arg("check"), py::arg("status"), py::arg("src_region_elems") = 0);
  m.def("scatter_accumulate", &scatter_accumulate, py::arg("inp2d"), py::arg("acc_table"), py::arg("ctr_table"),
        py::arg("n"), py::arg("acc_dtype"), py::arg("my_index"), py::arg("scale"), py::arg("check"), py::arg("status"),
        py::arg("acc_region_elems") = 0, py::arg("scale_tensor") = py::none());
  m.def("scatter_accumulate_segments", &scatter_accumulate_segments, py::arg("grads"), py::arg("chunk_numels"),
        py::arg("dst_offsets"), py::arg("acc_table"), py::arg("ctr_table"), py::arg("acc_dtype"), py::arg("my_index"),
        py::arg("scale"), py::arg("check") = false, py::arg("status") = py::none(), py::arg("acc_region_elems") = 0);
  m.def("embedding_scatter", &embedding_scatter);
  m.def("wait_counter", &wait_counter);
  m.def("post_counts", &post_counts);
  m.def("wait_posted", &wait_posted);
  m.def("post_and_wait", &post_and_wait);
  m.def("put_block", &put_block);
  m.def("get_block", &get_block);
  m.def("scalar_put_get", &scalar_put_get);
  m.def("atomic_test", &atomic_test);
  m.def("grid_barrier_test", &grid_barrier_test);
  m.def("gemm_wgrad_scatter", &gemm_wgrad_scatter);
  m.def("gemm_wgrad_scatter_tma", &gemm_wgrad_scatter_tma, py::arg("dy"), py::arg("x"), py::arg("acc_addrs"),
        py::arg("ctr_table"), py::arg("acc_offset"), py::arg("rows_per_rank"), py::arg("scale"), py::arg("start_rank") = 0);
  m.def("gemm_gather", &gemm_gather, py::arg("x"), py::arg("shard_table"), py::arg("w_local"), py::arg("bias"),
        py::arg("rows_per_rank"), py::arg("start_rank"), py::arg("residual") = py::none());
  m.def("gemm_gather_dgrad", &gemm_gather_dgrad, py::arg("dy"), py::arg("shard_table"), py::arg("w_local"),
        py::arg("rows_per_rank"), py::arg("start_rank") = 0);
  m.def("sm_count", &sm_count);
  register_ops(m);
}
