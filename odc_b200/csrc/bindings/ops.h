// Shared between the binding files: small helpers on tensors, streams and per-device state.
#pragma once
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../kernels/api.h"
#include "../kernels/tensor_map.h"

namespace odc_bind {

namespace py = pybind11;
using torch::Tensor;

inline void check(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e));
}
int sm_count();
inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }
inline int kind_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return odc::kF32;
    case at::kBFloat16: return odc::kBF16;
    case at::kHalf: return odc::kF16;
    default: TORCH_CHECK(false, "unsupported dtype ", t);
  }
}
unsigned int* next_done_slot(int device);
Tensor& device_status(int device);  // the one status word of a device, shared by every kernel of the package

// GEMMs fused with the primitives (bindings.cpp)
void gemm_wgrad_scatter(Tensor dy, Tensor x, Tensor acc_table, Tensor ctr_table, int64_t acc_offset, int64_t rows_per_rank,
                        double scale);
bool gemm_wgrad_scatter_tma(Tensor dy, Tensor x, std::vector<int64_t> acc_addrs, Tensor ctr_table, int64_t acc_offset,
                            int64_t rows_per_rank, double scale, int start_rank);
Tensor gemm_gather(Tensor x, Tensor shard_table, Tensor w_local, c10::optional<Tensor> bias, int64_t rows_per_rank,
                   int start_rank, c10::optional<Tensor> residual);
Tensor gemm_gather_dgrad(Tensor dy, Tensor shard_table, Tensor w_local, int64_t rows_per_rank, int start_rank);

void register_ops(py::module_& m);  // ops.cpp: the decoder's differentiable ops

}  // namespace odc_bind
