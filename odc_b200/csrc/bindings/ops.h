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

void register_ops(py::module_& m);  // ops.cpp: the decoder's differentiable ops

}  // namespace odc_bind
