// Shared by the operator registrations (iex_torch_ext.cpp) and the autograd layer (iex_autograd.cpp).
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>

#include <tuple>

#include "iex_b200.h"

namespace iex_torch {

inline void* stream_of(const at::Tensor& t) {
  return static_cast<void*>(at::cuda::getCurrentCUDAStream(t.get_device()).stream());
}

inline void check_status(int st, const char* what) {
  TORCH_CHECK(st == 0, what, " failed with status ", st, ": ", iex_error_string(st));
}

// Uninitialised tensor of `like`'s type and device from the caching allocator, without the dispatcher.
at::Tensor empty(const at::Tensor& like, at::IntArrayRef sizes);
at::Tensor empty_bytes(const at::Tensor& like, int64_t bytes);

inline void check_common(std::initializer_list<std::pair<const char*, const at::Tensor*>> named) {
  const at::Tensor* first = nullptr;
  for (const auto& [name, t] : named) {
    TORCH_CHECK(t->is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t->is_contiguous(), name, " must be a contiguous tensor");
    TORCH_CHECK(!t->is_sparse(), name, " must be a dense tensor");
    if (first == nullptr) first = t;
    TORCH_CHECK(t->device() == first->device(), name, " should be in the same device as the first argument");
  }
}

// `t` is read on the current stream although its owner may let go of it at any time (nothing to do on the stream it was
// allocated on).
inline void mark_stream(const at::Tensor& t) {
  c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), at::cuda::getCurrentCUDAStream(t.get_device()));
}

// Operator implementations (iex_torch_ext.cpp)
at::Tensor spmm_matrix(const at::Tensor& b, const at::Tensor& row_indices, const at::Tensor& values,
                       const at::Tensor& row_offsets, const at::Tensor& column_indices, int64_t m);
at::Tensor sddmm_matrix(const at::Tensor& a, const at::Tensor& b, const at::Tensor& row_indices,
                        const at::Tensor& row_offsets, const at::Tensor& column_indices);
at::Tensor spmm_tc_half(const at::Tensor& x, const at::Tensor& row_offsets, const at::Tensor& values,
                        const at::Tensor& column_indices, int64_t m);
at::Tensor linear_fp16(const at::Tensor& input, const at::Tensor& weight);
at::Tensor linear_fp16_dgrad(const at::Tensor& grad, const at::Tensor& weight);
at::Tensor linear_fp16_wgrad(const at::Tensor& grad, const at::Tensor& input);
std::tuple<at::Tensor, at::Tensor> fused_spmm_linear_half(const at::Tensor& x, const at::Tensor& row_offsets,
                                                          const at::Tensor& values, const at::Tensor& column_indices,
                                                          int64_t m, const at::Tensor& weight);
// With IEX_VALIDATE_CSR=1: device-side check of a CSR argument before it is used.
void maybe_validate(const at::Tensor& row_offsets, const at::Tensor& column_indices, int64_t m, int64_t k,
                    const at::Tensor* row_indices, bool require_ascending);

}  // namespace iex_torch
