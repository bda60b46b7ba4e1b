// The products of torch_binding.cpp as functions: what the operators `multiply` / `multiply_frozen` / `multiply_planned`
// do on CUDA tensors, with all their checks. torch_direct.cpp calls them without the operator dispatcher.
#pragma once

#include <ATen/core/Tensor.h>

#include <cstdint>

namespace macko_torch {

// y[rows] for V[cols]. `flags`: MACKO_SPMV_MATRIX_IMMUTABLE, MACKO_SPMV_ROWS_EVEN.
at::Tensor multiply_flags(const at::Tensor &values, const at::Tensor &deltas, const at::Tensor &ri, int64_t rows, int64_t cols,
                          const at::Tensor &V, uint32_t flags);

at::Tensor multiply_planned_cuda(const at::Tensor &values, const at::Tensor &deltas, const at::Tensor &ri, int64_t rows, int64_t cols,
                                 const at::Tensor &plan, int64_t virtual_rows, int64_t segment_elements, int64_t split_rows,
                                 const at::Tensor &V, bool frozen);

// y[batch, rows] for V[batch, cols] over the matrix's column windows.
at::Tensor multiply_windowed_cuda(const at::Tensor &values, const at::Tensor &deltas, const at::Tensor &ri, int64_t rows, int64_t cols,
                                  const at::Tensor &windows, const at::Tensor &V, bool frozen);

// Dense [rows, cols] of a compressed matrix.
at::Tensor decompress_cuda(const at::Tensor &values, const at::Tensor &deltas, const at::Tensor &ri, int64_t rows, int64_t cols);

}  // namespace macko_torch
