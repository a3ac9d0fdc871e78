// Arrays of the host (NumPy buffers) to and from CUDA tensors, with the element conversions the reference-shaped
// interface needs (64-bit indices to bytes and back, float widths).
#pragma once
#include <ATen/ATen.h>

#include <vector>

namespace tqhost {

enum class Elem { F16, F32, F64, I64, I32, U8, I8 };

size_t elem_size(Elem e);
at::ScalarType scalar_type(Elem e);

struct HostArray {
  void* data;
  int64_t count;
  Elem elem;
};

// src, converted to dst's type element by element, into the contiguous CUDA tensor dst.  Asynchronous for the device;
// when it returns src may be changed.
void to_device(const HostArray& src, const at::Tensor& dst);

// contiguous CUDA tensors into host arrays, converted to their types; returns when all have arrived
void to_host(const std::vector<std::pair<at::Tensor, HostArray>>& jobs);

}  // namespace tqhost
