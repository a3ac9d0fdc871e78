// A copy between pageable memory and the GPU goes through the driver's own staging buffer on one thread (3-10 GB/s), and a
// change of type around it -- 64-bit indices on the host are bytes on the device -- was a second and third pass on one
// thread, most of it page faults of the new array.  Here the conversion is the pass between the caller's array and a pinned
// staging buffer, done by torch's intra-op threads in pieces of a few MB while the neighbouring piece is on the bus: the
// index array of 65,536 x 128 vectors travels as 8 MB instead of 67, and the threads share the page faults.  The staging
// buffers come from torch's pinned allocator (two pieces per call), which keeps and reuses them.
#include "tq_host_copy.h"

#include <ATen/Parallel.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDAStream.h>
#include <string.h>

namespace tqhost {

size_t elem_size(Elem e) {
  switch (e) {
    case Elem::F64: case Elem::I64: return 8;
    case Elem::F32: case Elem::I32: return 4;
    case Elem::F16: return 2;
    default: return 1;
  }
}

at::ScalarType scalar_type(Elem e) {
  switch (e) {
    case Elem::F64: return at::kDouble;
    case Elem::F32: return at::kFloat;
    case Elem::F16: return at::kHalf;
    case Elem::I64: return at::kLong;
    case Elem::I32: return at::kInt;
    case Elem::U8: return at::kByte;
    default: return at::kChar;
  }
}

namespace {

constexpr int64_t PIECE = 4 << 20;    // bytes of the host array per piece: short against the whole, long against a launch
constexpr int64_t SMALL = 256 << 10;  // arrays up to this size travel in one piece, several of them behind one wait
constexpr int64_t GRAIN = 64 << 10;   // bytes per thread below which more threads do not pay

Elem elem_of(at::ScalarType t) {
  switch (t) {
    case at::kDouble: return Elem::F64;
    case at::kFloat: return Elem::F32;
    case at::kHalf: return Elem::F16;
    case at::kLong: return Elem::I64;
    case at::kInt: return Elem::I32;
    case at::kByte: return Elem::U8;
    case at::kChar: return Elem::I8;
    default: TORCH_CHECK(false, "no host copy for ", t);
  }
}

template <typename S, typename D>
void convert_as(const void* src, void* dst, int64_t n) {
  const S* s = static_cast<const S*>(src);
  D* d = static_cast<D*>(dst);
  at::parallel_for(0, n, GRAIN / (int64_t)(sizeof(S) > sizeof(D) ? sizeof(S) : sizeof(D)), [=](int64_t lo, int64_t hi) {
    if constexpr (std::is_same_v<S, D>) {
      memcpy(d + lo, s + lo, (size_t)(hi - lo) * sizeof(S));
    } else {
      for (int64_t i = lo; i < hi; ++i) d[i] = static_cast<D>(s[i]);
    }
  });
}

template <typename S>
void convert_from(const void* src, void* dst, Elem de, int64_t n) {
  switch (de) {
    case Elem::F64: return convert_as<S, double>(src, dst, n);
    case Elem::F32: return convert_as<S, float>(src, dst, n);
    case Elem::F16: return convert_as<S, at::Half>(src, dst, n);
    case Elem::I64: return convert_as<S, int64_t>(src, dst, n);
    case Elem::I32: return convert_as<S, int32_t>(src, dst, n);
    case Elem::U8: return convert_as<S, uint8_t>(src, dst, n);
    case Elem::I8: return convert_as<S, int8_t>(src, dst, n);
  }
}

void convert(const void* src, Elem se, void* dst, Elem de, int64_t n) {
  switch (se) {
    case Elem::F64: return convert_from<double>(src, dst, de, n);
    case Elem::F32: return convert_from<float>(src, dst, de, n);
    case Elem::F16: return convert_from<at::Half>(src, dst, de, n);
    case Elem::I64: return convert_from<int64_t>(src, dst, de, n);
    case Elem::I32: return convert_from<int32_t>(src, dst, de, n);
    case Elem::U8: return convert_from<uint8_t>(src, dst, de, n);
    case Elem::I8: return convert_from<int8_t>(src, dst, de, n);
  }
}

at::Tensor pinned(int64_t count, at::ScalarType type) {
  return at::empty({count}, at::TensorOptions().dtype(type).pinned_memory(true));
}

// elements per piece of an array whose wider side has `width` bytes per element
int64_t piece_elems(int64_t count, size_t width) {
  const int64_t whole = count * (int64_t)width;
  return whole <= SMALL ? count : PIECE / (int64_t)width;
}

size_t wider(Elem a, Elem b) { return elem_size(a) > elem_size(b) ? elem_size(a) : elem_size(b); }

}  // namespace

void to_device(const HostArray& src, const at::Tensor& dst) {
  if (src.count == 0) return;
  const Elem de = elem_of(dst.scalar_type());
  const int64_t step = piece_elems(src.count, wider(src.elem, de));
  const at::Tensor flat = dst.view({-1});
  at::Tensor stage[2];
  std::optional<c10::Event> sent[2];
  const c10::Stream stream = c10::cuda::getCurrentCUDAStream(dst.get_device()).unwrap();
  int64_t at = 0;
  for (int i = 0; at < src.count; ++i, at += step) {
    const int b = i & 1;
    const int64_t n = std::min(step, src.count - at);
    if (!stage[b].defined()) {
      stage[b] = pinned(std::min(step, src.count), dst.scalar_type());
      sent[b].emplace(c10::DeviceType::CUDA);
    } else {
      sent[b]->synchronize();   // the piece before last has left this buffer
    }
    convert(static_cast<const uint8_t*>(src.data) + at * (int64_t)elem_size(src.elem), src.elem, stage[b].data_ptr(), de, n);
    // (the copy tells the pinned allocator that the buffer is in use until it has completed)
    flat.narrow(0, at, n).copy_(n == stage[b].numel() ? stage[b] : stage[b].narrow(0, 0, n), /*non_blocking=*/true);
    if (at + step < src.count) sent[b]->record(stream);
  }
}

void to_host(const std::vector<std::pair<at::Tensor, HostArray>>& jobs) {
  std::vector<std::pair<at::Tensor, size_t>> small;   // staged, job
  c10::Device dev(c10::DeviceType::CUDA, 0);
  bool any = false;
  for (const auto& [t, h] : jobs)
    if (h.count) dev = t.device(), any = true;
  if (!any) return;
  const c10::Stream stream = c10::cuda::getCurrentCUDAStream(dev.index()).unwrap();
  for (size_t j = 0; j < jobs.size(); ++j) {
    const auto& [t, h] = jobs[j];
    if (h.count == 0 || h.count * (int64_t)wider(elem_of(t.scalar_type()), h.elem) > SMALL) continue;
    small.emplace_back(pinned(h.count, t.scalar_type()), j);
    small.back().first.copy_(t.view({-1}), true);
  }
  c10::Event small_done(c10::DeviceType::CUDA);
  if (!small.empty()) small_done.record(stream);
  for (size_t j = 0; j < jobs.size(); ++j) {
    const auto& [t, h] = jobs[j];
    const Elem se = elem_of(t.scalar_type());
    if (h.count == 0 || h.count * (int64_t)wider(se, h.elem) <= SMALL) continue;
    const int64_t step = piece_elems(h.count, wider(se, h.elem));
    const at::Tensor flat = t.view({-1});
    at::Tensor stage[2] = {pinned(step, t.scalar_type()), pinned(step, t.scalar_type())};
    c10::Event arrived[2] = {c10::Event(c10::DeviceType::CUDA), c10::Event(c10::DeviceType::CUDA)};
    const int64_t pieces = (h.count + step - 1) / step;
    auto fetch = [&](int64_t p) {
      const int64_t n = std::min(step, h.count - p * step);
      stage[p & 1].narrow(0, 0, n).copy_(flat.narrow(0, p * step, n), true);
      arrived[p & 1].record(stream);
    };
    fetch(0);
    for (int64_t p = 0; p < pieces; ++p) {
      if (p + 1 < pieces) fetch(p + 1);   // (its buffer was emptied by the conversion of piece p - 1)
      arrived[p & 1].synchronize();
      convert(stage[p & 1].data_ptr(), se, static_cast<uint8_t*>(h.data) + p * step * (int64_t)elem_size(h.elem), h.elem,
              std::min(step, h.count - p * step));
    }
  }
  if (!small.empty()) {
    small_done.synchronize();
    for (const auto& [stage, j] : small)
      convert(stage.data_ptr(), elem_of(stage.scalar_type()), jobs[j].second.data, jobs[j].second.elem, jobs[j].second.count);
  }
}

}  // namespace tqhost
