// A copy between pageable memory and the GPU goes through the driver's own staging buffer on one thread (3-10 GB/s), and a
// change of type around it -- 64-bit indices on the host are bytes on the device -- was a second and third pass on one
// thread, most of it page faults of the new array.  Here the conversion is the pass between the caller's array and a pinned
// staging buffer, in pieces that a few threads take from a counter, so that one thread's piece is on the bus while others
// convert theirs: the index array of 65,536 x 128 vectors travels as 8 MB instead of 67.  A piece is one
// 2 MB page of a large array (NumPy asks for those), so that the threads clear different pages: with all of them inside one
// piece the faults of a fresh 67 MB array took 4 ms.  The threads live for one call and block when they wait; the caller
// works too, and on a busy machine (BLAS threads spin for some 30 ms after a product) does not wait for a helper that has
// not got to run yet.  The buffers come from torch's pinned allocator in one block of at most 32 MB, which keeps and
// reuses it.  Pieces move by plain CUDA copies: a helper thread does not have the caller's torch state (inference mode,
// dispatch modes), and a torch operation on a tensor made under it may be refused there.
#include "tq_host_copy.h"

#include <ATen/core/CachingHostAllocator.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <sched.h>
#include <string.h>

#include <algorithm>
#include <condition_variable>
#include <exception>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

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

constexpr int64_t PAGE = 2 << 20;       // most bytes of the wider side per piece
constexpr int64_t LEAST = 256 << 10;    // fewest: arrays up to this size travel in one piece, several behind one wait
constexpr int MOST_THREADS = 8;

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
  if constexpr (std::is_same_v<S, D>) {
    memcpy(d, s, (size_t)n * sizeof(S));
  } else {
    for (int64_t i = 0; i < n; ++i) d[i] = static_cast<D>(s[i]);
  }
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

size_t wider(Elem a, Elem b) { return elem_size(a) > elem_size(b) ? elem_size(a) : elem_size(b); }

// Elements [begin(p), begin(p + 1)) of an array are piece p; pieces of PAGE bytes end on multiples of PAGE in the host's
// address space.
struct Pieces {
  int64_t count, step, first, n;
  Pieces(const HostArray& h, Elem dev) : count(h.count) {
    const int64_t w = (int64_t)wider(h.elem, dev), bytes = count * w;
    const int64_t piece = std::min(PAGE, std::max(LEAST, bytes / (2 * MOST_THREADS)));
    step = piece / w;
    first = step;
    if (piece == PAGE && (int64_t)elem_size(h.elem) == w) {
      const int64_t to_page = (int64_t)(PAGE - (reinterpret_cast<uintptr_t>(h.data) & (PAGE - 1))) / w;
      if (to_page > 0) first = to_page;
    }
    first = std::min(first, count);
    n = 1 + (count - first + step - 1) / step;
  }
  int64_t begin(int64_t p) const { return p == 0 ? 0 : std::min(count, first + (p - 1) * step); }
  int64_t length(int64_t p) const { return begin(p + 1) - begin(p); }
  int64_t longest() const { return std::min(count, std::max(first, step)); }
};

// What the threads of one call share.  A helper that starts after the caller has closed it touches nothing else.
struct Crew {
  std::mutex lock;
  std::condition_variable idle;
  int64_t at = 0, pieces = 0;
  int active = 0, buffers = 0;
  bool closed = false;
  std::exception_ptr failed;

  int64_t next() {
    const std::lock_guard<std::mutex> hold(lock);
    return at < pieces && !failed ? at++ : -1;
  }
};

// work(buffer, p) for every piece p, on the caller and up to threads - 1 helpers; `buffer` is a thread's own number
template <typename F>
void on_threads(int64_t pieces, int threads, const c10::cuda::CUDAStream& stream, const F& work) {
  auto crew = std::make_shared<Crew>();
  crew->pieces = pieces;
  auto take_part = [&work, stream](Crew& c) {
    int mine;
    {
      const std::lock_guard<std::mutex> hold(c.lock);
      if (c.closed || c.at >= c.pieces) return;
      mine = c.buffers++;
      ++c.active;
    }
    try {
      const c10::cuda::CUDAStreamGuard guard(stream);
      for (int64_t p; (p = c.next()) >= 0;) work(mine, p);
    } catch (...) {
      const std::lock_guard<std::mutex> hold(c.lock);
      if (!c.failed) c.failed = std::current_exception();
    }
    const std::lock_guard<std::mutex> hold(c.lock);
    if (--c.active == 0) c.idle.notify_all();
  };
  for (int w = 1; w < threads; ++w) {
    try {
      std::thread([crew, take_part] { take_part(*crew); }).detach();
    } catch (const std::system_error&) {
      break;   // no more threads to be had: fewer do the work
    }
  }
  take_part(*crew);
  std::unique_lock<std::mutex> hold(crew->lock);
  crew->closed = true;
  crew->idle.wait(hold, [&] { return crew->active == 0; });
  if (crew->failed) std::rethrow_exception(crew->failed);
}

// cores that this process may run on (hardware_concurrency counts those of the machine)
int64_t usable_cores() {
  cpu_set_t set;
  CPU_ZERO(&set);
  if (sched_getaffinity(0, sizeof(set), &set) == 0) return CPU_COUNT(&set);
  return std::thread::hardware_concurrency();
}

int thread_count(const Pieces& p, size_t width) {
  const int64_t cores = usable_cores(), mega = p.count * (int64_t)width >> 20;
  return (int)std::max<int64_t>(1, std::min({(int64_t)MOST_THREADS, p.n, cores / 2, 1 + mega}));
}

void move(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, const c10::cuda::CUDAStream& stream) {
  C10_CUDA_CHECK(cudaMemcpyAsync(dst, src, bytes, kind, stream.stream()));
}

// tells the pinned allocator that a block is in use until what the stream holds so far has completed
void in_use(const at::Tensor& t, const c10::cuda::CUDAStream& stream) {
  at::getHostAllocator(at::kCUDA)->record_event(t.data_ptr(), t.storage().data_ptr().get_context(), stream.unwrap());
}

// two buffers per thread: [thread][2] of `room` elements
struct Staging {
  int64_t room;
  size_t size;                     // bytes of an element
  c10::cuda::CUDAStream stream;
  at::Tensor all;
  std::vector<c10::Event> moved;
  std::vector<int> uses;
  Staging(const Pieces& p, int threads, at::ScalarType type, const c10::cuda::CUDAStream& st)
      : room(p.longest()), size(at::elementSize(type)), stream(st), all(pinned(2 * threads * room, type)), uses(threads, 0) {
    for (int i = 0; i < 2 * threads; ++i) moved.emplace_back(c10::DeviceType::CUDA);
  }
  ~Staging() {
    try {
      in_use(all, stream);
    } catch (...) {   // an earlier error of the device, reported where it was met
    }
  }
  // the next of a thread's two buffers, free: what was copied from it before has left it
  int take(int thread) {
    const int b = 2 * thread + (uses[thread] & 1);
    if (uses[thread]++ >= 2) moved[b].synchronize();
    return b;
  }
  uint8_t* buffer(int b) const { return static_cast<uint8_t*>(all.data_ptr()) + (size_t)(b * room) * size; }
};

}  // namespace

void to_device(const HostArray& src, const at::Tensor& dst) {
  if (src.count == 0) return;
  const Elem de = elem_of(dst.scalar_type());
  const Pieces pieces(src, de);
  auto* const to = static_cast<uint8_t*>(dst.data_ptr());
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dst.get_device());
  const int threads = thread_count(pieces, wider(src.elem, de));
  Staging stage(pieces, threads, dst.scalar_type(), stream);
  on_threads(pieces.n, threads, stream, [&](int thread, int64_t p) {
    const int64_t at = pieces.begin(p), n = pieces.length(p);
    const int b = stage.take(thread);
    uint8_t* const buf = stage.buffer(b);
    convert(static_cast<const uint8_t*>(src.data) + at * (int64_t)elem_size(src.elem), src.elem, buf, de, n);
    move(to + (size_t)at * stage.size, buf, (size_t)n * stage.size, cudaMemcpyHostToDevice, stream);
    stage.moved[b].record(stream.unwrap());
  });
}

void to_host(const std::vector<std::pair<at::Tensor, HostArray>>& jobs) {
  std::vector<std::pair<at::Tensor, size_t>> small;   // staged, job
  c10::DeviceIndex dev = -1;
  for (const auto& [t, h] : jobs)
    if (h.count) dev = (c10::DeviceIndex)t.get_device();
  if (dev < 0) return;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dev);
  auto is_small = [](const at::Tensor& t, const HostArray& h) {
    return h.count * (int64_t)wider(elem_of(t.scalar_type()), h.elem) <= LEAST;
  };
  for (size_t j = 0; j < jobs.size(); ++j) {
    const auto& [t, h] = jobs[j];
    if (h.count == 0 || !is_small(t, h)) continue;
    small.emplace_back(pinned(h.count, t.scalar_type()), j);
    move(small.back().first.data_ptr(), t.const_data_ptr(), t.nbytes(), cudaMemcpyDeviceToHost, stream);
    in_use(small.back().first, stream);
  }
  c10::Event small_done(c10::DeviceType::CUDA);
  if (!small.empty()) small_done.record(stream.unwrap());
  for (const auto& [t, h] : jobs) {
    if (h.count == 0 || is_small(t, h)) continue;
    const Elem se = elem_of(t.scalar_type());
    const Pieces pieces(h, se);
    const auto* const from = static_cast<const uint8_t*>(t.const_data_ptr());
    const int threads = thread_count(pieces, wider(se, h.elem));
    Staging stage(pieces, threads, t.scalar_type(), stream);
    const HostArray to = h;
    on_threads(pieces.n, threads, stream, [&](int thread, int64_t p) {
      const int64_t at = pieces.begin(p), n = pieces.length(p);
      const int b = stage.take(thread);
      uint8_t* const buf = stage.buffer(b);
      move(buf, from + (size_t)at * stage.size, (size_t)n * stage.size, cudaMemcpyDeviceToHost, stream);
      stage.moved[b].record(stream.unwrap());
      stage.moved[b].synchronize();
      convert(buf, se, static_cast<uint8_t*>(to.data) + at * (int64_t)elem_size(to.elem), to.elem, n);
    });
  }
  if (!small.empty()) {
    small_done.synchronize();
    for (const auto& [stage, j] : small)
      convert(stage.data_ptr(), elem_of(stage.scalar_type()), jobs[j].second.data, jobs[j].second.elem, jobs[j].second.count);
  }
}

}  // namespace tqhost
