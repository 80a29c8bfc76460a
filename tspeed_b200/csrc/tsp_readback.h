// Large device-to-host copies into pageable memory (internal header of
// tspeed_b200).
//
// A plain copy into pageable memory goes through the driver's staging on one
// thread, which also takes the page faults of a fresh destination: 4.3 GB/s
// measured for the 215 MB wavefield of 64 shots on 10,000 triangles. Here the
// device writes pieces into three pinned buffers in turn and a few threads
// move each piece to its destination while the next is on its way.
//
// The pinned buffers are one set per process (24 MiB, returned by
// tsp_release_cached_memory). Pinning them takes 11 to 15 ms, about what 50 to
// 80 MB of staged copies save, so they are allocated by the copy with which the
// process has asked for 48 MiB: the first wavefield of 7.2 MB that a process
// read took 14 to 39 ms with the buffers, 2.0 to 3.8 ms by the plain path. A copy that finds them
// taken by another thread, or cannot start a thread or get host memory for its
// bookkeeping, takes the plain path.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace tsp {

class Staging {
 public:
  static constexpr size_t kPiece = size_t(8) << 20;
  static constexpr int kBufs = 3;
  static constexpr size_t kWorth = size_t(48) << 20;  // bytes asked for before the buffers are allocated

  static Staging& get() {
    static Staging* s = new Staging();  // outlives the CUDA context: never destroyed
    return *s;
  }
  // The buffers for a copy of `bytes` by this thread, or null while another one
  // uses them or they are not worth allocating yet.
  unsigned char* take(size_t bytes = kWorth) {
    std::lock_guard<std::mutex> lk(m_);
    if (busy_) return nullptr;
    if (!mem_) {
      asked_ += std::min(bytes, kWorth);
      if (asked_ < kWorth) return nullptr;
      void* p = nullptr;
      if (cudaHostAlloc(&p, kPiece * kBufs, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();  // the plain path serves instead
        return nullptr;
      }
      mem_ = static_cast<unsigned char*>(p);
    }
    busy_ = true;
    return mem_;
  }
  void give_back() {
    std::lock_guard<std::mutex> lk(m_);
    busy_ = false;
  }
  void release() {
    std::lock_guard<std::mutex> lk(m_);
    if (busy_ || !mem_) return;
    cudaFreeHost(mem_);
    mem_ = nullptr;
    asked_ = 0;
  }

 private:
  std::mutex m_;
  bool busy_ = false;
  size_t asked_ = 0;
  unsigned char* mem_ = nullptr;
};

// Queues a copy of `rows` rows of `width` bytes (pitches in bytes) from the
// device. 2-D copies are documented for pitches up to the device's maximum,
// 2^31 - 1 bytes; beyond (one shot's seismogram ring may hold more) every row
// is a copy of its own.
inline cudaError_t copy_rows(unsigned char* dst, size_t dpitch, const unsigned char* src, size_t spitch, size_t width,
                             size_t rows, cudaStream_t st) {
  constexpr size_t kMaxPitch = (size_t(1) << 31) - 1;
  if (rows > 1 && dpitch <= kMaxPitch && spitch <= kMaxPitch)
    return cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, cudaMemcpyDeviceToHost, st);
  cudaError_t e = cudaSuccess;
  for (size_t r = 0; r < rows && e == cudaSuccess; ++r)
    e = cudaMemcpyAsync(dst + r * dpitch, src + r * spitch, width, cudaMemcpyDeviceToHost, st);
  return e;
}

// Copies `height` rows of `width` bytes (pitches in bytes) from the device,
// ordered on `st` and complete on return.
inline cudaError_t read_back(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t height,
                             cudaStream_t st) {
  if (width == 0 || height == 0) return cudaSuccess;
  if (dpitch == width && spitch == width) {
    width *= height;
    height = 1;
  }
  unsigned char* d = static_cast<unsigned char*>(dst);
  const unsigned char* s = static_cast<const unsigned char*>(src);
  auto plain = [&]() {
    const cudaError_t e = copy_rows(d, dpitch, s, spitch, width, height, st);
    const cudaError_t done = cudaStreamSynchronize(st);
    return e == cudaSuccess ? done : e;
  };
  const size_t total = width * height;
  if (total < (size_t(2) << 20)) return plain();
  struct Lease {  // the pinned buffers, given back however the copy ends
    unsigned char* mem;
    ~Lease() {
      if (mem) Staging::get().give_back();
    }
  } lease = {Staging::get().take(total)};
  unsigned char* pin = lease.mem;
  if (!pin) return plain();

  struct Piece {
    unsigned char* dst;
    const unsigned char* src;
    size_t width, rows;
  };
  std::vector<Piece> pieces;
  std::vector<int> moved;
  std::vector<std::thread> threads;
  const int want = int(std::min<size_t>(std::max(1u, std::min(8u, std::thread::hardware_concurrency() / 2)),
                                        1 + total / (size_t(4) << 20)));
  try {
    if (width > Staging::kPiece) {
      for (size_t r = 0; r < height; ++r)
        for (size_t o = 0; o < width; o += Staging::kPiece)
          pieces.push_back({d + r * dpitch + o, s + r * spitch + o, std::min(Staging::kPiece, width - o), 1});
    } else {
      const size_t n = Staging::kPiece / width;
      for (size_t r = 0; r < height; r += n)
        pieces.push_back({d + r * dpitch, s + r * spitch, width, std::min(n, height - r)});
    }
    moved.assign(pieces.size(), 0);
    threads.reserve(want);
  } catch (const std::bad_alloc&) {  // no host memory for the bookkeeping
    return plain();
  }

  // ready: pieces whose data is in its buffer; moved[b]: threads done with the
  // piece in buffer b.
  std::mutex m;
  std::condition_variable cv;
  size_t ready = 0;
  int nthreads = 0;
  bool stop = false;
  auto work = [&](int t) {
    for (size_t i = 0; i < pieces.size(); ++i) {
      int n;
      {
        std::unique_lock<std::mutex> lk(m);
        cv.wait(lk, [&] { return ready > i || stop; });
        if (stop) return;
        n = nthreads;
      }
      const Piece& p = pieces[i];
      const unsigned char* from = pin + (i % Staging::kBufs) * Staging::kPiece;
      const size_t bytes = p.width * p.rows;
      size_t lo = (bytes * t / n) & ~size_t(63), hi = t + 1 == n ? bytes : (bytes * (t + 1) / n) & ~size_t(63);
      while (lo < hi) {
        const size_t r = lo / p.width, o = lo - r * p.width, len = std::min(hi - lo, p.width - o);
        std::memcpy(p.dst + r * dpitch + o, from + lo, len);
        lo += len;
      }
      std::lock_guard<std::mutex> lk(m);
      if (++moved[i] == n) cv.notify_all();
    }
  };
  try {
    for (int t = 0; t < want; ++t) threads.emplace_back(work, t);
  } catch (const std::exception&) {  // no thread, or no memory for one: those that started do the work
  }
  if (threads.empty()) return plain();
  {
    std::lock_guard<std::mutex> lk(m);
    nthreads = int(threads.size());
  }
  cudaEvent_t ev[Staging::kBufs] = {};
  cudaError_t e = cudaSuccess;
  for (int b = 0; b < Staging::kBufs && e == cudaSuccess; ++b) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
  auto publish = [&](size_t i) {
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[i % Staging::kBufs]);
    if (e != cudaSuccess) return;
    std::lock_guard<std::mutex> lk(m);
    ready = i + 1;
    cv.notify_all();
  };
  for (size_t i = 0; i < pieces.size() && e == cudaSuccess; ++i) {
    const int b = int(i % Staging::kBufs);
    if (i >= size_t(Staging::kBufs)) {
      std::unique_lock<std::mutex> lk(m);
      cv.wait(lk, [&] { return moved[i - Staging::kBufs] == nthreads; });
    }
    const Piece& p = pieces[i];
    unsigned char* to = pin + size_t(b) * Staging::kPiece;
    e = copy_rows(to, p.width, p.src, spitch, p.width, p.rows, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
    if (i > 0) publish(i - 1);
  }
  if (e == cudaSuccess) publish(pieces.size() - 1);
  if (e != cudaSuccess) {
    cudaStreamSynchronize(st);  // nothing of this copy stays in flight to the buffers
    std::lock_guard<std::mutex> lk(m);
    stop = true;
    cv.notify_all();
  }
  for (std::thread& t : threads) t.join();
  for (cudaEvent_t v : ev)
    if (v) cudaEventDestroy(v);
  return e;
}

}  // namespace tsp
