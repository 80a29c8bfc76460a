// tsp_readback.h against a stand-in for the CUDA runtime on host memory: the
// copies happen at once, 2-D copies refuse pitches above the documented maximum
// of 2^31 - 1 bytes. Rows lie in sparsely backed address space, so pitches of
// several GiB cost no memory.
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <new>

#include "tsp_readback.h"

// Host allocations fail while the countdown is at zero (below: they never do).
static int g_allocs_left = -1;
void* operator new(size_t n) {
  if (g_allocs_left == 0) throw std::bad_alloc();
  if (g_allocs_left > 0) --g_allocs_left;
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

namespace {
int copies_1d = 0, copies_2d = 0, host_allocs = 0;
}

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  ++host_allocs;
  *p = std::malloc(n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  ++copies_1d;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  if (dp > 0x7fffffffu || sp > 0x7fffffffu) return cudaErrorInvalidPitchValue;
  ++copies_2d;
  for (size_t r = 0; r < h; ++r)
    std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
}

#define CHECK(c)                                                  \
  do {                                                            \
    if (!(c)) {                                                   \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #c);        \
      std::exit(1);                                               \
    }                                                             \
  } while (0)

namespace {

unsigned char* space(size_t n) {
  void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  CHECK(p != MAP_FAILED);
  return static_cast<unsigned char*>(p);
}

void rows(size_t dpitch, size_t spitch, size_t width, size_t height) {
  const size_t nd = dpitch * (height - 1) + width + 1, ns = spitch * (height - 1) + width;
  unsigned char *dst = space(nd), *src = space(ns);
  for (size_t r = 0; r < height; ++r)
    for (size_t i = 0; i < width; ++i) src[r * spitch + i] = (unsigned char)(i * 7 + i / 251 + r * 31 + 1);
  CHECK(tsp::read_back(dst, dpitch, src, spitch, width, height, nullptr) == cudaSuccess);
  for (size_t r = 0; r < height; ++r) {
    CHECK(std::memcmp(dst + r * dpitch, src + r * spitch, width) == 0);
    CHECK(dpitch == width || dst[r * dpitch + width] == 0);  // nothing between the rows
  }
  munmap(dst, nd);
  munmap(src, ns);
}

}  // namespace

int main() {
  const size_t KiB = 1024, MiB = 1024 * KiB, GiB = 1024 * MiB;
  rows(64, 64, 64, 5);                                // one run
  rows(96, 128, 64, 5);                               // plain 2-D copy
  CHECK(copies_2d == 1);
  rows(4 * MiB, 5 * MiB, 3 * MiB, 7);                 // staged, two rows per piece
  rows(9 * MiB, 10 * MiB, 9 * MiB - 5, 3);            // rows above one piece
  rows(20 * MiB, 20 * MiB, 20 * MiB, 1);
  rows(4 * KiB, 2 * GiB - 1, 4 * KiB, 3);             // the largest pitch of a 2-D copy
  const int n2 = copies_2d, n1 = copies_1d;
  rows(4 * KiB, 2 * GiB, 4 * KiB, 3);                 // above it: plain path
  rows(2 * GiB + 8, 4 * KiB, 4 * KiB, 3);
  rows(MiB, 2 * GiB + 160, MiB - 16, 4);              // above it: staged, eight rows per piece
  rows(3 * GiB, 2 * GiB + 160, MiB + 16, 3);
  CHECK(copies_2d == n2 && copies_1d == n1 + 3 + 3 + 4 + 3);
  // The n-th host allocation of a copy and all later ones fail: the copy is
  // whole, and the pinned buffers are free again for the next one.
  for (int n = 0; n < 24; ++n) {
    g_allocs_left = n;
    rows(4 * MiB, 5 * MiB, 3 * MiB, 9);
    g_allocs_left = -1;
    unsigned char* pin = tsp::Staging::get().take();
    CHECK(pin != nullptr);
    tsp::Staging::get().give_back();
  }
  // The buffers are allocated by the copy that reaches the bytes they are worth.
  tsp::Staging::get().release();
  const int n0 = host_allocs;
  for (int n = 0; n < 2; ++n) rows(20 * MiB, 20 * MiB, 20 * MiB, 1);
  CHECK(host_allocs == n0);
  for (int n = 0; n < 3; ++n) rows(4 * MiB, 5 * MiB, 4 * MiB, 1);
  CHECK(host_allocs == n0 + 1);
  std::puts("read-back checks passed");
  return 0;
}
