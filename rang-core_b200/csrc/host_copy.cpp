#include "host_copy.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace wg {

void check_cuda(cudaError_t e, const char* what);

TestLimits& test_limits() {
  static thread_local TestLimits l;
  return l;
}

namespace {

constexpr size_t PIECE = (size_t)1 << 20;        // bytes of a pinned buffer
constexpr size_t STAGED_MIN = (size_t)4 << 20;   // smaller arrays: one plain copy
constexpr size_t POOL_MAX = 32;                  // buffers kept (32 MB) over all devices
constexpr unsigned MAX_THREADS = 8;              // 8 threads fill 55 GB/s; 16 measured no faster

// A pinned buffer and the event after its last copy on `dev`.
struct Buffer {
  void* p = nullptr;
  cudaEvent_t ev = nullptr;
  int dev = -1;
};

// The buffers no copy is using (a fixed array: the worker threads that give
// them back must not throw).
std::mutex g_mu;
std::array<Buffer, POOL_MAX> g_free;
size_t g_nfree = 0;

cudaError_t acquire(int dev, bool no_pinned, Buffer& b) {
  if (no_pinned) return cudaErrorMemoryAllocation;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    for (size_t i = g_nfree; i-- > 0;)
      if (g_free[i].dev == dev) {
        b = g_free[i];
        g_free[i] = g_free[--g_nfree];
        return cudaSuccess;
      }
  }
  b = Buffer{};
  b.dev = dev;
  cudaError_t e = cudaHostAlloc(&b.p, PIECE, cudaHostAllocDefault);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.ev, cudaEventDisableTiming);
  return e;
}

void destroy(Buffer& b) {
  if (b.ev) {
    cudaEventSynchronize(b.ev);
    cudaEventDestroy(b.ev);
  }
  if (b.p) cudaFreeHost(b.p);
  b = Buffer{};
}

void give_back(Buffer& b) {
  if (!b.p || !b.ev) {
    destroy(b);
    return;
  }
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_nfree < POOL_MAX) {
      g_free[g_nfree++] = b;
      return;
    }
  }
  destroy(b);
}

bool pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// One worker: takes pieces by the shared counter, two buffers in turn. A piece
// for which no buffer can be had goes as the driver copies pageable arrays.
void work(bool to_device, unsigned char* dst, const unsigned char* src, size_t bytes, int dev, cudaStream_t s,
          bool no_pinned, std::atomic<size_t>& next, std::atomic<int>& error) {
  auto fail = [&](cudaError_t e) {
    int none = cudaSuccess;
    if (e != cudaSuccess) error.compare_exchange_strong(none, (int)e);
    return e != cudaSuccess;
  };
  if (fail(cudaSetDevice(dev))) return;
  Buffer buf[2];
  bool plain = false;
  size_t held[2] = {0, 0}, at[2] = {0, 0};  // bytes on their way to the host, and where they go
  for (int k = 0; error.load() == cudaSuccess; k ^= 1) {
    Buffer& b = buf[k];
    if (b.p && fail(cudaEventSynchronize(b.ev))) break;
    if (held[k]) {
      std::memcpy(dst + at[k], b.p, held[k]);
      held[k] = 0;
    }
    const size_t o = next.fetch_add(1) * PIECE;
    if (o >= bytes) {
      if (!held[k ^ 1]) break;
      continue;
    }
    const size_t n = std::min(PIECE, bytes - o);
    if (!b.p && !plain) {
      if (acquire(dev, no_pinned, b) != cudaSuccess) {
        cudaGetLastError();
        destroy(b);
        plain = true;
      } else if (fail(cudaEventSynchronize(b.ev))) {
        break;
      }
    }
    if (!b.p) {
      if (fail(cudaMemcpyAsync(dst + o, src + o, n, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, s)))
        break;
      continue;
    }
    if (to_device) {
      std::memcpy(b.p, src + o, n);
      if (fail(cudaMemcpyAsync(dst + o, b.p, n, cudaMemcpyHostToDevice, s))) break;
    } else {
      if (fail(cudaMemcpyAsync(b.p, src + o, n, cudaMemcpyDeviceToHost, s))) break;
      held[k] = n;
      at[k] = o;
    }
    if (fail(cudaEventRecord(b.ev, s))) {
      cudaStreamSynchronize(s);  // the copy in flight still uses the buffer
      break;
    }
  }
  for (Buffer& b : buf)
    if (b.p || b.ev) give_back(b);
}

void staged(bool to_device, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "no CUDA device");
  const size_t pieces = (bytes + PIECE - 1) / PIECE;
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  const unsigned n = (unsigned)std::min<size_t>(pieces, std::min(hw, MAX_THREADS));
  const bool no_pinned = test_limits().no_pinned;  // the calling thread's
  std::atomic<size_t> next{0};
  std::atomic<int> error{cudaSuccess};
  auto run = [&] {
    work(to_device, static_cast<unsigned char*>(dst), static_cast<const unsigned char*>(src), bytes, dev, s, no_pinned,
         next, error);
  };
  std::vector<std::thread> threads;
  threads.reserve(n);
  try {
    for (unsigned i = 1; i < n; i++) threads.emplace_back(run);
  } catch (const std::system_error&) {
    // fewer threads: this one takes the pieces that are left
  }
  run();
  for (std::thread& t : threads) t.join();
  check_cuda((cudaError_t)error.load(), to_device ? "copy to device" : "copy to host");
}

}  // namespace

void copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes >= STAGED_MIN && pageable(src))
    staged(true, dst, src, bytes, s);
  else if (bytes)
    check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s), "copy to device");
}

void copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes >= STAGED_MIN && pageable(dst))
    staged(false, dst, src, bytes, s);
  else if (bytes)
    check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "copy to host");
}

void release_host_buffers() {
  std::array<Buffer, POOL_MAX> out;
  size_t n;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    out = g_free;
    n = g_nfree;
    g_nfree = 0;
  }
  for (size_t i = 0; i < n; i++) destroy(out[i]);
}

}  // namespace wg
