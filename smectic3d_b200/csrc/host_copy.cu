// Staged host copies (host_copy.cuh).
#include "host_copy.cuh"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

namespace shb {
namespace {

constexpr int kWorkers = 6;               // memcpy threads; 6 x 8 GB/s is about the link rate
constexpr size_t kChunk = size_t(1) << 19;  // per buffer, two buffers per worker: 6 MB pinned in all
// Below kMin the threads cost more than they save: 17 MB to the device take 820 us plain
// and 640 staged, but three fields of 8 MB only 0.1 ms less, and an array that the caller
// frees after other threads have touched it is slower to unmap (Solver.restore of a
// Neumann 128^3 FP32 handle 3.4 ms plain, 4.2 staged).
// To the host 17 MB take 850 us plain and 650 to 1100 staged when the array's pages
// exist, but 3 ms more plain when they do not (the page faults, which the threads share):
// staged from kMinToHost on (134 MB 7.8 -> 5.5 ms), below that only into untouched pages
// (adjoint of 128^3, T = 400: 24.6 -> 22.1 ms).
constexpr size_t kMin = size_t(12) << 20, kMinToHost = size_t(32) << 20;
// Making and freeing the buffers takes 6.6 ms here (2.5 even for 64 KB) and a staged
// copy saves some 85 us per MB: they are made once the plain copies since the last
// time would have paid for them, and freed with the last handle unless a copy went
// through them within the last second (then the next handle likely needs them again).
// Made and freed with every handle, as before, they cost a program of one 128^3 FP32
// gradient per handle more than the staged copies gain (12.3 -> 15.6 ms).
constexpr size_t kEarned = size_t(64) << 20;
constexpr std::chrono::seconds kIdle(1);

// One set of pinned buffers for the process: a copy that finds it taken (another
// handle's copy on another thread) goes the plain way.
struct Pool {
  std::mutex use;    // held for the whole of a staged copy
  std::mutex state;  // guards the members below
  int handles = 0;
  size_t plain = 0;  // bytes of large copies that found no buffers
  std::chrono::steady_clock::time_point last;  // end of the last staged copy
  char* pinned = nullptr;
};
Pool& pool() {
  static Pool p;
  return p;
}

bool pageable(const void* host) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

// whether most of the array's pages were never touched, by a sample of eight
bool untouched(const char* host, size_t bytes) {
  const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE));
  int n = 0;
  for (int i = 0; i < 8; ++i) {
    const uintptr_t at = (reinterpret_cast<uintptr_t>(host) + (2 * i + 1) * (bytes / 16)) & ~(page - 1);
    unsigned char in_memory = 1;
    if (mincore(reinterpret_cast<void*>(at), page, &in_memory) == 0 && !(in_memory & 1)) ++n;
  }
  return n >= 4;
}

// worker w of n: chunks w, w + n, ... through its two buffers
cudaError_t work(int w, int n, int device, char* pinned, char* host, char* dev, size_t bytes, bool to_device,
                 cudaStream_t stream) {
  cudaError_t e = cudaSetDevice(device);
  cudaEvent_t done[2] = {nullptr, nullptr};
  for (auto& ev : done)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  char* buf[2] = {pinned + size_t(2 * w) * kChunk, pinned + size_t(2 * w + 1) * kChunk};
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  size_t off[2] = {0, 0}, len[2] = {0, 0};  // chunk in flight in each buffer (len 0: none)
  auto finish = [&](int b) {
    if (e == cudaSuccess && len[b]) {
      e = cudaEventSynchronize(done[b]);
      if (e == cudaSuccess && !to_device) std::memcpy(host + off[b], buf[b], len[b]);
    }
    len[b] = 0;
  };
  int b = 0;
  for (size_t c = w; c < chunks && e == cudaSuccess; c += n, b ^= 1) {
    finish(b);
    if (e != cudaSuccess) break;
    off[b] = c * kChunk;
    len[b] = std::min(kChunk, bytes - off[b]);
    if (to_device) {
      std::memcpy(buf[b], host + off[b], len[b]);
      e = cudaMemcpyAsync(dev + off[b], buf[b], len[b], cudaMemcpyHostToDevice, stream);
    } else {
      e = cudaMemcpyAsync(buf[b], dev + off[b], len[b], cudaMemcpyDeviceToHost, stream);
    }
    if (e == cudaSuccess) e = cudaEventRecord(done[b], stream);
  }
  // the buffers are free for the next copy once these have passed
  finish(b);
  finish(b ^ 1);
  if (e != cudaSuccess) cudaStreamSynchronize(stream);  // nothing still reads or writes the buffers
  for (auto& ev : done)
    if (ev) cudaEventDestroy(ev);
  return e;
}

cudaError_t plain(void* dst, const void* src, size_t bytes, bool to_device, cudaStream_t stream) {
  const cudaError_t e =
      cudaMemcpyAsync(dst, src, bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, stream);
  return e != cudaSuccess || to_device ? e : cudaStreamSynchronize(stream);
}

cudaError_t staged(void* dst, const void* src, size_t bytes, bool to_device, cudaStream_t stream) {
  if (!dst || !src) return cudaErrorInvalidValue;  // chunks of a null array would have other addresses
  char* host = static_cast<char*>(to_device ? const_cast<void*>(src) : dst);
  char* dev = static_cast<char*>(to_device ? dst : const_cast<void*>(src));
  if (bytes < kMin || !pageable(host) || (!to_device && bytes < kMinToHost && !untouched(host, bytes))) return plain(dst, src, bytes, to_device, stream);
  Pool& p = pool();
  std::unique_lock<std::mutex> lock(p.use, std::try_to_lock);
  if (!lock.owns_lock()) return plain(dst, src, bytes, to_device, stream);
  char* pinned;
  {
    std::lock_guard<std::mutex> g(p.state);
    if (!p.pinned && p.handles > 0 && p.plain >= kEarned) {
      p.plain = 0;
      if (cudaHostAlloc(reinterpret_cast<void**>(&p.pinned), 2 * kWorkers * kChunk, cudaHostAllocPortable) !=
          cudaSuccess) {
        cudaGetLastError();
        p.pinned = nullptr;
      }
    }
    pinned = p.pinned;
    if (!pinned) p.plain += bytes;
  }
  if (!pinned) return plain(dst, src, bytes, to_device, stream);
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  std::thread th[kWorkers];
  cudaError_t r[kWorkers];
  bool run[kWorkers];
  for (int w = 1; w < kWorkers; ++w) {
    r[w] = cudaSuccess;
    run[w] = true;
    try {
      th[w] = std::thread([&, w] { r[w] = work(w, kWorkers, device, pinned, host, dev, bytes, to_device, stream); });
    } catch (...) {  // no thread to be had: its chunks follow on this one
      run[w] = false;
    }
  }
  e = work(0, kWorkers, device, pinned, host, dev, bytes, to_device, stream);
  for (int w = 1; w < kWorkers; ++w) {
    if (run[w]) th[w].join();
    else r[w] = work(w, kWorkers, device, pinned, host, dev, bytes, to_device, stream);
    if (e == cudaSuccess) e = r[w];
  }
  std::lock_guard<std::mutex> g(p.state);
  p.last = std::chrono::steady_clock::now();
  return e;
}

}  // namespace

cudaError_t copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  return staged(dst, src, bytes, true, stream);
}
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  return staged(dst, src, bytes, false, stream);
}

void host_copy_retain() {
  Pool& p = pool();
  std::lock_guard<std::mutex> g(p.state);
  ++p.handles;
}
void host_copy_release() {
  Pool& p = pool();
  // a copy in flight belongs to a handle that still exists, so the buffers are idle
  // when the count reaches 0
  std::lock_guard<std::mutex> g(p.state);
  if (--p.handles == 0 && p.pinned && std::chrono::steady_clock::now() - p.last > kIdle) {
    cudaFreeHost(p.pinned);
    p.pinned = nullptr;
  }
}

}  // namespace shb
