// Copies of a caller's pageable host arrays to the device through pinned staging.
//
// cudaMemcpyAsync from pageable memory stages it on one host thread: 31 MB of
// queries (10,000 x 784) took 1.6 to 2.9 ms, two to four times the search behind
// it.  Here up to four threads (the caller among them) copy 1 MB chunks into
// pinned slots, two slots a thread, and enqueue each chunk's DMA as soon as it is
// staged, so staging and DMA overlap: 31 MB in about 1 ms.  The copies of one call
// are enqueued on the caller's stream; when it returns the pageable source may be
// reused.
//
// The slots (8 MB a device) live as long as some index does.  One upload uses
// them at a time; a concurrent one, a small one, or one whose source is already
// page-locked takes the plain copy.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.cuh"

namespace b2k {
namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr int kMaxThreads = 4;
constexpr int kSlots = 2 * kMaxThreads;
// Below this the threads save nothing: 6.4 MB of radius queries took the same
// call time staged (4.9 ms) and plain (4.6), 31 MB 5.8 against 7.4.
constexpr size_t kMinBytes = (size_t)16 << 20;
constexpr int kMaxDevices = 64;

struct Staging {
  std::mutex mu;
  int users = 0;  // live indexes of the device
  unsigned char* buf = nullptr;
  cudaEvent_t free_at[kSlots] = {};  // the slot's last DMA
};

Staging& staging(int device) {
  static Staging all[kMaxDevices];
  return all[device];
}

// The slots of `s` (allocated on first use); false when they cannot be had.
bool ensure_slots(Staging& s) {
  if (s.buf) return true;
  void* p = nullptr;
  if (cudaHostAlloc(&p, kSlots * kChunk, cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  for (int i = 0; i < kSlots; ++i)
    if (cudaEventCreateWithFlags(&s.free_at[i], cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      while (i-- > 0) cudaEventDestroy(s.free_at[i]);
      cudaFreeHost(p);
      return false;
    }
  s.buf = static_cast<unsigned char*>(p);
  return true;
}

}  // namespace

void staging_acquire(int device) {
  if (device < 0 || device >= kMaxDevices) return;
  Staging& s = staging(device);
  std::lock_guard<std::mutex> lock(s.mu);
  ++s.users;
}

void staging_release(int device) {
  if (device < 0 || device >= kMaxDevices) return;
  Staging& s = staging(device);
  std::lock_guard<std::mutex> lock(s.mu);
  if (--s.users > 0 || !s.buf) return;
  for (auto& e : s.free_at) {
    cudaEventSynchronize(e);
    cudaEventDestroy(e);
  }
  cudaFreeHost(s.buf);
  s.buf = nullptr;
}

cudaError_t upload_host(void* dst, const void* src, size_t bytes, cudaStream_t st,
                        bool* pageable) {
  auto plain = [&] { return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st); };
  // (a small internal copy is followed by a wait of its caller: no need to ask)
  if (pageable) *pageable = false;
  if (bytes < kMinBytes && !pageable) return plain();
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, src) != cudaSuccess) {
    cudaGetLastError();
    return plain();
  }
  const bool registered = attr.type != cudaMemoryTypeUnregistered;
  if (pageable) *pageable = !registered;
  // (the per-thread default stream is another stream in each helper thread)
  if (bytes < kMinBytes || registered || st == cudaStreamPerThread) return plain();
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices)
    return plain();
  Staging& s = staging(device);
  std::unique_lock<std::mutex> lock(s.mu, std::try_to_lock);
  if (!lock.owns_lock() || s.users == 0 || !ensure_slots(s)) return plain();

  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  std::atomic<size_t> next{0};
  std::atomic<int> error{(int)cudaSuccess};
  auto work = [&](int w) {
    cudaError_t e = cudaSetDevice(device);
    for (int round = 0; e == cudaSuccess && error.load() == (int)cudaSuccess; ++round) {
      const size_t c = next.fetch_add(1);
      if (c >= chunks) break;
      const int slot = 2 * w + (round & 1);
      unsigned char* stage = s.buf + slot * kChunk;
      const size_t off = c * kChunk, len = std::min(kChunk, bytes - off);
      e = cudaEventSynchronize(s.free_at[slot]);  // the slot's DMA, an earlier call's included
      if (e != cudaSuccess) break;
      memcpy(stage, static_cast<const unsigned char*>(src) + off, len);
      e = cudaMemcpyAsync(static_cast<unsigned char*>(dst) + off, stage, len,
                          cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaEventRecord(s.free_at[slot], st);
    }
    if (e != cudaSuccess) error.store((int)e);
  };
  std::vector<std::thread> helpers;
  const int threads = (int)std::min<size_t>({(size_t)kMaxThreads, chunks,
                                             std::max(1u, std::thread::hardware_concurrency())});
  try {
    helpers.reserve((size_t)threads);
    for (int w = 1; w < threads; ++w) helpers.emplace_back(work, w);
  } catch (...) {
    // fewer helpers: the others take their chunks
  }
  work(0);
  for (auto& t : helpers) t.join();
  return (cudaError_t)error.load();
}

}  // namespace b2k

using namespace b2k;

extern "C" B2K_API int b2k_upload(void* d_dst, const void* src, int64_t bytes, void* stream) {
  if (bytes < 0) return report_error(B2K_EINVAL, "negative byte count");
  if (bytes == 0) return B2K_OK;
  if (!d_dst || !src) return report_error(B2K_EINVAL, "pointers must not be NULL");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  bool pageable = false;
  cudaError_t e = upload_host(d_dst, src, (size_t)bytes, st, &pageable);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (e == cudaSuccess && !pageable) e = cudaStreamIsCapturing(st, &capture);
  if (e == cudaSuccess && !pageable && capture == cudaStreamCaptureStatusNone)
    e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return report_error(B2K_ECUDA, cudaGetErrorString(e));
  return B2K_OK;
}
