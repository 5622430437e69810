// Copies between pageable host memory and the device through pinned staging,
// shared by several host threads.
//
// cudaMemcpy of pageable memory moves about 11 GB/s on one B200 host (one thread
// fills the driver's staging buffer), and a fresh destination array adds its page
// faults (2.6 GB/s for a download).  Here each thread takes every n-th chunk
// through two pinned buffers of its own: while one crosses the bus on the thread's
// own stream, the other is filled or emptied by the CPU.
#pragma once

#include <algorithm>
#include <cstring>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace rcb {
namespace host {

constexpr size_t kChunk = size_t(2) << 20;  // bytes per pinned buffer
constexpr int kMaxThreads = 8;

// One thread's share: chunks first, first + step, ...  buffers: two kChunk buffers.
inline bool copy_share(void* host, void* device, size_t bytes, bool upload, unsigned char* buffers, size_t first,
                       size_t step, int gpu) {
  if (cudaSetDevice(gpu) != cudaSuccess) return false;
  cudaStream_t stream = nullptr;
  cudaEvent_t done[2] = {nullptr, nullptr};
  bool ok = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) == cudaSuccess;
  for (auto& e : done) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  unsigned char* h = static_cast<unsigned char*>(host);
  unsigned char* d = static_cast<unsigned char*>(device);
  size_t waiting[2] = {SIZE_MAX, SIZE_MAX};  // offset of the download a buffer holds
  auto drain = [&](int b) {
    ok = ok && cudaEventSynchronize(done[b]) == cudaSuccess;
    if (ok && !upload && waiting[b] != SIZE_MAX)
      std::memcpy(h + waiting[b], buffers + b * kChunk, std::min(kChunk, bytes - waiting[b]));
    waiting[b] = SIZE_MAX;
  };
  int b = 0;
  for (size_t at = first * kChunk; ok && at < bytes; at += step * kChunk, b ^= 1) {
    const size_t n = std::min(kChunk, bytes - at);
    unsigned char* pinned = buffers + b * kChunk;
    drain(b);
    if (!ok) break;
    if (upload) {
      std::memcpy(pinned, h + at, n);
      ok = cudaMemcpyAsync(d + at, pinned, n, cudaMemcpyHostToDevice, stream) == cudaSuccess;
    } else {
      ok = cudaMemcpyAsync(pinned, d + at, n, cudaMemcpyDeviceToHost, stream) == cudaSuccess;
      waiting[b] = at;
    }
    ok = ok && cudaEventRecord(done[b], stream) == cudaSuccess;
  }
  drain(b);  // the older of the two first
  drain(b ^ 1);
  if (stream) {
    cudaStreamSynchronize(stream);  // no copy still reads the buffers
    cudaStreamDestroy(stream);
  }
  for (auto& e : done)
    if (e) cudaEventDestroy(e);
  return ok;
}

// Copies `bytes` and returns when they have arrived.  pinned: staging of any
// size from two chunks on; every 2 * kChunk of it feeds one thread.
inline bool copy(void* host, void* device, size_t bytes, bool upload, void* pinned, size_t pinned_bytes) {
  int gpu = 0;
  if (cudaGetDevice(&gpu) != cudaSuccess) return false;
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
  const size_t n = std::min({pinned_bytes / (2 * kChunk), chunks, size_t(kMaxThreads), size_t(cores)});
  if (n == 0) return false;
  unsigned char* buffers = static_cast<unsigned char*>(pinned);
  std::vector<char> ok(n, 0);
  std::vector<std::thread> threads;
  threads.reserve(n);
  auto share = [&](size_t i) {
    ok[i] = copy_share(host, device, bytes, upload, buffers + i * 2 * kChunk, i, n, gpu) ? 1 : 0;
  };
  size_t started = 1;
  try {
    for (; started < n; ++started) threads.emplace_back(share, started);
  } catch (...) {
    // No more threads, or no memory for one: the calling thread takes the remaining
    // shares.  Nothing may leave here while threads run: their destructors would abort.
  }
  share(0);
  for (size_t i = started; i < n; ++i) share(i);
  for (auto& t : threads) t.join();
  return std::all_of(ok.begin(), ok.end(), [](char c) { return c != 0; });
}

}  // namespace host
}  // namespace rcb
