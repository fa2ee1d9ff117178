// Large host arrays to and from the device through a pinned staging buffer, the
// host side of the copy on several threads.
//
// A copy between pageable host memory and the device is bound by one host thread
// moving it through the driver's staging area (about 11 GB/s) and, into a fresh
// array, taking its page faults (3 GB/s); the link carries about 50.  Here the
// arrays are cut into chunks: worker threads move chunks between the arrays and
// the slots of the staging buffer while the caller's thread enqueues the
// transfers of the slots in order.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/rfxb200.h"

namespace {

constexpr int kSlots = 8;

struct Chunk {
  char* host;
  char* dev;
  size_t bytes;
};

struct Slots {
  cudaEvent_t ev[kSlots] = {};
  bool ok = true;
  Slots() {
    for (auto& e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) ok = false;
  }
  ~Slots() {
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
  }
};

int copy_chunks(const std::vector<Chunk>& chunks, bool to_host, char* stage, size_t slot_bytes, cudaStream_t st) {
  const int n = (int)chunks.size();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RFXB_E_LAUNCH;
  Slots slots;
  if (!slots.ok) return RFXB_E_LAUNCH;
  std::atomic<int> next{0}, issued{0};   // next chunk of the workers; transfers enqueued
  std::atomic<bool> err{false};
  std::unique_ptr<std::atomic<char>[]> done(new std::atomic<char>[n]());   // the worker's part of a chunk
  auto work = [&]() {
    if (cudaSetDevice(dev) != cudaSuccess) err = true;
    for (int k = next++; k < n && !err; k = next++) {
      char* slot = stage + (size_t)(k % kSlots) * slot_bytes;
      // to the host: the chunk's own transfer; to the device: the slot's last one
      const int need = to_host ? k : k - kSlots;
      while (issued.load(std::memory_order_acquire) <= need && !err) std::this_thread::yield();
      if (err) break;
      if (need >= 0 && cudaEventSynchronize(slots.ev[k % kSlots]) != cudaSuccess) { err = true; break; }
      if (to_host) std::memcpy(chunks[k].host, slot, chunks[k].bytes);
      else std::memcpy(slot, chunks[k].host, chunks[k].bytes);
      done[k].store(1, std::memory_order_release);
    }
  };
  std::vector<std::thread> workers;
  const unsigned hc = std::thread::hardware_concurrency();
  const int want = (int)std::min<unsigned>(8u, std::max(1u, hc / 2));
  try {
    workers.reserve(want);
    for (int t = 0; t < std::min(want, n); ++t) workers.emplace_back(work);
  } catch (...) {   // as many as could be started
  }
  if (workers.empty()) {
    for (const Chunk& c : chunks) {
      const cudaError_t e = to_host ? cudaMemcpyAsync(c.host, c.dev, c.bytes, cudaMemcpyDeviceToHost, st)
                                    : cudaMemcpyAsync(c.dev, c.host, c.bytes, cudaMemcpyHostToDevice, st);
      if (e != cudaSuccess) return RFXB_E_LAUNCH;
    }
    return cudaStreamSynchronize(st) == cudaSuccess ? RFXB_OK : RFXB_E_LAUNCH;
  }
  for (int k = 0; k < n && !err; ++k) {
    const int need = to_host ? k - kSlots : k;   // the worker's part that comes before this transfer
    while (need >= 0 && !done[need].load(std::memory_order_acquire) && !err) std::this_thread::yield();
    if (err) break;
    char* slot = stage + (size_t)(k % kSlots) * slot_bytes;
    const Chunk& c = chunks[k];
    if ((to_host ? cudaMemcpyAsync(slot, c.dev, c.bytes, cudaMemcpyDeviceToHost, st)
                 : cudaMemcpyAsync(c.dev, slot, c.bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        cudaEventRecord(slots.ev[k % kSlots], st) != cudaSuccess) {
      err = true;
      break;
    }
    issued.store(k + 1, std::memory_order_release);
  }
  for (std::thread& t : workers) t.join();
  // the staging buffer is free again when its last transfers are over
  if (cudaStreamSynchronize(st) != cudaSuccess) err = true;
  return err ? RFXB_E_LAUNCH : RFXB_OK;
}

int copy_arrays(int n, void* const* host, void* const* dev, const int64_t* bytes, bool to_host, void* stage,
                int64_t stage_bytes, void* stream) {
  if (n <= 0 || !host || !dev || !bytes || !stage || stage_bytes < kSlots * 4096) return RFXB_E_INVALID;
  try {
    const size_t slot = (size_t)stage_bytes / kSlots / 4096 * 4096;
    std::vector<Chunk> chunks;
    for (int q = 0; q < n; ++q) {
      if (bytes[q] < 0 || (bytes[q] > 0 && (!host[q] || !dev[q]))) return RFXB_E_INVALID;
      for (size_t o = 0; o < (size_t)bytes[q]; o += slot)
        chunks.push_back(Chunk{static_cast<char*>(host[q]) + o, static_cast<char*>(dev[q]) + o,
                               std::min(slot, (size_t)bytes[q] - o)});
    }
    if (chunks.empty()) return RFXB_OK;
    return copy_chunks(chunks, to_host, static_cast<char*>(stage), slot, static_cast<cudaStream_t>(stream));
  } catch (...) {
    return RFXB_E_NOMEM;
  }
}

}  // namespace

extern "C" {

int rfxb_copy_to_host(int n, void* const* host, void* const* dev, const int64_t* bytes, void* stage,
                      int64_t stage_bytes, void* stream) {
  return copy_arrays(n, host, dev, bytes, true, stage, stage_bytes, stream);
}

int rfxb_copy_to_device(int n, void* const* host, void* const* dev, const int64_t* bytes, void* stage,
                        int64_t stage_bytes, void* stream) {
  return copy_arrays(n, host, dev, bytes, false, stage, stage_bytes, stream);
}

}  // extern "C"
