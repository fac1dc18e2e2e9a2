// Copies between device memory and pageable host memory (a numpy array, a malloc'd buffer).
//
// cudaMemcpyAsync takes such a buffer through the driver's own staging on the calling thread,
// page faults of a fresh array included: 38 MB into a new numpy array took 8.2 ms, 4.6 GB/s. Here
// up to 12 threads take pieces of 1 MB, each through a pinned piece of its own, so that the
// faults, the host copies and the transfers of different pieces overlap (that copy: 1.7 ms, 16 host
// cores). Copies of less than 4 MB stay one cudaMemcpyAsync, as threads would cost more than they save
// (12 of them start in some 0.2 ms), and so do those to or from memory that CUDA knows: pinned, where
// there is nothing to save, and managed memory or a device's, which cudaMemcpyAsync takes too and the
// host copy may not reach.
#pragma once

#include "device.h"

#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

namespace idx2g
{

constexpr size_t kHostPiece = (size_t)1 << 20;
constexpr size_t kHostCopyMin = (size_t)4 << 20;
constexpr unsigned kHostCopyThreads = 12;

inline bool is_memory(const void* p, cudaMemoryType type)
{
  cudaPointerAttributes pa;
  const bool is = cudaPointerGetAttributes(&pa, p) == cudaSuccess && pa.type == type;
  cudaGetLastError();
  return is;
}
inline bool is_pinned(const void* p) { return is_memory(p, cudaMemoryTypeHost); }
// memory that CUDA does not know; managed memory, or a device pointer given as a host one, is neither
inline bool is_pageable(const void* p) { return is_memory(p, cudaMemoryTypeUnregistered); }

// `bytes` from src to dst, one of them in device memory (to_host: src), in order after the work
// of stream `st`. On return a copy to the host is done, or enqueued on `st` where it took the
// plain form; a pageable source is no longer read. Returns an error code; then nothing is in flight
// on `st` any more, neither the copies of the threads nor earlier ones of the caller's.
inline int host_copy(device_ctx* ctx, void* dst, const void* src, size_t bytes, bool to_host, cudaStream_t st)
{
  const size_t n = (bytes + kHostPiece - 1) / kHostPiece;
  unsigned nt = std::thread::hardware_concurrency();
  nt = nt > kHostCopyThreads ? kHostCopyThreads : nt;
  if (nt > n)
    nt = (unsigned)n;
  uint8_t* slots = nullptr;
  if (bytes >= kHostCopyMin && nt >= 2 && is_pageable(to_host ? dst : src))
    slots = (uint8_t*)ctx->pinned("host.slots", nt * kHostPiece);
  for (unsigned t = 0; slots && t < nt; ++t)
    if (!ctx->copy_ev(t))
      slots = nullptr;
  if (!slots)
  {
    if (cudaMemcpyAsync(dst, src, bytes, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st) == cudaSuccess)
      return NoError;
    cudaStreamSynchronize(st);
    return CudaError;
  }
  std::atomic<size_t> next{ 0 };
  std::atomic<int> bad{ 0 };
  auto work = [&](unsigned t) {
    uint8_t* slot = slots + t * kHostPiece;
    const cudaEvent_t ev = ctx->copy_events[t];
    bool ok = cudaSetDevice(ctx->device) == cudaSuccess;
    for (size_t k; ok && (k = next.fetch_add(1)) < n;)
    {
      const size_t o = k * kHostPiece, b = bytes - o < kHostPiece ? bytes - o : kHostPiece;
      if (!to_host)
        memcpy(slot, (const uint8_t*)src + o, b);
      ok = (to_host ? cudaMemcpyAsync(slot, (const uint8_t*)src + o, b, cudaMemcpyDeviceToHost, st)
                    : cudaMemcpyAsync((uint8_t*)dst + o, slot, b, cudaMemcpyHostToDevice, st)) == cudaSuccess &&
           cudaEventRecord(ev, st) == cudaSuccess && cudaEventSynchronize(ev) == cudaSuccess;
      if (ok && to_host)
        memcpy((uint8_t*)dst + o, slot, b);
    }
    if (!ok)
      bad = 1;
  };
  std::vector<std::thread> th;
  th.reserve(nt);
  try
  {
    for (unsigned t = 1; t < nt; ++t)
      th.emplace_back(work, t);
  }
  catch (const std::system_error&)
  {
    // fewer threads than asked for
  }
  work(0);
  for (auto& t : th)
    t.join();
  if (!bad)
    return NoError;
  cudaStreamSynchronize(st);
  return CudaError;
}

} // namespace idx2g
