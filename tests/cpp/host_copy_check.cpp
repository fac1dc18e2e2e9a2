// Test driver: host_copy (host_copy.h) over a fake CUDA runtime. "Device memory" is ordinary memory
// here; the fake counts the copies, and gives pointers the type that a case asks for. Runs the case
// named on the command line, prints "ok" or the first failure; exit code 0 on success.
#include "host_copy.h"

#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

using namespace idx2g;

namespace
{
cudaMemoryType g_type = cudaMemoryTypeUnregistered;
std::atomic<int> g_copies{ 0 };
std::atomic<size_t> g_events{ 0 };
std::mutex g_lock;
std::vector<cudaEvent_t> g_recorded;
int g_fail_copy = -1, g_fail_record = -1;  // the call, counted from 0, that fails
bool g_in_flight = false;                  // copies since the last wait for the stream
} // namespace

extern "C"
{
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
  memset(a, 0, sizeof *a);
  a->type = g_type;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t)
{
  {
    const std::lock_guard<std::mutex> lock(g_lock);
    if (g_copies == g_fail_copy)
      return cudaErrorInvalidValue;
    ++g_copies;
    g_in_flight = true;
  }
  memcpy(dst, src, n);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e)
{
  *e = (cudaEvent_t)(++g_events);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
  const std::lock_guard<std::mutex> lock(g_lock);
  if ((int)g_recorded.size() == g_fail_record)
    return cudaErrorInvalidResourceHandle;
  g_recorded.push_back(e);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
  const std::lock_guard<std::mutex> lock(g_lock);
  g_in_flight = false;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n)
{
  *p = malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
  free(p);
  return cudaSuccess;
}
} // extern "C"

namespace
{

int fail(const char* what, long long v)
{
  std::printf("FAIL %s %lld\n", what, v);
  return 1;
}

// n bytes each way; the number of copies it took, or -1 where they do not arrive
int copies_of(device_ctx* ctx, size_t n, bool to_host)
{
  std::vector<uint8_t> a(n), b(n, 0);
  for (size_t i = 0; i < n; ++i)
    a[i] = (uint8_t)(i * 31 + (i >> 8) + (i >> 16));
  g_copies = 0;
  if (host_copy(ctx, b.data(), a.data(), n, to_host, nullptr) != NoError || a != b)
    return -1;
  return g_copies;
}

// memory that CUDA knows (pinned, managed, a device's) stays one cudaMemcpyAsync, which takes any of
// them; only memory that it does not know goes through the threads
int registered()
{
  device_ctx ctx;
  const bool threads = std::thread::hardware_concurrency() >= 2;
  const size_t sizes[] = { 100, kHostCopyMin - 1, kHostCopyMin, kHostCopyMin + 3, 7 * kHostPiece + 12345 };
  for (size_t n : sizes)
    for (int to_host = 0; to_host < 2; ++to_host)
    {
      for (cudaMemoryType t : { cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged })
      {
        g_type = t;
        if (const int c = copies_of(&ctx, n, to_host != 0); c != 1)
          return fail("registered: copies", c);
      }
      g_type = cudaMemoryTypeUnregistered;
      const int want = n < kHostCopyMin || !threads ? 1 : (int)((n + kHostPiece - 1) / kHostPiece);
      if (const int c = copies_of(&ctx, n, to_host != 0); c != want)
        return fail("pageable: copies", c);
    }
  return 0;
}

// the threads' events are no event of the pool that encodes, decodes and the packer number for
// themselves (the packer one for every 32 MB of an image, without a bound)
int events()
{
  device_ctx ctx;
  std::vector<cudaEvent_t> pool;
  for (size_t i = 0; i < 400; ++i)
    pool.push_back(ctx.ev(i));
  g_type = cudaMemoryTypeUnregistered;
  g_recorded.clear();
  if (copies_of(&ctx, 5 * kHostPiece, true) < 1)
    return fail("events: copies", -1);
  for (cudaEvent_t e : g_recorded)
    for (size_t i = 0; i < pool.size(); ++i)
      if (e == pool[i])
        return fail("events: of the pool", (long long)i);
  return 0;
}

// a copy that fails, in either form and at any call, says so, and leaves none in flight on the stream:
// the caller returns with the error, and its buffers may go
int failures()
{
  device_ctx ctx;
  std::vector<uint8_t> a(6 * kHostPiece), b(6 * kHostPiece);
  g_type = cudaMemoryTypeUnregistered;
  for (size_t n : { (size_t)1000, b.size() })
    for (int to_host = 0; to_host < 2; ++to_host)
      for (int k = 0; k < 12; ++k)
      {
        g_copies = 0;
        g_recorded.clear();
        g_fail_copy = k % 2 ? -1 : k / 2;
        g_fail_record = k % 2 ? k / 2 : -1;
        if (n < kHostCopyMin && k)
          continue;
        g_in_flight = true;  // an earlier copy of the caller's
        if (host_copy(&ctx, b.data(), a.data(), n, to_host != 0, nullptr) == NoError &&
            std::thread::hardware_concurrency() >= 2)
          return fail("failures: not said", k);
        if (g_in_flight && std::thread::hardware_concurrency() >= 2)
          return fail("failures: in flight", k);
      }
  return 0;
}

} // namespace

int main(int argc, char** argv)
{
  const std::string name = argc > 1 ? argv[1] : "";
  int rc = 2;
  if (name == "registered")
    rc = registered();
  else if (name == "events")
    rc = events();
  else if (name == "failures")
    rc = failures();
  if (rc == 0)
    std::printf("ok\n");
  return rc;
}
