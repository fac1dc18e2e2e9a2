// Test driver: raise_smem_limits (device.h) with a fake of cudaFuncSetAttribute that fails at each
// call in turn. Prints "ok" or the first failure; exit code 0 on success.
#include "device.h"

#include <cstdio>

using namespace idx2g;

int main()
{
  const char kernels[4] = {};
  const std::initializer_list<kernel_smem> list = {
    { kernels, 100 }, { kernels + 1, 200 }, { kernels + 2, 300 }, { kernels + 3, 400 }
  };
  for (int bad = 0; bad <= 4; ++bad)
  {
    bool done = false;
    int calls = 0;
    size_t limit[4] = {};
    auto set = [&](const void* k, size_t n) {
      if (calls++ == bad)
        return false;
      limit[(const char*)k - kernels] = n;
      return true;
    };
    const bool ok = raise_smem_limits(&done, list, set);
    if (ok != (bad == 4) || done != ok)
    {
      std::printf("FAIL call %d: %d %d\n", bad, ok, done);
      return 1;
    }
    // the next call raises what is missing, the one after it nothing
    if (!raise_smem_limits(&done, list, set) || !done)
    {
      std::printf("FAIL not raised after %d\n", bad);
      return 1;
    }
    const int before = calls;
    if (!raise_smem_limits(&done, list, set) || calls != before)
    {
      std::printf("FAIL raised again after %d\n", bad);
      return 1;
    }
    for (int i = 0; i < 4; ++i)
      if (limit[i] != 100 * (size_t)(i + 1))
      {
        std::printf("FAIL limit %d\n", i);
        return 1;
      }
  }
  std::printf("ok\n");
  return 0;
}
