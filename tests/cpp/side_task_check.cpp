// Test driver: side_task (parallel.h). Prints "ok" or the first failure; exit code 0 on success.
#include "parallel.h"

#include <chrono>
#include <cstdio>
#include <new>

using namespace idx2g;

int main()
{
  // what the function throws comes out of wait(), once, and not out of the thread
  for (int i = 0; i < 50; ++i)
  {
    side_task t([i] {
      if (i % 2)
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
      throw std::bad_alloc();
    });
    bool thrown = false;
    try
    {
      t.wait();
    }
    catch (const std::bad_alloc&)
    {
      thrown = true;
    }
    if (!thrown)
    {
      std::printf("FAIL not thrown\n");
      return 1;
    }
    t.wait();
  }
  // it runs once, has run after wait(), and is joined where nobody waits, throwing or not
  int runs = 0;
  {
    side_task t([&] { ++runs; });
    t.wait();
    t.wait();
    if (runs != 1)
    {
      std::printf("FAIL runs %d\n", runs);
      return 1;
    }
  }
  {
    side_task t([&] {
      std::this_thread::sleep_for(std::chrono::milliseconds(5));
      ++runs;
    });
    side_task u([] { throw 3; });
  }
  if (runs != 2)
  {
    std::printf("FAIL joined %d\n", runs);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
