// Host thread pool for the pack, write and open stages: f(i) for i in [0, n) on up to 32
// threads (the calling thread included), items handed out one at a time.
#pragma once

#include <atomic>
#include <cstddef>
#include <exception>
#include <functional>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace idx2g
{

template <typename F>
void parallel_for(size_t n, F&& f)
{
  unsigned nt = std::thread::hardware_concurrency();
  nt = nt ? (nt > 32 ? 32 : nt) : 4;
  if (nt > n)
    nt = (unsigned)(n ? n : 1);
  std::atomic<size_t> next{ 0 };
  auto work = [&]() {
    for (size_t i; (i = next.fetch_add(1)) < n;)
      f(i);
  };
  std::vector<std::thread> th;
  for (unsigned t = 1; t < nt; ++t)
    th.emplace_back(work);
  work();
  for (auto& t : th)
    t.join();
}

// f(i0, i1) over [0, n) cut into about 8 ranges per thread
template <typename F>
void parallel_ranges(size_t n, F&& f)
{
  unsigned nt = std::thread::hardware_concurrency();
  nt = nt ? (nt > 32 ? 32 : nt) : 4;
  const size_t nr = (size_t)nt * 8;
  const size_t step = (n + nr - 1) / nr;
  if (!step)
    return;
  parallel_for((n + step - 1) / step, [&](size_t r) {
    const size_t i0 = r * step;
    f(i0, i0 + step < n ? i0 + step : n);
  });
}

// A function that runs on a thread of its own beside its maker, or inside wait() where no thread
// is to be had. wait() returns once it has run, and throws what it threw, which must not leave the
// thread (the process would end there); a task destroyed without wait() is joined.
class side_task
{
public:
  explicit side_task(std::function<void()> f) : f_(std::move(f))
  {
    try
    {
      thread_ = std::thread([this] { run(); });
    }
    catch (const std::system_error&)
    {
      // no thread: wait() runs it
    }
  }
  ~side_task()
  {
    if (thread_.joinable())
      thread_.join();
  }
  side_task(const side_task&) = delete;
  side_task& operator=(const side_task&) = delete;
  void wait()
  {
    if (thread_.joinable())
      thread_.join();
    else if (f_)
      run();
    if (error_)
      std::rethrow_exception(std::exchange(error_, nullptr));
  }

private:
  void run()
  {
    try
    {
      f_();
    }
    catch (...)
    {
      error_ = std::current_exception();
    }
    f_ = nullptr;
  }
  std::function<void()> f_;
  std::exception_ptr error_;
  std::thread thread_;
};

} // namespace idx2g
