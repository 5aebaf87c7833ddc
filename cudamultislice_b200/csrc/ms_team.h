// ms_team.h -- a share of host work per thread.
#pragma once
#include <cstddef>
#include <thread>

namespace ms {

// work(0) .. work(n - 1), each exactly once, on up to n <= MAX threads (share 0
// on the caller's); returns when all are done.  A thread that cannot be started,
// be it for lack of threads or of memory, leaves its share and the following ones
// to the caller's: no started thread is ever dropped unjoined.  work must not
// throw.
template <size_t MAX, class F>
void run_team(size_t n, const F& work) {
  std::thread th[MAX];
  size_t started = 1;
  try {
    for (; started < n && started < MAX; ++started) th[started] = std::thread(work, started);
  } catch (...) {
  }
  work(0);
  for (size_t t = started; t < n; ++t) work(t);
  for (size_t t = 1; t < started; ++t) th[t].join();
}

}  // namespace ms
