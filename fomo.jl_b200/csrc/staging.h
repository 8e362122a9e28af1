// staging.h -- copies through a ring of staging slots, filled by helper threads.
#pragma once
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace fomo {

// Moves chunks 0 .. n - 1 through `slots` slots, chunk k through slot k % slots:
//   wait(slot)      the copy that last read the slot is done   (any thread)
//   fill(k, slot)   chunk k into the slot                      (any thread)
//   issue(k, slot)  starts the copy out of the slot            (calling thread, in order of k)
// Only the calling thread issues: cudaStreamPerThread is one handle that names another
// stream on every thread, so what a helper enqueued there would not be ordered before what
// the caller enqueues next.  The callables return 0 or an error code; the first error ends
// the copy and is returned.  With no helper (none wanted, or no thread to be had) the caller
// fills every slot itself.
template <class Wait, class Fill, class Issue>
int staged_copy(size_t n, size_t slots, int helpers, Wait wait, Fill fill, Issue issue) {
  std::mutex mu;
  std::condition_variable cv;
  size_t next = 0, issued = 0;          // chunks claimed by a filler, chunks issued
  std::vector<size_t> full(slots, 0);   // chunk + 1 that a slot holds
  int err = 0;
  // claims and fills the next chunk; `lk` holds mu on entry and exit
  auto fill_next = [&](std::unique_lock<std::mutex>& lk) {
    const size_t k = next++, slot = k % slots;
    cv.wait(lk, [&] { return err || k < issued + slots; });  // the slot's last chunk is issued
    if (err) return;
    lk.unlock();
    int e = wait(slot);
    if (!e) e = fill(k, slot);
    lk.lock();
    if (e) {
      if (!err) err = e;
    } else {
      full[slot] = k + 1;
    }
    cv.notify_all();
  };
  std::vector<std::thread> th;
  try {
    for (int i = 0; i < helpers; ++i)
      th.emplace_back([&] {
        std::unique_lock<std::mutex> lk(mu);
        while (!err && next < n) fill_next(lk);
      });
  } catch (...) {  // no thread or no memory for one
  }
  std::unique_lock<std::mutex> lk(mu);
  for (size_t k = 0; k < n && !err; ++k) {
    const size_t slot = k % slots;
    cv.wait(lk, [&] { return err || full[slot] == k + 1 || next == k; });
    if (!err && full[slot] != k + 1) fill_next(lk);  // nobody has claimed chunk k
    if (err) break;
    lk.unlock();
    const int e = issue(k, slot);
    lk.lock();
    if (e) {
      if (!err) err = e;
    } else {
      ++issued;
    }
    cv.notify_all();
  }
  lk.unlock();
  for (auto& t : th) t.join();
  return err;
}

}  // namespace fomo
