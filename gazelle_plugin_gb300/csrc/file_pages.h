// The pages of the memory a data file's bytes are copied into (Splitter::EmitData), made present ahead of
// the copy.
#pragma once
#include <errno.h>
#include <fcntl.h>
#include <stdint.h>
#include <sys/uio.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

namespace gz {

// Makes the pages of bytes [lo, hi) of the fresh memory at `map` present; false when one of a mapping cannot
// be.
//
// A mapping's file system may be out of space for a page at any time (other writers, a user's quota), and
// a store would then be a SIGBUS.  So the kernel does it: readv of /dev/zero (`zero`, open for reading), a
// byte into every page, which returns an error instead.  Eight threads, tmpfs files of 47 / 283 / 720 MB: 0.7 /
// 2.9 / 6.7 ms (bare stores 0.6 / 2.5 / 6.2; MADV_POPULATE_WRITE, which moves every page to the active list
// under its lock, 1.3 / 7.0 / 16).  Where one thread works on each of many files, the space is allocated first
// (`file`, else -1) and stores follow: that is serial under a file's lock (with eight threads 1.0 / 4.7 / 12 ms),
// but the stores' faults take no lock of the address space, which the kernel's own do: 16 map tasks at
// once, 283 MB: 10.2 ms against 11.6.  Heap memory (zero: -1): stores.
inline bool MakePresent(uint8_t* map, int64_t lo, int64_t hi, int zero, int file) {
  const int64_t page = sysconf(_SC_PAGESIZE);
  // a byte of lo's page, then the first of each that follows
  auto next = [&](int64_t x) { return x + page - (int64_t)(reinterpret_cast<uintptr_t>(map + x) & (uintptr_t)(page - 1)); };
  bool stores = zero < 0;
  if (file >= 0) {
    int r;
    while ((r = fallocate(file, 0, lo, hi - lo)) != 0 && errno == EINTR) {
    }
    if (r != 0 && errno != EOPNOTSUPP && errno != ENOSYS) return false;
    stores = r == 0;
  }
  if (stores) {
    for (int64_t x = lo; x < hi; x = next(x)) *reinterpret_cast<volatile uint8_t*>(map + x) = 0;
    return true;
  }
  constexpr int kBytes = 512;  // a call (at most 1024 ranges, the system's limit)
  iovec v[kBytes];
  while (lo < hi) {
    int n = 0;
    for (int64_t x = lo; x < hi && n < kBytes; x = next(x)) v[n++] = iovec{map + x, 1};
    const ssize_t r = readv(zero, v, n);
    if (r > 0) lo = next(static_cast<uint8_t*>(v[r - 1].iov_base) - map);
    else if (r == 0 || errno != EINTR) return false;
  }
  return true;
}

// Makes the pages of fresh memory (a file's mapping, a heap block) present, in order, on helper threads
// and on the calling one whenever it has to wait.
class PageToucher {
 public:
  // [m, m + n) in windows of w bytes; zero (closed here) and file: as MakePresent takes them.
  PageToucher(uint8_t* m, int64_t n, int64_t w, int zero, int file = -1)
      : map_(m), total_(n), window_(w), unit_(w / 8), zero_(zero), file_(file), left_((size_t)((n + w - 1) / w)) {
    for (size_t i = 0; i < left_.size(); i++)
      left_[i].store((int)((std::min(w, n - (int64_t)i * w) + unit_ - 1) / unit_));
  }
  ~PageToucher() {
    if (zero_ >= 0) close(zero_);
  }
  PageToucher(const PageToucher&) = delete;
  PageToucher& operator=(const PageToucher&) = delete;

  int64_t unit() const { return unit_; }
  // One unit; false when there are none left.
  bool Work() {
    const int64_t lo = next_.fetch_add(unit_);
    if (lo >= total_) return false;
    if (!failed_.load() && !MakePresent(map_, lo, std::min(total_, lo + unit_), zero_, file_)) failed_.store(true);
    left_[(size_t)(lo / window_)].fetch_sub(1);
    return true;
  }
  // Until window w's pages are there; false when some page of the mapping cannot be.
  bool Wait(size_t w) {
    while (left_[w].load() > 0)
      if (!Work()) std::this_thread::yield();
    return !failed_.load();
  }

 private:
  uint8_t* const map_;
  const int64_t total_, window_, unit_;
  const int zero_, file_;
  std::atomic<int64_t> next_{0};
  std::vector<std::atomic<int>> left_;  // units of each window not touched yet
  std::atomic<bool> failed_{false};
};

}  // namespace gz
