// A fresh result array has no pages yet; a device copy into it would fault them in
// one by one (some 4 us each), and far from the core that reads them next.  They are
// touched, contents kept, by another thread while the device works, or by the caller.
#pragma once
#include <stddef.h>

#include <system_error>
#include <thread>

inline void touch_pages(double* a, size_t count) {
  volatile char* p = (volatile char*)a;
  for (size_t q = 0; p && q < count * sizeof(double); q += 4096) p[q] = p[q];
}

// Joined when it goes out of scope, however that happens.
class PageToucher {
 public:
  PageToucher() = default;
  PageToucher(const PageToucher&) = delete;
  PageToucher& operator=(const PageToucher&) = delete;
  ~PageToucher() { join(); }
  // Two arrays, one after the other; false if there is no thread to be had.
  bool start(double* a, size_t na, double* b, size_t nb) {
    try {
      th_ = std::thread([=] {
        touch_pages(a, na);
        touch_pages(b, nb);
      });
    } catch (const std::system_error&) {
      return false;
    }
    return true;
  }
  void join() {
    if (th_.joinable()) th_.join();
  }

 private:
  std::thread th_;
};
