// The thread that touches result pages: joined when the call that started it ends by
// an exception, and no loss when no thread can be started.
#include <sys/resource.h>
#include <unistd.h>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <stdexcept>
#include <vector>

#include "page_touch.h"

#define CHECK(x)                                \
  if (!(x)) {                                   \
    std::printf("line %d: %s\n", __LINE__, #x); \
    return 1;                                   \
  }

int main() {
  {  // no room for a thread's stack (first: the C library keeps the stacks of ended threads)
    std::vector<double> c(10, 1.5);
    std::ifstream f("/proc/self/statm");
    long pages = 0;
    f >> pages;
    rlimit old, lim;
    CHECK(getrlimit(RLIMIT_AS, &old) == 0);
    lim = old;
    lim.rlim_cur = (rlim_t)pages * (rlim_t)sysconf(_SC_PAGESIZE) + (1 << 20);
    CHECK(setrlimit(RLIMIT_AS, &lim) == 0);
    PageToucher t;
    CHECK(!t.start(c.data(), c.size(), nullptr, 0));
    CHECK(setrlimit(RLIMIT_AS, &old) == 0);
  }
  const size_t n = (size_t)1 << 24;
  double* a = (double*)std::calloc(n, sizeof(double));
  std::vector<double> b(1000, 3.5);
  CHECK(a);
  bool caught = false;
  try {
    PageToucher t;
    CHECK(t.start(a, n, b.data(), b.size()));
    throw std::runtime_error("a call that fails meanwhile");
  } catch (const std::runtime_error&) {
    caught = true;
  }
  CHECK(caught);
  for (size_t q = 0; q < n; q += 511) CHECK(a[q] == 0.0);
  for (double v : b) CHECK(v == 3.5);
  {
    PageToucher t;
    CHECK(t.start(nullptr, n, b.data(), b.size()));  // no L wanted
    t.join();
    t.join();
  }
  std::free(a);
  std::puts("ok");
  return 0;
}
