// int_mul / int_mul_dense / int_div of ieee_int.h against the host's IEEE arithmetic, bit for
// bit, on random and structured significands over the whole int_safe range.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "ieee_int.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rn() {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
static double of(uint64_t b) {
  double d;
  memcpy(&d, &b, 8);
  return d;
}
static bool same(double a, double b) { return memcmp(&a, &b, 8) == 0; }
static double draw() {
  const uint64_t ones = (1ull << 52) - 1;
  uint64_t m = rn() & ones;
  switch (rn() % 8) {  // few significant bits (exact products and ties), next to a power of two
    case 1: m &= ~0ull << (rn() % 53); break;
    case 2: m = rn() & 3; break;
    case 3: m = ones - (rn() & 3); break;
    case 4: m &= ~0ull << (20 + rn() % 33); break;
    case 5: m = (m & ~0ull << 25) | 1ull << 25; break;  // the most trailing zeros of a dense factor
    default: break;
  }
  uint64_t e = 513 + rn() % 1022;
  if (rn() % 64 == 0) e = rn() % 2 ? 513 : 1534;
  if (rn() % 200 == 0) m = e = 0;
  return of((m & ones) | e << 52 | (rn() & 1) << 63);
}

int main() {
  for (int i = 0; i < 3000000; ++i) {
    const double x = draw(), y = draw();
    if (!int_safe(x) || !int_safe(y)) return printf("not safe: %a %a\n", x, y), 1;
    if (!same(int_mul(int_split(x), int_split(y)), x * y)) return printf("mul %a %a\n", x, y), 1;
    if (int_dense(x) && int_dense(y) && !same(int_mul_dense(dense_split(x), dense_split(y)), x * y))
      return printf("dense %a %a\n", x, y), 1;
    if (y != 0 && !same(int_div(x, int_divisor(y)), x / y)) return printf("div %a %a\n", x, y), 1;
  }
  for (uint64_t e : {0ull, 1ull, 512ull, 1535ull, 2046ull, 2047ull})  // outside the range, but for the zero
    for (uint64_t m : {0ull, 1ull, (1ull << 52) - 1})
      if (int_safe(of(m | e << 52)) != (e == 0 && m == 0)) return printf("safe %llu\n", (unsigned long long)e), 1;
  puts("ok");
  return 0;
}
