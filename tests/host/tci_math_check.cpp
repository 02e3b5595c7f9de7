// tci_exp, tci_cos and division by a constant against the same steps written with
// plain operations (rint, separate products, IEEE division), bit for bit, over the
// usual range of arguments, its ends and beyond.
#pragma GCC optimize("fp-contract=off")  // as the header asks
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <cmath>

#include "tci_functions.h"

static double plain_exp(double x) {
  if (x != x) return x;
  if (x > 709.782712893384) return INFINITY;
  if (x < -745.1332191019412) return 0.0;
  const double n = std::rint(x * TCI_INV_LN2);
  volatile double h = n * TCI_LN2_HI, l = n * TCI_LN2_LO;
  const double r = (x - h) - l;
  return tci_scale2(tci_exp_poly(r), (int)n);
}
static double plain_cos(double x) {
  if (x - x != 0.0) return x - x;
  const double n = std::rint(x * TCI_TWO_OVER_PI);
  volatile double a = n * TCI_PIO2_1, b = n * TCI_PIO2_2, c = n * TCI_PIO2_3;
  const double r = ((x - a) - b) - c;
  switch ((int)((int64_t)n & 3)) {
    case 0: return tci_cos_poly(r);
    case 1: return -tci_sin_poly(r);
    case 2: return -tci_cos_poly(r);
    default: return tci_sin_poly(r);
  }
}

static uint64_t s = 88172645463325252ull;
static uint64_t rn() {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
static bool same(double a, double b) { return memcmp(&a, &b, 8) == 0 || (a != a && b != b); }
static int bad = 0;
static void check(double x) {
  const IntDivisor d4 = tci_const_divisor(0x001a36e2eb1c432dull, 0x3f100000u, 0x9c3ffffffffffde4ull);
  const IntDivisor d2 = tci_const_divisor(0x00147ae147ae147bull, 0x3f800000u, 0xc7fffffffffffed4ull);
  const double got[4] = {tci_exp(x), std::fabs(x) < 4e6 || x - x != 0.0 ? tci_cos(x) : 0.0, tci_quo(x, 1e-4, d4),
                         tci_quo(x, 0.01, d2)};
  const double want[4] = {plain_exp(x), std::fabs(x) < 4e6 || x - x != 0.0 ? plain_cos(x) : 0.0, x / 1e-4, x / 0.01};
  for (int k = 0; k < 4; ++k)
    if (!same(got[k], want[k]) && ++bad < 10) printf("%d at %a: %a, not %a\n", k, x, got[k], want[k]);
}

int main() {
  const double edges[] = {0.0, 704.0, 709.782712893384, 745.1332191019412, 708.3, 1048576.0, 0.5, 1e-320, 1e-300,
                          0.34657359027997264, 0.7853981633974483, 1.5707963267948966, 3.141592653589793, INFINITY,
                          NAN, 1e300, 2147483648.0};
  for (double e : edges)
    for (int k = -3; k <= 3; ++k)
      for (int sign = 0; sign < 2; ++sign) {
        uint64_t b;
        memcpy(&b, &e, 8);
        b += (uint64_t)(int64_t)k;
        b ^= (uint64_t)sign << 63;
        double x;
        memcpy(&x, &b, 8);
        check(x);
      }
  for (int i = 0; i < 2000000; ++i) {
    const double u = (double)(int64_t)rn() * 0x1p-63;  // (-1, 1)
    check(u);
    check(u * 800.0);
    check(u * 7000.0);
    check(u * 2e6);
    check(std::rint(u * 700.0 * TCI_INV_LN2 * 2) / TCI_INV_LN2 / 2);       // near the reduction's edges
    check(std::rint(u * 1e5) * 0.7853981633974483);                         // near multiples of pi / 4
    uint64_t b = rn();
    double x;
    memcpy(&x, &b, 8);
    check(x);
  }
  printf(bad ? "%d differ\n" : "ok\n", bad);
  return bad != 0;
}
