// face_len (scheme_math.cuh) against the reference's sqrt((0 + a a) + b b) on
// the host: components over the whole exponent range, in particular around
// the ratio from which the smaller one's square no longer counts, squares next
// to powers of two, zeros.  Prints the number of differences.
#include <cmath>
#include <cstdio>
#include <random>

#include "kernels/scheme_math.cuh"

int main() {
  std::mt19937_64 g(20261205);
  long long bad = 0, n = 0;
  auto check = [&](double a, double b) {
    volatile double aa = a * a, bb = b * b;
    volatile double r = 0.0 + aa;
    r = r + bb;
    const double want = std::sqrt(r);
    const double got = hydro::face_len(a, b);
    ++n;
    if (hydro::ubits(want) != hydro::ubits(got) && !(want != want && got != got)) ++bad;
  };
  auto mant = [&]() {
    const unsigned long long x = g();
    switch (x & 3) {
      case 0: return 1.0;                               // a power of two
      case 1: return 2.0 - 0x1p-52;                     // just below one
      case 2: return 1.0 + 0x1p-52 * (double)(x >> 61);  // just above one
      default: return 1.0 + (double)(g() >> 12) * 0x1p-52;
    }
  };
  for (int k = 0; k < 6000000; ++k) {
    const int ea = (int)(g() % 1400) - 700;
    const int d = (int)(g() % 64) - 4;  // the other component 2^-d of it
    double a = std::ldexp(mant(), ea), b = std::ldexp(mant(), ea - d);
    if (g() & 1) a = -a;
    if (g() & 1) b = -b;
    if ((g() & 1023) == 0) b = 0.0;
    check(a, b);
    check(b, a);
  }
  std::printf("%lld %lld\n", n, bad);
  return bad != 0;
}
