// Host check of the integer face flux (csrc/softflux.cuh): soft_flux(s, a, b) has the bits of the
// hardware's RN(s * RN(b - a)) for every operand triple it covers, soft_sub those of RN(b - a), and pack undoes unpack, over
// random bit patterns, values of near and far exponents, neighbours a few ulps apart, sparse and
// dense significands (ties), subnormals, huge values and specials.  Prints "cases N", "covered N"
// and "bad N"; for ordinary values (exponents within +-60) "uncovered" must be 0.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "softflux.cuh"

using namespace nebo;

static unsigned long long st;
static unsigned long long rnd() {
  st ^= st << 13;
  st ^= st >> 7;
  st ^= st << 17;
  return st * 2685821657736338717ull;
}
static double from(unsigned long long b) { return fixmath::from_bits(b); }
static unsigned long long bits(double d) { return fixmath::bits(d); }

static double draw(int mode, double near) {
  const unsigned long long r = rnd(), sign = r & (1ull << 63), m = r & 0xFFFFFFFFFFFFFull;
  switch (mode) {
    case 0: return from(r);
    case 1: return from(sign | ((unsigned long long)(1023 - 8 + rnd() % 16) << 52) | m);
    case 2: return near * (1 + ldexp((double)(long long)rnd(), -63 - (int)(rnd() % 60)));
    case 3: {
      unsigned long long q = (rnd() & 1) ? 0 : 0xFFFFFFFFFFFFFull;
      q ^= 1ull << (rnd() % 52);
      if (rnd() & 1) q &= ~((1ull << (rnd() % 52)) - 1);
      return from(sign | ((unsigned long long)(1023 - 35 + rnd() % 70) << 52) | q);
    }
    case 4: {
      const double sp[] = {0.0, -0.0, 1.0, -1.0, 5e-324, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                           INFINITY, -INFINITY, NAN, 0.5, 8.98846567431158e307};
      return sp[rnd() % 13];
    }
    case 5: return from(sign | ((unsigned long long)(rnd() % 60) << 52) | m);
    case 6: return from(sign | ((unsigned long long)(2046 - rnd() % 60) << 52) | m);
    default: return from(bits(near) + rnd() % 9 - 4);
  }
}

int main(int argc, char** argv) {
  const long n = atol(argv[1]);
  st = strtoull(argv[2], nullptr, 10) * 2654435761ull + 88172645463325252ull;
  long covered = 0, bad = 0, uncovered = 0;
  for (long i = 0; i < n; ++i) {
    const double a = draw((int)(rnd() % 7), 1.0), b = draw((int)(rnd() % 8), a), s = draw((int)(rnd() % 7), 1.0);
    const softfp::SoftVal A = softfp::unpack(a), B = softfp::unpack(b);
    if (bits(softfp::pack(A)) != bits(a)) ++bad;
    bool ok, okd;
    const double diff = softfp::soft_sub(A, B, okd);
    volatile double wantd = b - a;
    if (okd && bits(diff) != bits(wantd)) ++bad;
    const double got = softfp::soft_flux(s, A, B, ok);
    auto ordinary = [](double v) { return v == 0.0 ? !std::signbit(v) : (std::fabs(v) > 1e-18 && std::fabs(v) < 1e18); };
    if (!ok) {
      if (ordinary(a) && ordinary(b) && ((ordinary(s) && s != 0.0) || !okd)) ++uncovered;
      continue;
    }
    ++covered;
    volatile double d = b - a;
    volatile double want = s * d;
    if (bits(want) != bits(got)) ++bad;
  }
  std::printf("cases %ld\ncovered %ld\nuncovered %ld\nbad %ld\n", n, covered, uncovered, bad);
  return 0;
}
