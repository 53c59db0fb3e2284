// Host check of the friction term's cube root (de_plain.cuh dcbrt) and of
// h^(7/3) formed with it, against the long double library.
//
// Bounds.  With y from FP32 within 2^-22.6 of the root (operand cut 2^-23, a
// third of it in the root; library 1 ulp) e = (h - y^3) / h is below 2^-21.
// The series' third term 14/81 e^3 is then below 2^-65.5 of the result and the
// roundings in the correction (4 of 2^-53, on a term of e / 3) below 2^-73:
// with the final rounding the error stays below 0.5 + 2^-12 ulp.  The long double
// root is allowed one unit of its own 64 bits, 2^-10 ulp here.  h^(7/3) takes
// three roundings of at most 2^-53, each at most an ulp of the result.
// Prints the largest errors in ulp and exits non-zero beyond the bounds;
// outside 2^-100 .. 2^100 the library's cbrt is used as it is.
#include <cmath>
#include <cstdio>
#include <random>
struct int4 { int x, y, z, w; };
#include "../../anuga_core_gb300/csrc/de_plain.cuh"

static long g_bad = 0;
static double g_root = 0.0, g_power = 0.0;

static double ulps(double got, long double want) {
  int e;
  std::frexp((double)want, &e);
  return (double)(std::fabs((long double)got - want) / std::ldexp(1.0L, e - 53));
}

static void check(double h) {
  const double got = agx::dcbrt(h);
  if (h < std::ldexp(1.0, -100) || h >= std::ldexp(1.0, 101)) {
    if (!(got == std::cbrt(h))) g_bad++;
    return;
  }
  const long double r = cbrtl((long double)h);
  const double u = ulps(got, r);
  g_root = std::fmax(g_root, u);
  if (!(u <= 0.5 + 0.000244140625 + 0.0009765625)) {
    if (g_bad++ < 10) std::printf("cbrt(%.17g): %.17g, %.4f ulp\n", h, got, u);
  }
  const double p = ulps(agx::h_pow_7_3(h), (long double)h * (long double)h * r);
  g_power = std::fmax(g_power, p);
  if (!(p <= 3.0)) {
    if (g_bad++ < 10) std::printf("h^(7/3) of %.17g: %.4f ulp\n", h, p);
  }
}

int main() {
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> u(1.0, 8.0);
  std::uniform_int_distribution<int> any(-100, 98), depth(-40, 14);
  for (int it = 0; it < 3000000; it++) {
    check(std::ldexp(u(rng), depth(rng)));
    check(std::ldexp(u(rng), any(rng)));
  }
  for (int e = -1074; e <= 1023; e++) {          // the ends of every binade and cubes, the switch at 2^+-100 among them
    const double p = std::ldexp(1.0, e);
    check(p);
    check(std::nextafter(p, 0.0) > 0.0 ? std::nextafter(p, 0.0) : p);
    check(std::nextafter(p, 2.0 * p));
  }
  for (int i = 1; i < 20000; i++) check((double)i * i * i);
  std::printf("largest error: root %.5f ulp, power %.5f ulp; failures %ld\n", g_root, g_power, g_bad);
  return g_bad ? 1 : 0;
}
