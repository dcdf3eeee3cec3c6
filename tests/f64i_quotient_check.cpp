// Host check of f64i_quotient_f32 (diffrax_gb300/csrc/gbdx_f64i.cuh): the place of a save
// in its step against the long-double quotient.  Usage: <n_random> <seed>; prints the
// largest error in units of 2^-24 of the quotient, exits 1 above 1 + 2^-12 of them (the
// last rounding is half a binary32 ulp, at most 2^-24 of the value) or on a wrong
// special case.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "gbdx_f64i.cuh"

using namespace gbdx;

static uint64_t g_state;
static double unif() {
  g_state = g_state * 6364136223846793005ull + 1442695040888963407ull;
  return double(g_state >> 11) * 0x1.0p-53;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  g_state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
  double worst = 0.0;
  long bad = 0;
  for (long i = 0; i < n; i++) {
    // a step and a save at any place in it, next to its ends too
    const double b = exp2(-80.0 + 130.0 * unif()) * (i & 1 ? 1.0 : -1.0);
    double th = unif();
    if (i % 4 == 1) th = exp2(-50.0 * th);
    if (i % 4 == 2) th = 1.0 - exp2(-50.0 * th);
    if (i % 4 == 3) th = float(th);
    const double a = b * th;
    const float q = f64i_quotient_f32(a, b);
    const long double x = (long double)a / (long double)b;
    if (x != 0.0L) worst = fmax(worst, double(fabsl(((long double)q - x) / x) * 0x1.0p24L));
    bad += f64i_quotient_f32(b, b) != 1.f || f64i_quotient_f32(0.0, b) != 0.f || q > 1.f;
  }
  // outside the two-part range the division itself
  const double ed[] = {1e-300, 1e-45, 1e-30, 1e20, 1e300, 1.0, INFINITY, NAN};
  for (double a : ed)
    for (double b : ed) {
      const float q = f64i_quotient_f32(a, b), x = float(a / b);
      bad += !((q != q && x != x) || q == x);
    }
  printf("quotient worst %.6f units, %ld wrong\n", worst, bad);
  return worst > 1.0 + 0x1.0p-12 || bad ? 1 : 0;
}
