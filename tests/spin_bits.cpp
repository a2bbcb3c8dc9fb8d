// The short forms of the FP64 particle update (pg_math.cuh, host build)
// against the general ones, bit for bit: exp_terms against exp_series, the
// settled spin update against spin_iso, and an unturned rotation against the
// product with exp(0).  Random values over many magnitudes, zeros of both
// signs, powers of two, subnormals, infinities and NaNs.  Prints cases,
// mismatches, and how many of each short form were taken.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "../parmec_gb300/csrc/pg_math.cuh"

using namespace pg;

static std::mt19937_64 g(7);
static double uni() { return (g() >> 11) * 0x1p-53; }
static double sgn() { return g() & 1 ? 1.0 : -1.0; }
static bool same(double a, double b) { return dbits(a) == dbits(b) || (a != a && b != b); }

// a value of magnitude 10^lo .. 10^hi, now and then a special one
static double value(double lo, double hi, int special)
{
  if (special && g() % special == 0)
  {
    const double s[] = {0.0, -0.0, 1.0, -2.0, 0.25, 5e-324, -1e-310, INFINITY, -INFINITY, NAN, 1e200, -1e-200};
    return s[g() % 12];
  }
  return sgn() * pow(10.0, lo + (hi - lo) * uni());
}

int main(int argc, char **argv)
{
  const long n = argc > 1 ? atol(argv[1]) : 200000;
  long cases = 0, bad = 0, spin = 0, turn = 0;
  for (long i = 0; i < 4 * n; i ++)
  {
    const double a = fabs(i % 4 ? pow(10.0, -20.0 + 18.0 * uni()) : pow(10.0, -9.0 + 4.0 * uni()));
    double s0, c0, s1, c1;
    exp_series(a, &s0, &c0);
    exp_terms(a, &s1, &c1);
    cases ++;
    bad += !same(s0, s1) || !same(c0, c1);
  }
  for (long i = 0; i < n; i ++)
  {
    const int special = i % 3 ? 0 : 6;
    const double r = pow(10.0, -4.0 + 4.0 * uni()), js = 0.4 * 2500.0 * 4.19 * r*r*r*r*r;
    const double is = i % 7 ? 1.0 / js : value(-3.0, 12.0, 9), step = pow(10.0, -8.0 + 6.0 * uni()), half = 0.5 * step;
    double O[3], T[3], a[3], b[3], Ta[3];
    const double w = -6.0 + 9.0 * uni(), q = -14.0 + 14.0 * uni();
    for (int k = 0; k < 3; k ++) { O[k] = value(w - 2.0 * (i & 1), w, special); T[k] = js * value(q, q + 4.0, special); }
    if (i % 5 == 0) T[0] = T[1] = T[2] = g() & 1 ? 0.0 : -0.0;
    if (i % 11 == 0) O[0] = O[1] = O[2] = 0.0;
    for (int k = 0; k < 3; k ++) { a[k] = b[k] = O[k]; Ta[k] = T[k]; }
    cases ++;
    if (!gyro_settled(O, T, js, is, step, half)) continue;
    spin ++;
    spin_iso(a, Ta, js, is, step, half, i & 1);
    bool torque = false;
    for (int k = 0; k < 3; k ++) torque |= T[k] != 0.0;
    for (int k = 0; k < 3; k ++) if (torque) b[k] = b[k] + is*(step*T[k]);
    for (int k = 0; k < 3; k ++) bad += !same(a[k], b[k]);
  }
  for (long i = 0; i < n; i ++)
  {
    double L[9], DL[9], A[9], o[3], z[3] = {0.0, 0.0, 0.0};
    const int special = i % 4 ? 0 : 12;
    for (int k = 0; k < 9; k ++) L[k] = value(-3.0, 0.0, special);
    const double h = value(-8.0, 0.0, 10);
    cases ++;
    if (!turn_is_identity(L, h)) continue;
    turn ++;
    expmap(h*z[0], h*z[1], h*z[2], DL, i & 1);
    nnmul(L, DL, A);
    nvmul(A, z, o);
    for (int k = 0; k < 9; k ++) bad += !same(A[k], L[k]);
    for (int k = 0; k < 3; k ++) bad += dbits(o[k]) != (dbits(L[k]) & dbits(L[3+k]) & dbits(L[6+k]) & 0x8000000000000000ull);
  }
  printf("%ld %ld %ld %ld\n", cases, bad, spin, turn);
  return 0;
}
