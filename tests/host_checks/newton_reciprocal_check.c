/* Host check of the reciprocal in the exact Gelu of the contraction epilogue (gelu_erf2 in
 * oxionnx_b200/csrc/umma_kernel.cuh): t = fma(r, fma(-d, r, 1), r), one Newton step with a fused residual on an
 * approximation r of 1/d, must be the correctly rounded quotient 1/d for every float d from 1 to 2^100, except where
 * Markstein's theorem makes its one exception: d's significand is all ones and r is the power of two below 1/d.  Of those
 * d the Gelu could only meet 2 - 2^-23 (from 4 - 2^-22 on the factor exp(-x^2) leaves nothing of t in 1 - t * q * exp), and
 * d = 1 + 0.3275911 x takes that value for no float x.
 *
 * rcp.approx.ftz.f32 is documented to be off by at most one unit in the last place, so r is any float within one such
 * unit of 1/d: all of them are tried, for each of the 2^23 significands.  The exponent needs no loop: scaling d by a power of
 * two scales r, t and the quotient by its inverse exactly (down to 2^-100 every value is normal, and the residual
 * fma(-d, r, 1) does not change).  Both ends are tried anyhow.
 * Prints "significands N tried M exceptions E bad B", exit status 1 when B > 0. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static float u2f(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}
static uint32_t f2u(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}

int main(void) {
  long tried = 0, bad = 0, exceptions = 0, significands = 0;
  static const int exponents[] = {0, 1, 50, 99};
  for (int ei = 0; ei < 4; ++ei)
    for (uint32_t m = 0; m < (1u << 23); ++m) {
      const float d = u2f((uint32_t)(127 + exponents[ei]) << 23 | m);
      const float want = 1.0f / d;
      const double exact = 1.0 / (double)d; /* off by 2^-53 of it: far less than the units compared below */
      significands += ei == 0;
      for (int k = -2; k <= 2; ++k) {
        const float r = u2f(f2u(want) + (uint32_t)k);
        int e;
        frexp(exact, &e); /* exact in [2^(e-1), 2^e): one unit in the last place is 2^(e-24) */
        if (fabs((double)r - exact) > ldexp(1.0, e - 24)) continue;
        tried++;
        const float t = fmaf(r, fmaf(-d, r, 1.0f), r);
        if (t != want && m == 0x7fffff && (f2u(r) & 0x7fffff) == 0) {
          exceptions++;
        } else if (t != want) {
          if (bad < 10) printf("d=%a r=%a got=%a want=%a\n", d, r, t, want);
          bad++;
        }
      }
    }
  const float ones = u2f(0x3fffffffu); /* 2 - 2^-23 */
  long met = 0;
  for (float x = 3.0f; x < 3.1f; x = nextafterf(x, 4.0f)) { /* d grows with x: 1.98 .. 2.02 */
    volatile float product = x * 0.3275911f;
    volatile float d = 1.0f + product;
    met += d == ones;
  }
  bad += met;
  printf("significands %ld tried %ld exceptions %ld bad %ld\n", significands, tried, exceptions, bad);
  return bad != 0;
}
