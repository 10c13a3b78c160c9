// Host build of the integer-pipe comparisons of the laws (liggghts-inl_gb300/
// csrc/contact_law.cuh: order_key, key_lt, key_gt, gt_nonneg) against the plain ones, for
// every pair of a table of doubles.  Built and called by tests/test_order_key.py.
#include <math.h>
#include <stdint.h>
#include <string.h>

inline long long __double_as_longlong(double x) {
  long long b;
  memcpy(&b, &x, sizeof b);
  return b;
}
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double rsqrt(double x) { return 1.0 / sqrt(x); }
template <class T>
inline T __ldg(const T *p) {
  return *p;
}

#include "contact_law.cuh"

using namespace gb300;

// wrong answers; a: key_lt and key_gt take a NaN on the side that may hold one
extern "C" int check_order(const double *x, int n) {
  int wrong = 0;
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      const double a = x[i], b = x[j];
      if (!isnan(a)) {
        wrong += key_lt(order_key(a), b) != (a < b);
        wrong += key_gt(b, order_key(a)) != (b > a);
      }
      if (!isnan(a) && !isnan(b)) {
        wrong += (order_key(a) > order_key(b)) != (a > b);
        wrong += (order_key(a) >= order_key(b)) != (a >= b);
        if (!signbit(a) && !signbit(b)) wrong += gt_nonneg(a, b) != (a > b);
      }
      // a distance that is NaN is within nothing
      if (isnan(b) && !isnan(a) && !signbit(a)) wrong += gt_nonneg(a, b);
    }
  return wrong;
}
