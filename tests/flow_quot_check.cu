// Host check of the flow sweeps' quotient with a reciprocal known beforehand (flowRecip, flowQuot of
// pdem_flow.cuh): the bits of a / b on random operands over the whole range of exponents, around the bounds
// between which the corrections are taken, and on divisors whose significand is all ones or next to it.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "pdem_flow.cuh"

template <class R, class U>
static long check(int mantissa, int bias, int maxExp, int pairs) {
  std::mt19937_64 rng(17);
  const U ones = (U(1) << mantissa) - 1;
  auto make = [&](int kind, int mid) {  // an operand: kind 0 any exponent, 1 within 40 of mid, 2 special
    U u = (U)rng() & ones;
    if (kind == 2) {
      const R special[] = {R(0), R(-0.0), R(1), R(-1), R(INFINITY), R(-INFINITY), R(NAN), R(1e-38), R(3e38f)};
      return special[rng() % 9];
    }
    const int e = kind == 0 ? (int)(rng() % (maxExp + 1)) : bias + mid + (int)(rng() % 81) - 40;
    const int pick = (int)(rng() % 8);
    if (pick < 3)
      u = pick == 0 ? ones : (pick == 1 ? ones - 1 : U(rng() % 4));
    u |= U(e < 0 ? 0 : (e > maxExp ? maxExp : e)) << mantissa;
    u |= U(rng() & 1) << (sizeof(U) * 8 - 1);
    R r;
    std::memcpy(&r, &u, sizeof r);
    return r;
  };
  // the bounds' exponents: a and b are compared with 1e+-100 (double), 1e+-10 and 1e15 / 1e-25 (float)
  const int mids[] = {0, 332, -332, 33, -33, 50, -83};
  long bad = 0;
  for (int k = 0; k < pairs; ++k) {
    const R a = make(k % 50 == 0 ? 2 : k % 3 ? 1 : 0, mids[rng() % 7]);
    const R b = make(k % 47 == 0 ? 2 : k % 3 ? 1 : 0, mids[rng() % 7]);
    const R got = pdem::flowQuot<R>(a, pdem::flowRecip<R>(b)), want = a / b;
    if (std::memcmp(&got, &want, sizeof got) && !(std::isnan(got) && std::isnan(want))) {
      if (bad++ < 5)
        std::printf("%a / %a = %a, not %a\n", (double)a, (double)b, (double)want, (double)got);
    }
  }
  return bad;
}

int main() {
  const long d = check<double, uint64_t>(52, 1023, 2046, 4000000), f = check<float, uint32_t>(23, 127, 254, 4000000);
  std::printf("double %ld float %ld differ\n", d, f);
  return d || f ? 1 : 0;
}
