// divide_by (relax_math.cuh) against the IEEE division, compared as bits, on the host: random
// operands, divisors with all-ones mantissas, both ends of its guarded range, zeros of either sign,
// infinities and NaN.  Divisors span 2^-20..2^20; the diagonals that are divided by lie in 1..9.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>

#include "relax_math.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t next() {
  state ^= state << 13;
  state ^= state >> 7;
  return state ^= state << 17;
}

template <typename T, typename U, int MANT, int BIAS>
static long run(int top, int guard, long count) {
  auto make = [](uint64_t sign, int e, uint64_t m) {
    const U w = (U)((U)(sign & 1) << (8 * sizeof(T) - 1) | (U)(e + BIAS) << MANT | ((U)m & (((U)1 << MANT) - 1)));
    T v;
    std::memcpy(&v, &w, sizeof(v));
    return v;
  };
  long bad = 0;
  auto check = [&](T n, T d) {
    const T got = ocub::divide_by(n, d, (T)1 / d), want = n / d;
    const bool same = std::memcmp(&got, &want, sizeof(T)) == 0 || (std::isnan(got) && std::isnan(want));
    if (!same && bad++ < 4) std::printf("%a / %a: %a, not %a\n", (double)n, (double)d, (double)got, (double)want);
  };
  const uint64_t ones = ~0ull;
  for (long t = 0; t < count; t++) {
    const uint64_t a = next(), b = next(), c = next();
    const uint64_t md = t % 3 == 0 ? b : t % 3 == 1 ? ones : ones << (b % 8);
    const T d = make(0, (int)(c % 41) - 20, md);
    check(make(a >> 63, (int)((c >> 8) % (2 * top + 1)) - top, a), d);
    for (int e : {-guard - 1, -guard, guard - 1, guard}) check(make(a >> 62, e, t % 2 ? a : t % 4 ? 0 : ones), d);
    const T inf = std::numeric_limits<T>::infinity();
    for (T n : {(T)0, -(T)0, inf, -inf, std::numeric_limits<T>::quiet_NaN(), std::numeric_limits<T>::denorm_min(),
                -std::numeric_limits<T>::min(), std::numeric_limits<T>::max()})
      check(n, d);
  }
  return bad;
}

int main() {
  const long f = run<float, uint32_t, 23, 127>(100, 90, 1000000), d = run<double, uint64_t, 52, 1023>(900, 800, 1000000);
  std::printf("%ld float and %ld double quotients differ\n", f, d);
  return f || d;
}
