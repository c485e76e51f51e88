// div_by_recip and div_by_pair (csrc/row_stencil.cuh) against the divide on
// the host: random numerators and divisors over the whole range of the type,
// the ends of the ranges in which it corrects a product, significands of all
// ones, zeros of both signs, subnormals, infinities and NaN. Prints the pairs
// whose bits differ; NaN equals NaN.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "row_stencil.cuh"

template <typename T, typename U> static U bits(T v) {
  U u;
  memcpy(&u, &v, sizeof(u));
  return u;
}

template <typename T, typename U> static long run(const char *name) {
  using L = std::numeric_limits<T>;
  using R = pmg::DivRange<T>;
  std::mt19937_64 rng(7);
  std::vector<T> special;
  const T ends[] = {R::c_min, R::c_max, R::q_min, R::q_max, T(1), T(3),
                    L::min(), L::denorm_min(), L::max(), L::min() * 3};
  for (T e : ends)
    for (T v : {e, std::nextafter(e, T(0)), std::nextafter(e, L::infinity())})
      for (T s : {v, -v})
        special.push_back(s);
  for (T v : {T(0), L::infinity()})
    for (T s : {v, -v})
      special.push_back(s);
  special.push_back(L::quiet_NaN());
  auto any = [&]() { // any bit pattern
    const U u = (U)rng();
    T v;
    memcpy(&v, &u, sizeof(v));
    return v;
  };
  std::uniform_real_distribution<double> mant(1.0, 2.0);
  auto near_one = [&](int e) { // about 2^-e .. 2^e, all ones now and then
    T m = (T)mant(rng);
    if (rng() % 8 == 0)
      m = T(2) - L::epsilon();
    return std::ldexp(m, (int)(rng() % (2 * e)) - e);
  };
  long bad = 0, n = 0;
  auto same = [&](T s, T c, T got) {
    const T want = s / c;
    ++n;
    if (std::isnan(got) && std::isnan(want))
      return;
    if (bits<T, U>(got) != bits<T, U>(want) && ++bad <= 5)
      printf("%s: %a / %a = %a, not %a\n", name, (double)s, (double)c,
             (double)want, (double)got);
  };
  auto check = [&](T s, T c) {
    same(s, c, pmg::div_by_recip(s, c, pmg::recip_of(c)));
    if constexpr (sizeof(T) == sizeof(float))
      same(s, c, pmg::div_by_pair(s, pmg::recip_pair(c)));
  };
  for (T s : special)
    for (T c : special)
      check(s, c);
  for (int q = 0; q < 300000; ++q) {
    check(any(), any());
    check(any(), near_one(20)); // divisors as operators have them
    check(near_one(20), near_one(20));
    const T c = near_one(20);
    check(std::ldexp(near_one(3), L::min_exponent + (int)(rng() % 80) - 20),
          c);
    for (T s : special)
      if (q % 100 == 0)
        check(s, c);
    // quotients midway between two subnormals
    const T even = (T)(2 + 2 * (rng() % 60));
    check(even * (T)(1 + 2 * (rng() % 2000)) / 2 * L::denorm_min(), even);
  }
  printf("%s: %ld of %ld differ\n", name, bad, n);
  return bad;
}

int main() {
  return run<float, uint32_t>("float") + run<double, uint64_t>("double") ? 1
                                                                         : 0;
}
