// Host tables of the FFT engine.
#pragma once
#include <cmath>
#include <vector>

namespace c3d {

// exp(-2 pi i q r / n) of the stage over the whole span, radix R: [r][q], q < n/R
template <typename C>
std::vector<C> edge_twiddles(int n, int R) {
  std::vector<C> t(n);
  const long double pi = 3.141592653589793238462643383279502884L;
  const int M = n / R;
  for (int r = 0; r < R; ++r)
    for (int q = 0; q < M; ++q) {
      const long double a = -2.0L * pi * (long double)((long long)q * r % n) / (long double)n;
      t[(size_t)r * M + q].x = (decltype(C::x))cosl(a);
      t[(size_t)r * M + q].y = (decltype(C::x))sinl(a);
    }
  return t;
}

}  // namespace c3d
