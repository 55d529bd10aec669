// The place of the largest of a row's uniform draws divided by their sum
// (the first maxr, pqdts.f90:1565-1575), for the device and, in its test, the
// host.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define PQDTS_HD __host__ __device__ __forceinline__
#else
#define PQDTS_HD inline
#endif

namespace pqdts {

// u 2^-53 for an integer u < 2^53, by its bits (the FP64 pipe, which a
// conversion takes, needs 64 cycles an instruction).
PQDTS_HD double draw_value(uint64_t u) {
  if (u == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int p = 63 - __clzll((long long)u);
#else
  const int p = 63 - __builtin_clzll(u);
#endif
  const uint64_t b = ((uint64_t)(969 + p) << 52) + (u << (52 - p));
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double v;
  std::memcpy(&v, &b, sizeof v);
  return v;
#endif
}

// draw(n): the n-th draw as an integer below 2^53.  The sum is added in order;
// the first largest quotient wins.  Quotients are ordered as the draws are
// unless two running maxima lie within 4 of one another (a distance of 5 is
// over two units in the last place of a quotient), where the quotients
// themselves decide.
template <class Draw>
PQDTS_HD int first_largest(Draw draw, int N) {
  double s = 0.0;
  uint64_t most = 0;
  int am = 0;
  bool close = false;
#pragma unroll 4
  for (int n = 0; n < N; ++n) {
    const uint64_t u = draw(n);
    s = s + draw_value(u);
    if (u > most) {
      close |= n > 0 && u - most < 5;
      most = u;
      am = n;
    }
  }
  if (!close) return am;
  double best = draw_value(draw(0)) / s;
  am = 0;
  for (int n = 1; n < N; ++n) {
    const double q = draw_value(draw(n)) / s;
    if (q > best) {
      best = q;
      am = n;
    }
  }
  return am;
}

}  // namespace pqdts
