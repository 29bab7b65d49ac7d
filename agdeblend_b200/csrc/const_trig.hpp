// cos and sin of 2 pi m / n at compile time, in double precision, so that the
// register DFTs of odd length have literal coefficients.  The angle is
// reduced to at most pi / 4 in whole numbers first: a Taylor sum at an angle
// near pi cancels, and the rounding of the angle itself grows with it (rms
// error over the odd lengths 5 to 27: cosines 0.4e-16 and sines 0.3e-16;
// unreduced 1.1e-16 and 1.5e-16, the library's functions of the rounded
// angle 0.8e-16 and 1.0e-16).
#pragma once

namespace agd {

// Taylor sums about 0 at x in [0, pi / 4], in Horner form
constexpr double taylor_cos(double x) {
  double s = 1.0;
  for (int i = 10; i >= 1; --i) s = 1.0 - s * (x * x) / ((2.0 * i - 1.0) * (2.0 * i));
  return s;
}
constexpr double taylor_sin(double x) {
  double s = 1.0;
  for (int i = 10; i >= 1; --i) s = 1.0 - s * (x * x) / ((2.0 * i) * (2.0 * i + 1.0));
  return x * s;
}

constexpr double turn_angle(int a, int b) { return 6.283185307179586476925286766559 * a / b; }

// at a / b of a turn, 0 <= 4 a <= b (above an eighth: pi / 2 less the angle)
constexpr double quarter_cos(int a, int b) {
  return 8 * a > b ? taylor_sin(turn_angle(b - 4 * a, 4 * b)) : taylor_cos(turn_angle(a, b));
}
constexpr double quarter_sin(int a, int b) {
  return 8 * a > b ? taylor_cos(turn_angle(b - 4 * a, 4 * b)) : taylor_sin(turn_angle(a, b));
}

// at m / n of a turn, 0 <= m <= n
constexpr double const_cos(int m, int n) {
  if (2 * m > n) m = n - m;
  return 4 * m > n ? -quarter_cos(n - 2 * m, 2 * n) : quarter_cos(m, n);
}
constexpr double const_sin(int m, int n) {
  if (2 * m > n) return -const_sin(n - m, n);
  return 4 * m > n ? quarter_sin(n - 2 * m, 2 * n) : quarter_sin(m, n);
}

}  // namespace agd
