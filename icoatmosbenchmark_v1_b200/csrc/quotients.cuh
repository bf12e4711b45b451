// Several FP64 quotients with one divisor.
#pragma once

namespace icoadv {

// Several quotients with one divisor, each the division's own result: y = 1/b is correctly rounded (an
// IEEE division), q1 = q0 + (a - b q0) y is faithful, and one more such step with its exact
// residual is a/b correctly rounded (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990).  The residuals are exact while nothing under- or overflows:
// quotients outside [2^-800, 2^1000) other than those of a zero, and divisors outside
// [2^-100, 2^101) (so all that are not positive), take the division itself.
// A zero keeps the sign a/b has, which the vertical limiter reads off a Courant number: the
// residual is formed as b q - a and subtracted.  With b > 0, a zero a gives q0 = +-0 of its own sign, the
// residual +0 for either (a - b q0 would be +0 too, and adding it would lose a -0), and q0 - (+0) y = q0.
struct Recip {
  double b, y;
  bool ok;
};
__device__ __forceinline__ bool recip_ok(double b) {
  return (unsigned)__double2hiint(b) - 0x39b00000u < 0x0c900000u;
}
__device__ __forceinline__ Recip recip(double b) { return Recip{b, 1.0 / b, recip_ok(b)}; }
template <int N>
__device__ __forceinline__ void quotients(double (&a)[N], const Recip &d) {
  double q[N];
  bool ok = d.ok;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double q0 = a[i] * d.y, q1 = __fma_rn(-__fma_rn(d.b, q0, -a[i]), d.y, q0);
    q[i] = __fma_rn(-__fma_rn(d.b, q1, -a[i]), d.y, q1);
    ok = ok && (((unsigned)__double2hiint(q[i]) & 0x7fffffffu) - 0x0df00000u < 0x70800000u || a[i] == 0.0);
  }
  if (ok) {
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = q[i];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = a[i] / d.b;
  }
}

}  // namespace icoadv
