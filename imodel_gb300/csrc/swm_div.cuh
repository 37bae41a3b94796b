// FP64 division by a divisor whose reciprocal is known in advance (internal
// header of the FP64 kernels).
#pragma once
#include <cuda_runtime.h>

namespace imodel {

// RN(1 / 6), rounded on the host
constexpr double kSixth = 1.0 / 6.0;

static __device__ __noinline__ double div_full(double a, double b) { return a / b; }

// a / b rounded to nearest, as IEEE division rounds it, from rb = RN(1 / b):
// one product and two fused corrections, q = RN(a rb), r = RN(a - q b), q' =
// RN(q + r rb), which give RN(a / b) when rb is correctly rounded and nothing
// under- or overflows (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; N.
// Brisebarre, J.-M. Muller and S. K. Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans.
// Comput. 53, 2004).  Three FP64 operations; a / b compiles to about ten on
// GB300's FP64 pipe, which bounds the step.  A quotient outside 2^-895 ..
// 2^896 (zero, infinities, NaN and every divisor with rb = NaN among them)
// takes the division itself, so every input gets a / b.  rb is given for |b|
// from kRecipLow to kRecipHigh: a smaller b with a quotient in range could have
// a remainder below the normal numbers.
__device__ __forceinline__ double div_by(double a, double b, double rb) {
  const double q = a * rb;
  const double z = __fma_rn(__fma_rn(-q, b, a), rb, q);
  const unsigned ex = (static_cast<unsigned>(__double2hiint(q)) >> 20) & 0x7FFu;
  if (ex - 128u < 1792u) return z;
  // zeros are common (fluid at rest, switched-off sources): a rb has 0 / b's
  // sign
  if (((__double2hiint(a) << 1) | __double2loint(a)) == 0 && ex == 0) return q;
  return div_full(a, b);
}

}  // namespace imodel
