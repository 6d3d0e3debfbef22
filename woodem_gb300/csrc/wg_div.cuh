// Correctly rounded FP64 quotients by a divisor whose reciprocal is at hand.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so a division is a dozen slots of the pipe that
// bounds the FP64 kernels. Where several numerators share a divisor b (the components of a vector
// and its norm, a force and its node's mass) one reciprocal z = RN(1/b) serves all of them:
//   q = RN(a z),  r = RN(a - b q),  a / b = RN(q + r z)
// which is the correctly rounded quotient when nothing over- or underflows (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34(1), 1990; N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans. Comput. 53(8), 2004):
// bit for bit what `a / b` gives, in one multiplication and two FMAs. Outside the exponent range in
// which every intermediate is normal (and for negative, zero or non-finite divisors) the
// plain division is used.
#pragma once
#include "wg_math.cuh"

namespace wg {

// positive, exponent within [-500, 500]
__device__ __forceinline__ bool divisorInRange(double b) { return ((unsigned)__double2hiint(b) >> 20) - 523u <= 1000u; }
// zero, or exponent within [-500, 500]
__device__ __forceinline__ bool numeratorInRange(double a) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return (h >> 20) - 523u <= 1000u || (h | (unsigned)__double2loint(a)) == 0u;
}
__device__ __forceinline__ double quotient(double a, double b, double z) {
    const double q = __dmul_rn(a, z);
    const double v = __fma_rn(__fma_rn(-b, q, a), z, q);
    // a zero keeps its sign (the sum of the two FMAs would lose that of -0)
    return (((unsigned)__double2hiint(a) & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0u ? a : v;
}
// out of line: inlined, the plain divisions would become predicated FP64 instructions in every warp
static __device__ __noinline__ D3 divPlain(D3 a, double b) { return D3{a.x / b, a.y / b, a.z / b}; }
static __device__ __noinline__ D3 divPlain3(D3 a, D3 b) { return D3{a.x / b.x, a.y / b.y, a.z / b.z}; }

// a / b, z = RN(1/b)
__device__ __forceinline__ D3 divBy(D3 a, double b, double z) {
    if (!(divisorInRange(b) && numeratorInRange(a.x) && numeratorInRange(a.y) && numeratorInRange(a.z))) return divPlain(a, b);
    return D3{quotient(a.x, b, z), quotient(a.y, b, z), quotient(a.z, b, z)};
}
__device__ __forceinline__ D3 divBy(D3 a, double b) { return divBy(a, b, __drcp_rn(b)); }
// component by component, z = RN(1/b) of each
__device__ __forceinline__ D3 divBy3(D3 a, D3 b, D3 z) {
    if (!(divisorInRange(b.x) && divisorInRange(b.y) && divisorInRange(b.z) && numeratorInRange(a.x) && numeratorInRange(a.y) &&
          numeratorInRange(a.z)))
        return divPlain3(a, b);
    return D3{quotient(a.x, b.x, z.x), quotient(a.y, b.y, z.y), quotient(a.z, b.z, z.z)};
}
// Eigen's normalize(), as wg_math.cuh's normalized()
__device__ __forceinline__ D3 normalizedQ(D3 a) {
    const double z = sqn(a);
    return z > 0 ? divBy(a, sqrt(z)) : a;
}
static __device__ __noinline__ DQ qdivPlain(DQ q, double n) { return DQ{q.w / n, q.x / n, q.y / n, q.z / n}; }
__device__ __forceinline__ DQ qnormalizedQ(DQ q) {
    const double n = sqrt(((q.x * q.x + q.y * q.y) + q.z * q.z) + q.w * q.w);
    if (!(divisorInRange(n) && numeratorInRange(q.w) && numeratorInRange(q.x) && numeratorInRange(q.y) && numeratorInRange(q.z)))
        return qdivPlain(q, n);
    const double z = __drcp_rn(n);
    return DQ{quotient(q.w, n, z), quotient(q.x, n, z), quotient(q.y, n, z), quotient(q.z, n, z)};
}

}  // namespace wg
