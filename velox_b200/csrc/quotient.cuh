// Quotients by a prepared divisor. A host-side check defines VXD, __fmaf_rn and
// __float_as_uint before including this.
#pragma once
#include <cstdint>

#ifndef VXD
#define VXD __device__ __forceinline__
#endif

namespace vxb {

// Correctly rounded x / k from y = 1 / k (correctly rounded): Markstein's
// theorem (IBM J. Res. Dev. 34, 1990), q + (x - k q) y rounded once is the
// quotient when q is within an ulp of it, which the first correction makes
// it. Five dependent operations instead of the general division's reciprocal,
// refinement and range branch (about 20 against 80 cycles). Exact while no
// remainder underflows: k in [2^-30, 2^30] (quotientBase), x zero or in
// [2^-80, 2^60] (quotientRange). A zero quotient may carry the other sign.
VXD float quotient(float x, float k, float y) {
    const float q = x * y;
    const float p = __fmaf_rn(__fmaf_rn(-k, q, x), y, q);
    return __fmaf_rn(__fmaf_rn(-k, p, x), y, p);
}
VXD bool quotientRange(float x) {
    const uint32_t b = __float_as_uint(x) << 1;  // exponent and mantissa
    return (b - (47u << 24) <= (140u << 24)) | (b == 0u);
}
VXD bool quotientBase(float k) { return k >= 9.5e-10f && k <= 1.0e9f; }

}  // namespace vxb
