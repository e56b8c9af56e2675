// quotient.h -- a / b in REAL from the rounded reciprocal of b.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define RTB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define RTB_HOST_DEVICE inline
#endif

namespace rtb {

// a / b rounded to nearest, r the reciprocal of b rounded to nearest: the estimate
// a r corrected by its exact remainder (Markstein, IBM J. Res. Dev. 34, 1990, on
// divisions by fused multiply-adds).  For many numerators over one b: three
// operations and a select each.  An infinite a, whose remainder is NaN, keeps the
// estimate.
RTB_HOST_DEVICE float quotient(float a, float b, float r) {
    const float q = a * r;
    const float p = fmaf(fmaf(-b, q, a), r, q);
    return p == p ? p : q;
}

}  // namespace rtb
