// 1 / d in FP64 by Newton's method, for the refinement's solve.
#pragma once

#include <math.h>

#include "detmath.h"

namespace bdmath {

// 1 / d for 1e-12 <= d < 3.4e38 (float's range): Newton steps r + r (1 - d r) from the
// float reciprocal, whose error of 2^-23 each step squares, so that the last
// rounding alone is left: within one unit in the last place of the quotient.
// FP64 is narrow on this GPU, and a division is twice as many of its instructions.
BDM_FN double reciprocal(double d) {
#if defined(__CUDA_ARCH__)
    double r = static_cast<double>(__frcp_rn(static_cast<float>(d)));
    r = __fma_rn(r, __fma_rn(-d, r, 1.0), r);
    return __fma_rn(r, __fma_rn(-d, r, 1.0), r);
#else
    double r = static_cast<double>(1.0f / static_cast<float>(d));
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
#endif
}

}  // namespace bdmath
