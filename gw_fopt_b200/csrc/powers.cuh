// Powers of the separable scaling (device).
#pragma once

#include <cuda_runtime.h>

namespace bgw {

// x^p: binary powering for integral |p| <= 32 (a few ulp), pow() otherwise.
__device__ __forceinline__ double tpow(double x, double p) {
    const double r = rint(p);
    if (r == p && fabs(r) <= 32.0) {
        unsigned n = (unsigned)fabs(r);
        double acc = 1.0, b = x;
        while (n) {
            if (n & 1u) acc *= b;
            b *= b;
            n >>= 1;
        }
        return r < 0.0 ? 1.0 / acc : acc;
    }
    return pow(x, p);
}

}  // namespace bgw
