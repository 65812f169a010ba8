// sin and cos of an FP64 argument by table lookup (device).
//
// Table-driven evaluation (P. T. P. Tang, "Table-lookup algorithms for elementary functions and
// their error analysis", ARITH 1991): x = n (2 pi / N) + r with N = 256 and |r| <= pi / N, the
// table entry (cos, sin)(2 pi n / N), and the Taylor polynomials of sin r and cos r - 1 (first
// terms left out: r^7 / 5040 < 9e-18 and r^8 / 40320 < 2e-20).  2 pi / N is held as C1 + C2 to 106
// bits; the fused multiply-adds keep r to one rounding while |n| < 2^40.  The absolute error is about
// 2^-53 (the last rounding) plus the table entry's own (sincospi's).
// 15 FP64 operations and one 16-byte shared-memory load against about twice the operations (and a
// branch) for the library's sincos.
#pragma once

#include <cuda_runtime.h>

namespace bgw {

constexpr int kPhaseTable = 256;            // N
constexpr double kPhaseMax = 1.0e9;         // largest |x| the reduction is meant for

// Fills the table (N entries of shared memory) with the threads of a block.
__device__ __forceinline__ void phase_table_fill(double2* tab) {
    for (int q = threadIdx.x; q < kPhaseTable; q += blockDim.x) {
        double s, c;
        sincospi((double)q * (2.0 / kPhaseTable), &s, &c);
        tab[q] = make_double2(c, s);
    }
}

__device__ __forceinline__ void table_sincos(const double2* __restrict__ tab, double x, double& s, double& c) {
    constexpr double kInv = 40.74366543152521;          // N / (2 pi)
    constexpr double kC1 = 0.02454369260617026;         // 2 pi / N rounded to double
    constexpr double kC2 = 9.567553118338697e-19;       // 2 pi / N - C1
    constexpr double kMagic = 6755399441055744.0;       // 1.5 2^52: x + kMagic rounds x to an integer
    const double t = fma(x, kInv, kMagic);
    const double2 e = tab[__double2loint(t) & (kPhaseTable - 1)];
    const double n = t - kMagic;
    const double r = fma(n, -kC2, fma(n, -kC1, x));
    const double r2 = r * r;
    const double sr = fma(fma(r2, 1.0 / 120.0, -1.0 / 6.0) * r2, r, r);                         // sin r
    const double cm = fma(fma(r2, -1.0 / 720.0, 1.0 / 24.0), r2, -0.5) * r2;                     // cos r - 1
    c = fma(-e.y, sr, fma(e.x, cm, e.x));
    s = fma(e.x, sr, fma(e.y, cm, e.y));
}

}  // namespace bgw
