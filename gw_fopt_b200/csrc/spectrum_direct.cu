// Plain FP64 spectrum: the default kernel, the tensor form and the time-resolved integrand.
//
// Per radiating bubble a, cos-theta row i and step k the reference forms
//   B_{g,s}(a,i,k) = sum_j q_g(j) f_s(t_k - t_a, tau_j),
//   f_s = 1 before the patch collides, sum_m a_{sm} (tau/dt)^{p_{sm}} e^{-(dt - tau)/width} after,
// and sums B e^{-i w dt c_i} over rows, then times e^{i w (t_k - z_a)} over steps and bubbles
// (generalized_bulk_flow.rs:481-873; the tensor form new_generalized_bulk_flow.rs:592-1203 has six
// weights q_g instead of cos 2phi and sin 2phi).  Here the two sums are two kernels:
//
//   k_direct_b  one warp per (frame, bubble, row, block of 32 NS steps), lane = step.  Collided and
//               uncollided patches are told apart by the reference's own comparison, so most patches
//               are in one state over the whole block; their sums are formed once, lanes over
//               patches.  Only the patches that collide inside the block are looked at step by step.
//               The scaling is separable: (tau/dt)^p e^{-(dt - tau)/width} is the product of a patch
//               factor with dt at the block's last step (at most 1) and a step factor.
//   k_direct_a  one warp per (frame, bubble, block of 32 steps, NW frequencies), lane = step: the row
//               sum with one phase per (row, step, frequency).  The phase argument w (-dt c_i) is
//               rounded as the reference rounds it.  Rows i and n_cos - 1 - i have c of opposite sign
//               up to rounding, so one table sincos serves both: the second argument is -x + e with e
//               formed exactly, and a first-order correction in e (|e| < 1e-10, e^2 below 2^-66).
//
// What bounds it: FP64 issue in k_direct_a (about 14 operations and 4 per column for each phase);
// k_direct_b is a few per cent.  The single kernel this replaces (one block per bubble, pow() for
// every patch and step, a barrier per step) took 53.6 ms for 5 bubbles x 50 x 100 patches x 800 steps
// x 120 w and 38.2 ms for 4 frames of 64 bubbles x 64 x 64 x 256 x 64 w with 3 sets; see the
// measured lines at the launches below.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "bgw_internal.h"
#include "device_common.cuh"
#include "fast_phase.cuh"
#include "powers.cuh"
#include "spectrum_direct.cuh"

namespace bgw {

namespace {

constexpr int kDirWarps = 8;

struct DirArgs {
    DirectInputs in;
    size_t n_tot;
    int n_sel, n_cos, n_phi, n_t, n_w;
    int S, M;
    int has_damp;
    double damp;
    double dphi, dcos, dt;
    size_t fs0;       // first (frame, slot) pair of this launch
    size_t n_fs;      // pairs
    int k0, k1;       // steps [k0, k1) of this launch, k0 a multiple of 32
    int tp;           // row length of B (multiple of 32)
    double* B;        // (n_fs, n_cos, S G, tp): column s G + g
};

// phi weight g of patch j without its trapezoid end weight
template <int G>
__device__ __forceinline__ double phi_weight(const DirArgs& A, int j, int g) {
    if constexpr (G == 2) return g == 0 ? A.in.cos2[j] : A.in.sin2[j];
    const double cp = A.in.cosphi[j], sp = A.in.sinphi[j];
    switch (g) {
        case 0: return __dmul_rn(cp, cp);
        case 1: return __dmul_rn(cp, sp);
        case 2: return cp;
        case 3: return __dmul_rn(sp, sp);
        case 4: return sp;
        default: return 1.0;
    }
}

// factor of weight g that depends on the row only
template <int G>
__device__ __forceinline__ double row_weight(double c, int g) {
    if constexpr (G == 2) return 0.5 * (1.0 - c * c);
    const double st = sqrt(fmax(__dsub_rn(1.0, __dmul_rn(c, c)), 0.0));
    switch (g) {
        case 0:
        case 1:
        case 3: return __dmul_rn(st, st);
        case 2:
        case 4: return __dmul_rn(st, c);
        default: return __dmul_rn(c, c);
    }
}

// sum_j of the row's weights with no patch collided, row factor included.  Over a full turn the
// weights cos 2phi, sin 2phi, ... add up to nothing but rounding, and a bubble that collides with
// nothing leaves only that in the result; so the terms are rounded and added as the reference does
// (ndarray's sum: eight partial sums over j mod 8, combined in pairs, then the tail).  Called by a
// whole warp; lane u < 8 forms partial sum u.
template <int G>
__device__ __forceinline__ void quiet_row(const DirArgs& A, double c, double (&sum)[G]) {
    const int lane = threadIdx.x & 31;
    const int nfull = A.n_phi & ~7;
    for (int g = 0; g < G; ++g) {
        const double rw = row_weight<G>(c, g);
        auto term = [&](int j) {
            const double x = G == 2 ? phi_weight<G>(A, j, g) : __dmul_rn(phi_weight<G>(A, j, g), rw);
            return __dmul_rn(x, (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0);
        };
        double p = 0.0;
        for (int j = lane & 7; j < nfull; j += 8) p = __dadd_rn(p, term(j));
        p = __dadd_rn(p, __shfl_sync(0xffffffffu, p, (lane + 4) & 7));  // lane u: p_u + p_{u+4}
        double acc = 0.0;
        for (int u = 0; u < 4; ++u) acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, p, u));
        for (int j = nfull; j < A.n_phi; ++j) acc = __dadd_rn(acc, term(j));
        sum[g] = G == 2 ? acc * rw : acc;
    }
}

// least delay of a row's patches (infinity: none collides)
__device__ __forceinline__ double first_collision(const double* __restrict__ trow, int n_phi) {
    double least = CUDART_INF;
    for (int j = threadIdx.x & 31; j < n_phi; j += 32) {
        const double t = trow[j];
        if (t > 0.0) least = fmin(least, t);
    }
    for (int o = 16; o > 0; o >>= 1) least = fmin(least, __shfl_xor_sync(0xffffffffu, least, o));
    return least;
}

// NS: steps per lane.  EXACT: every patch and step by pow and exp as the reference forms them, for
// exponents and damping widths whose separated factors could leave the FP64 range (see direct_exact).
template <int G, int NS, bool EXACT>
__global__ void __launch_bounds__(32 * kDirWarps) k_direct_b(DirArgs A) {
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nkb = (A.k1 - A.k0 + 32 * NS - 1) / (32 * NS);
    const size_t wid = (size_t)blockIdx.x * kDirWarps + (threadIdx.x >> 5);
    if (wid >= A.n_fs * A.n_cos * nkb) return;
    const int kb = (int)(wid % nkb);
    const size_t row = wid / nkb;  // (pair, row)
    const int i = (int)(row % A.n_cos);
    const size_t fs = A.fs0 + row / A.n_cos;
    const int slot = (int)(fs % A.n_sel);
    const size_t frame = fs / A.n_sel;
    const double ta = A.in.bub[frame * A.n_tot + A.in.sel[slot]].t;
    const double* trow = A.in.tau + (fs * A.n_cos + i) * A.n_phi;
    const int kbase = A.k0 + kb * 32 * NS;
    const int klast = min(kbase + 32 * NS, A.k1) - 1;
    const double dt_first = A.in.t_arr[kbase] - ta, dt_last = A.in.t_arr[klast] - ta;
    const int cols = A.S * G;
    double* out = A.B + row * cols * A.tp + (kbase - A.k0);
    double dta[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) dta[m] = A.in.t_arr[min(kbase + 32 * m + lane, klast)] - ta;
    const double c = A.in.cos_t[i];
    // row weight, dphi, dcos with its end weight, 1 / (6 pi)
    const double rowf = A.dphi * A.dcos * ((i == 0 || i == A.n_cos - 1) ? 0.5 : 1.0) * (1.0 / (6.0 * CUDART_PI));
    const bool live = dt_last > 0.0;
    double rw[G], quiet[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        rw[g] = row_weight<G>(c, g);
        quiet[g] = 0.0;
    }
    if (live && !(first_collision(trow, A.n_phi) <= dt_first)) quiet_row<G>(A, c, quiet);
    for (int s = 0; s < A.S; ++s) {
        double res[NS][G];
        bool hits[NS];  // some patch has collided by this step
#pragma unroll
        for (int m = 0; m < NS; ++m) hits[m] = false;
#pragma unroll
        for (int m = 0; m < NS; ++m)
#pragma unroll
            for (int g = 0; g < G; ++g) res[m][g] = 0.0;
        if (EXACT && live) {
            for (int j = 0; j < A.n_phi; ++j) {
                const double tj = trow[j];
                const double wj = (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0;
#pragma unroll
                for (int m = 0; m < NS; ++m) {
                    double f = 1.0;
                    if (tj > 0.0 && dta[m] >= tj) {
                        hits[m] = true;
                        const double ratio = tj / dta[m];
                        f = 0.0;
                        for (int q = 0; q < A.M; ++q)
                            f += A.in.coeffs[s * A.M + q] * pow(ratio, A.in.powers[s * A.M + q]);
                        if (A.has_damp) f *= exp(-dta[m] * (1.0 - ratio) / A.damp);
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g) res[m][g] += phi_weight<G>(A, j, g) * f * wj;
                }
            }
        } else if (live) {
            for (int q = 0; q < A.M; ++q) {
                const double p = A.in.powers[s * A.M + q], am = A.in.coeffs[s * A.M + q];
                double P[G], U[G], Pin[NS][G];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    P[g] = U[g] = 0.0;
#pragma unroll
                    for (int m = 0; m < NS; ++m) Pin[m][g] = 0.0;
                }
                for (int j0 = 0; j0 < A.n_phi; j0 += 32) {
                    const int j = j0 + lane;
                    const bool valid = j < A.n_phi;
                    const double tj = valid ? trow[j] : 0.0;
                    const double wj = valid ? ((j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0) : 0.0;
                    const bool col = tj > 0.0 && dt_last >= tj;   // collided at the block's last step
                    const bool pre = tj > 0.0 && dt_first >= tj;  // ... and at its first
                    if (__any_sync(full, pre)) {
#pragma unroll
                        for (int m = 0; m < NS; ++m) hits[m] = true;
                    }
                    double v = 0.0, x[G];
                    if (col) {
                        v = tpow(tj / dt_last, p);
                        if (A.has_damp) v *= exp(-(dt_last - tj) / A.damp);
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        x[g] = valid ? wj * phi_weight<G>(A, j, g) : 0.0;
                        if (pre) P[g] += x[g] * v;
                        if (!col) U[g] += x[g];
                    }
                    for (unsigned h = __ballot_sync(full, col && !pre); h; h &= h - 1) {
                        const int src = __ffs(h) - 1;
                        const double ts = __shfl_sync(full, tj, src), vs = __shfl_sync(full, v, src);
                        bool hit[NS];
#pragma unroll
                        for (int m = 0; m < NS; ++m) {
                            hit[m] = dta[m] >= ts;
                            hits[m] |= hit[m];
                        }
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const double xs = __shfl_sync(full, x[g], src), xv = xs * vs;
#pragma unroll
                            for (int m = 0; m < NS; ++m) {
                                if (hit[m]) Pin[m][g] += xv;
                                else if (q == 0) res[m][g] += xs;
                            }
                        }
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        P[g] += __shfl_xor_sync(full, P[g], o);
                        if (q == 0) U[g] += __shfl_xor_sync(full, U[g], o);
                    }
#pragma unroll
                for (int m = 0; m < NS; ++m) {
                    double cm = 0.0;
                    if (dta[m] > 0.0) {
                        cm = am * tpow(dt_last / dta[m], p);
                        if (A.has_damp) cm *= exp((dt_last - dta[m]) / A.damp);
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const double sum = P[g] + Pin[m][g];
                        if (q == 0) res[m][g] += U[g];
                        // before the first collision there is nothing to scale (cm may be huge there)
                        if (sum != 0.0) res[m][g] += cm * sum;
                    }
                }
            }
        }
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            const int k = kbase + 32 * m + lane;
            if (k - A.k0 >= A.tp) continue;
            const bool on = k < A.k1 && dta[m] > 0.0;
            const double wk = on ? rowf * (dta[m] * (dta[m] * dta[m])) * A.in.cutw[k] * A.dt *
                                       ((k == 0 || k == A.n_t - 1) ? 0.5 : 1.0)
                                 : 0.0;
#pragma unroll
            for (int g = 0; g < G; ++g)
                out[(size_t)(s * G + g) * A.tp + 32 * m + lane] =
                    on ? (hits[m] ? res[m][g] * rw[g] : quiet[g]) * wk : 0.0;
        }
    }
}

// Phase of one argument; BIG: arguments past the table reduction's range (or not finite).
template <bool BIG>
__device__ __forceinline__ void phase_of(const double2* tab, double x, double& s, double& c) {
    if constexpr (BIG)
        sincos(x, &s, &c);
    else
        table_sincos(tab, x, s, c);
}

struct RowSumArgs {
    DirArgs d;
    int per_warp;     // blocks of 32 steps (spectrum) or bubbles (integrand) taken in turn by one warp
    int n_parts;      // partial sums per (pair, column, w) over the whole job
    int part0;        // first part of this launch's steps
    double2* partial; // spectrum: (pairs of the job, n_parts, G, S, W); integrand: (bubble parts, G, S, W, n_t)
};

// NC columns from column c0 = blockIdx.z NC on.
template <int NC, int NW, bool BIG, bool PER_T>
__global__ void __launch_bounds__(32 * kDirWarps) k_direct_a(RowSumArgs R, int G) {
    extern __shared__ double s_c[];  // cos theta of the rows
    __shared__ double2 tab[kPhaseTable];
    const DirArgs& A = R.d;
    if constexpr (!BIG) phase_table_fill(tab);
    for (int q = threadIdx.x; q < A.n_cos; q += blockDim.x) s_c[q] = A.in.cos_t[q];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int w0 = (blockIdx.y * kDirWarps + (threadIdx.x >> 5)) * NW;
    if (w0 >= A.n_w) return;
    const int cols = A.S * G, c0 = blockIdx.z * NC;
    const int nkc = (A.k1 - A.k0 + 31) >> 5;
    double wv[NW];
#pragma unroll
    for (int u = 0; u < NW; ++u) wv[u] = A.in.w[min(w0 + u, A.n_w - 1)];
    double cr[NW][NC], cim[NW][NC];
#pragma unroll
    for (int u = 0; u < NW; ++u)
#pragma unroll
        for (int n = 0; n < NC; ++n) cr[u][n] = cim[u][n] = 0.0;
    // spectrum: blockIdx.x = (pair, group of step blocks); integrand: (bubble group, step block)
    const int n_grp = (nkc + R.per_warp - 1) / R.per_warp;
    size_t f_lo, f_hi;
    int b_lo, b_hi;
    if constexpr (PER_T) {
        f_lo = (size_t)(blockIdx.x / nkc) * R.per_warp;
        f_hi = min(f_lo + R.per_warp, A.n_fs);
        b_lo = blockIdx.x % nkc;
        b_hi = b_lo + 1;
    } else {
        f_lo = blockIdx.x / n_grp;
        f_hi = f_lo + 1;
        b_lo = (int)(blockIdx.x % n_grp) * R.per_warp;
        b_hi = min(b_lo + R.per_warp, nkc);
    }
    for (size_t f = f_lo; f < f_hi; ++f) {
        const size_t fs = A.fs0 + f;
        const D4 xa = A.in.bub[(fs / A.n_sel) * A.n_tot + A.in.sel[fs % A.n_sel]];
        for (int b = b_lo; b < b_hi; ++b) {
            const int k = A.k0 + 32 * b + lane;
            if (!(A.in.t_arr[min(A.k0 + 32 * b + 31, A.k1 - 1)] - xa.t > 0.0)) continue;  // not nucleated yet
            const double t = A.in.t_arr[min(k, A.k1 - 1)];
            const double dta = t - xa.t;
            double ar[NW][NC], ai[NW][NC];
#pragma unroll
            for (int u = 0; u < NW; ++u)
#pragma unroll
                for (int n = 0; n < NC; ++n) ar[u][n] = ai[u][n] = 0.0;
            const size_t rstep = (size_t)cols * A.tp;
            const double* b0 = A.B + f * A.n_cos * rstep + (size_t)c0 * A.tp + (32 * b + lane);
            const double* b1 = b0 + (A.n_cos - 1) * rstep;
            const int half = A.n_cos >> 1;
            for (int i = 0; i < half; ++i, b0 += rstep, b1 -= rstep) {
                double v0[NC], v1[NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    v0[n] = __ldg(b0 + (size_t)n * A.tp);
                    v1[n] = __ldg(b1 + (size_t)n * A.tp);
                }
                const double m0 = -dta * s_c[i], m1 = -dta * s_c[A.n_cos - 1 - i];
#pragma unroll
                for (int u = 0; u < NW; ++u) {
                    const double x0 = __dmul_rn(wv[u], m0), x1 = __dmul_rn(wv[u], m1);
                    double s0, q0, s1, q1;
                    phase_of<BIG>(tab, x0, s0, q0);
                    if constexpr (BIG) {
                        sincos(x1, &s1, &q1);
                    } else {
                        // exact: the (rounded) arguments are opposite to a few ulp
                        const double e = __dadd_rn(x0, x1);
                        q1 = fma(s0, e, q0);
                        s1 = fma(q0, e, -s0);
                    }
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        ar[u][n] = fma(v0[n], q0, fma(v1[n], q1, ar[u][n]));
                        ai[u][n] = fma(v0[n], s0, fma(v1[n], s1, ai[u][n]));
                    }
                }
            }
            if (A.n_cos & 1) {
                const double m0 = -dta * s_c[half];
#pragma unroll
                for (int u = 0; u < NW; ++u) {
                    double s0, q0;
                    phase_of<BIG>(tab, __dmul_rn(wv[u], m0), s0, q0);
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        const double v = __ldg(b0 + (size_t)n * A.tp);
                        ar[u][n] = fma(v, q0, ar[u][n]);
                        ai[u][n] = fma(v, s0, ai[u][n]);
                    }
                }
            }
            const double tz = t - xa.z;
#pragma unroll
            for (int u = 0; u < NW; ++u) {
                double s0, q0;
                phase_of<BIG>(tab, __dmul_rn(wv[u], tz), s0, q0);
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    cr[u][n] += ar[u][n] * q0 - ai[u][n] * s0;
                    cim[u][n] += ar[u][n] * s0 + ai[u][n] * q0;
                }
            }
        }
    }
    const size_t W = A.n_w;
    if constexpr (PER_T) {
        const int k = A.k0 + 32 * b_lo + lane;
        if (k >= A.k1) return;
        double2* o = R.partial + (size_t)(blockIdx.x / nkc) * cols * W * A.n_t;
#pragma unroll
        for (int u = 0; u < NW; ++u)
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                const int col = c0 + n, g = col % G, s = col / G;
                if (w0 + u < A.n_w)
                    o[(((size_t)g * A.S + s) * W + w0 + u) * A.n_t + k] = make_double2(cr[u][n], cim[u][n]);
            }
    } else {
        double2* o = R.partial + ((A.fs0 + f_lo) * R.n_parts + R.part0 + blockIdx.x % n_grp) * cols * W;
#pragma unroll
        for (int u = 0; u < NW; ++u)
#pragma unroll
            for (int n = 0; n < NC; ++n) {
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    cr[u][n] += __shfl_xor_sync(0xffffffffu, cr[u][n], off);
                    cim[u][n] += __shfl_xor_sync(0xffffffffu, cim[u][n], off);
                }
                const int col = c0 + n, g = col % G, s = col / G;
                if (lane == 0 && w0 + u < A.n_w)
                    o[((size_t)g * A.S + s) * W + w0 + u] = make_double2(cr[u][n], cim[u][n]);
            }
    }
}

// out[k][q] = sum over the n parts of partial[k][part][q] (+ out[k][q] with ADD), in an order that
// depends on n only: 8 strided lanes of the block's rows, then the lanes in order.
template <bool ADD>
__global__ void k_direct_reduce(const double2* __restrict__ partial, size_t n, size_t per, double2* __restrict__ out) {
    __shared__ double2 red[8][32];
    const size_t q = (size_t)blockIdx.x * 32 + threadIdx.x;
    const double2* p = partial + (size_t)blockIdx.y * n * per;
    double2 acc = make_double2(0.0, 0.0);
    if (q < per) {
#pragma unroll 4
        for (size_t a = threadIdx.y; a < n; a += 8) {
            const double2 v = p[a * per + q];
            acc.x += v.x;
            acc.y += v.y;
        }
    }
    red[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y || q >= per) return;
    double2& o = out[(size_t)blockIdx.y * per + q];
    double2 sum = ADD ? o : make_double2(0.0, 0.0);
    for (int y = 0; y < 8; ++y) {
        sum.x += red[y][threadIdx.x].x;
        sum.y += red[y][threadIdx.x].y;
    }
    o = sum;
}

// Separated factors need (tau / dt_last)^p, (dt_last / dt)^p and the damping exponentials inside the
// FP64 range: dt_last / dt is at most 1e17 or so (a step one ulp after the nucleation), so |p| <= 16
// is safe, and the damping exponents stay below 300.  Everything else takes the exact form.
bool direct_exact(const SpectrumJob& job) {
    for (size_t q = 0; q < job.n_sets * job.n_terms; ++q)
        if (!(std::fabs(job.powers[q]) <= 16.0) || !std::isfinite(job.coeffs[q])) return true;
    if (job.has_damping) {
        const double span = job.t_arr[job.n_t - 1] - job.t_arr[0];
        const double within = std::min(span, 128.0 * std::fabs(job.dt));
        if (!(job.damping > 0.0) || !(within / job.damping < 300.0)) return true;
    }
    return false;
}

// Arguments the table reduction covers: |w| times the largest time or position difference.
bool direct_big(const SpectrumJob& job) {
    double wmax = 0.0, xmax = 0.0;
    for (size_t q = 0; q < job.n_w; ++q) {
        if (!std::isfinite(job.w[q])) return true;
        wmax = std::max(wmax, std::fabs(job.w[q]));
    }
    double tmax = std::max(std::fabs(job.t_arr[0]), std::fabs(job.t_arr[job.n_t - 1]));
    for (size_t q = 0; q < job.n_sel; ++q) {
        const double* b = job.bubbles + 4 * (size_t)job.sel[q];
        // |z| of a rotated frame is at most the length of the position
        const double r = std::sqrt(b[1] * b[1] + b[2] * b[2] + b[3] * b[3]);
        if (!std::isfinite(b[0]) || !std::isfinite(r)) return true;
        xmax = std::max(xmax, std::max(std::fabs(b[0]), r));
    }
    return !(wmax * (tmax + xmax) < kPhaseMax);
}

struct DirectPlan {
    int G;
    int nw, nc;          // frequencies per warp, columns per pass
    int nkc;             // blocks of 32 steps
    int per_warp;        // step blocks per warp
    int n_parts;
};

// Columns per pass: all six of the tensor form, or up to four sets' two; frequencies per warp: as
// many as keep the accumulators (4 NC NW doubles) in registers.  A warp takes several step blocks
// once there are enough warps (about 16 per SM sub-partition) to fill the chip.
DirectPlan direct_plan(const Device* dev, const SpectrumJob& job, size_t pairs) {
    DirectPlan p;
    p.G = job.tensor ? 6 : 2;
    const int S = (int)job.n_sets;
    p.nc = job.tensor ? 6 : S % 3 == 0 ? 6 : S % 2 == 0 ? 4 : 2;
    p.nw = p.nc == 2 ? 4 : 2;
    p.nkc = (int)((job.n_t + 31) / 32);
    const size_t warps = pairs * ((job.n_w + p.nw - 1) / p.nw) * (S * p.G / p.nc) * p.nkc;
    const size_t want = (size_t)dev->n_sm * 4 * 16;
    p.per_warp = (int)std::max<size_t>(1, std::min<size_t>(p.nkc, warps / want));
    p.n_parts = (p.nkc + p.per_warp - 1) / p.per_warp;
    return p;
}

DirArgs direct_args(const SpectrumJob& job, const DirectInputs& in) {
    DirArgs A;
    A.in = in;
    A.n_tot = job.n_tot;
    A.n_sel = (int)job.n_sel;
    A.n_cos = (int)job.n_cos;
    A.n_phi = (int)job.n_phi;
    A.n_t = (int)job.n_t;
    A.n_w = (int)job.n_w;
    A.S = (int)job.n_sets;
    A.M = (int)job.n_terms;
    A.has_damp = job.has_damping ? 1 : 0;
    A.damp = job.damping;
    A.dphi = 2.0 * M_PI / (double)job.n_phi;
    A.dcos = 2.0 / (double)(job.n_cos - 1);
    A.dt = job.dt;
    return A;
}

template <int G, int NS>
void launch_b(const DirArgs& A, bool exact, cudaStream_t st) {
    const size_t nkb = (A.k1 - A.k0 + 32 * NS - 1) / (32 * NS);
    const size_t blocks = (A.n_fs * A.n_cos * nkb + kDirWarps - 1) / kDirWarps;
    if (blocks > 0x7fffffffULL) throw Error{"direct kernel: too many (bubble, row, step) blocks for one launch"};
    if (exact)
        k_direct_b<G, NS, true><<<(unsigned)blocks, 32 * kDirWarps, 0, st>>>(A);
    else
        k_direct_b<G, NS, false><<<(unsigned)blocks, 32 * kDirWarps, 0, st>>>(A);
    CUDA_OK(cudaGetLastError());
}

template <int NC, int NW, bool PER_T>
void launch_a(const RowSumArgs& R, int G, size_t gx, bool big, cudaStream_t st) {
    if (gx > 0x7fffffffULL) throw Error{"direct kernel: too many (bubble, step) blocks for one launch"};
    const size_t gy = (R.d.n_w + NW * kDirWarps - 1) / (NW * kDirWarps);
    if (gy > 65535) throw Error{"direct kernel: too many frequencies for one launch"};
    const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)(R.d.S * G / NC));
    const size_t smem = (size_t)R.d.n_cos * sizeof(double);
    if (big)
        k_direct_a<NC, NW, true, PER_T><<<grid, 32 * kDirWarps, smem, st>>>(R, G);
    else
        k_direct_a<NC, NW, false, PER_T><<<grid, 32 * kDirWarps, smem, st>>>(R, G);
    CUDA_OK(cudaGetLastError());
}

template <bool PER_T>
void dispatch_a(const RowSumArgs& R, const DirectPlan& P, size_t gx, bool big, cudaStream_t st) {
    switch (P.nc) {
        case 2: return launch_a<2, 4, PER_T>(R, P.G, gx, big, st);
        case 4: return launch_a<4, 2, PER_T>(R, P.G, gx, big, st);
        default: return launch_a<6, 2, PER_T>(R, P.G, gx, big, st);
    }
}

constexpr size_t kDirectBufferBytes = (size_t)1 << 30;  // B of one launch

}  // namespace

size_t direct_bytes_per_frame(const Device* dev, const SpectrumJob& job) {
    const DirectPlan P = direct_plan(dev, job, job.n_sel);
    return job.n_sel * P.n_parts * P.G * job.n_sets * job.n_w * sizeof(double2);
}

uint64_t launch_direct(Device* dev, const SpectrumJob& job, const DirectInputs& in, size_t kn, double2* out) {
    const size_t pairs = kn * job.n_sel;
    const DirectPlan P = direct_plan(dev, job, pairs);
    const size_t cols = (size_t)P.G * job.n_sets, per = cols * job.n_w;
    const bool exact = direct_exact(job), big = direct_big(job);
    dev->partial.ensure(pairs * P.n_parts * per * sizeof(double2));
    // B holds a range of pairs over a range of steps (whole groups of per_warp step blocks)
    const size_t group = (size_t)P.per_warp * 32;
    const size_t col_bytes = job.n_cos * cols * sizeof(double);
    size_t steps = std::min<size_t>((size_t)P.n_parts, std::max<size_t>(1, kDirectBufferBytes / (col_bytes * group))) * group;
    const size_t n_fs = std::min(pairs, std::max<size_t>(1, kDirectBufferBytes / (col_bytes * std::min(steps, (size_t)P.nkc * 32))));
    DirArgs A = direct_args(job, in);
    uint64_t launches = 0;
    for (size_t k0 = 0; k0 < job.n_t; k0 += steps) {
        A.k0 = (int)k0;
        A.k1 = (int)std::min(job.n_t, k0 + steps);
        A.tp = (A.k1 - A.k0 + 31) & ~31;
        dev->beta.ensure(n_fs * job.n_cos * cols * A.tp * sizeof(double));
        A.B = (double*)dev->beta.p;
        for (size_t f0 = 0; f0 < pairs; f0 += n_fs) {
            A.fs0 = f0;
            A.n_fs = std::min(n_fs, pairs - f0);
            if (job.tensor)
                launch_b<6, 2>(A, exact, dev->stream);
            else
                launch_b<2, 4>(A, exact, dev->stream);
            const RowSumArgs R{A, P.per_warp, P.n_parts, (int)(k0 / group), (double2*)dev->partial.p};
            const size_t groups = ((A.k1 - A.k0 + 31) / 32 + P.per_warp - 1) / P.per_warp;
            dispatch_a<false>(R, P, A.n_fs * groups, big, dev->stream);
            launches += 2;
        }
    }
    const dim3 gr((unsigned)((per + 31) / 32), (unsigned)kn);
    k_direct_reduce<false><<<gr, dim3(32, 8), 0, dev->stream>>>((const double2*)dev->partial.p, job.n_sel * P.n_parts,
                                                                per, out);
    CUDA_OK(cudaGetLastError());
    return launches + 1;
}

uint64_t launch_direct_integrand(Device* dev, const SpectrumJob& job, const DirectInputs& in, double2* out) {
    const size_t pairs = job.n_sel;
    DirectPlan P = direct_plan(dev, job, pairs);
    const size_t cols = (size_t)P.G * job.n_sets, per = cols * job.n_w * job.n_t;
    const bool exact = direct_exact(job), big = direct_big(job);
    // B holds a range of bubbles over all steps, or one bubble over a range of steps
    const size_t step_bytes = job.n_cos * cols * 32 * sizeof(double);
    const size_t nkc = std::min<size_t>(P.nkc, std::max<size_t>(1, kDirectBufferBytes / step_bytes));
    const size_t n_fs = std::min(pairs, std::max<size_t>(1, kDirectBufferBytes / (step_bytes * nkc)));
    // bubbles per warp: few enough for the chip to be full, as many as keep the partial outputs small
    const size_t warps = ((job.n_w + P.nw - 1) / P.nw) * (cols / P.nc) * P.nkc;
    const size_t want = (size_t)dev->n_sm * 4 * 8;
    size_t groups = std::min(n_fs, std::max<size_t>(1, (want + warps - 1) / warps));
    groups = std::min(groups, std::max<size_t>(1, kDirectBufferBytes / (per * sizeof(double2))));
    P.per_warp = (int)((n_fs + groups - 1) / groups);
    dev->partial.ensure(((n_fs + P.per_warp - 1) / P.per_warp) * per * sizeof(double2));
    dev->beta.ensure(n_fs * nkc * step_bytes);
    const size_t gx = (per + 31) / 32;
    if (gx > 0x7fffffffULL) throw Error{"direct kernel: integrand too large for one launch"};
    DirArgs A = direct_args(job, in);
    A.B = (double*)dev->beta.p;
    uint64_t launches = 0;
    for (size_t f0 = 0; f0 < pairs; f0 += n_fs) {
        A.fs0 = f0;
        A.n_fs = std::min(n_fs, pairs - f0);
        const size_t parts = (A.n_fs + P.per_warp - 1) / P.per_warp;
        for (size_t k0 = 0; k0 < job.n_t; k0 += 32 * nkc) {
            A.k0 = (int)k0;
            A.k1 = (int)std::min(job.n_t, k0 + 32 * nkc);
            A.tp = (A.k1 - A.k0 + 31) & ~31;
            if (job.tensor)
                launch_b<6, 2>(A, exact, dev->stream);
            else
                launch_b<2, 4>(A, exact, dev->stream);
            const RowSumArgs R{A, P.per_warp, 0, 0, (double2*)dev->partial.p};
            dispatch_a<true>(R, P, parts * (size_t)(A.tp / 32), big, dev->stream);
            launches += 2;
        }
        const dim3 gr((unsigned)gx, 1), block(32, 8);
        if (f0 == 0)
            k_direct_reduce<false><<<gr, block, 0, dev->stream>>>((const double2*)dev->partial.p, parts, per, out);
        else
            k_direct_reduce<true><<<gr, block, 0, dev->stream>>>((const double2*)dev->partial.p, parts, per, out);
        CUDA_OK(cudaGetLastError());
        ++launches;
    }
    return launches;
}

}  // namespace bgw
