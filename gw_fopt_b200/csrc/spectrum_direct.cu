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
//               formed exactly, and a first-order correction in e.  |e| is below 10 x 2^-53 |w| dt (5 for
//               the roundings of the two c, 2 each for -dt c and its product with w), so the e^2 / 2 left
//               out is below 2^-56 for the |w| dt < 4e6 that this form is used for; beyond, the library's
//               sincos for both.
//
// What bounds it: FP64 issue in k_direct_a (about 14 operations and 4 per column for each phase);
// k_direct_b is a few per cent.  The single kernel this replaces (one block per bubble, pow() for
// every patch and step, a barrier per step) took 53.6 ms for 5 bubbles x 50 x 100 patches x 800 steps
// x 120 w and 38.2 ms for 4 frames of 64 bubbles x 64 x 64 x 256 x 64 w with 3 sets; these two take
// 0.08 ms and 1.01 ms (k_direct_b 0.27, k_direct_a 0.75: FP64 pipe half busy, 0.34 ms of FP64 work).

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
    double* steps;    // (n_sel, 1 + S M, tf) step factors, see k_direct_steps
    int tf;           // row length of the step factors (multiple of kStepBlock)
};

constexpr int kStepsPerLane = 4;
constexpr int kStepBlock = 32 * kStepsPerLane;  // steps of a k_direct_b warp

// Step factors of the separable scaling, frame and row independent, for blocks of kStepBlock steps with
// dt_ref = dt at the block's last step: row 0 is dt^3 times the step weight (cutoff, dt, trapezoid
// end), row 1 + q the factor a_q (dt_ref / dt)^{p_q} e^{(dt_ref - dt) / width}.  Zero where dt <= 0.
__global__ void k_direct_steps(DirArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, slot = blockIdx.y + blockIdx.z * 65535;
    if (k >= A.tf || slot >= A.n_sel) return;
    const double ta = A.in.bub[A.in.sel[slot]].t;
    const int klast = min(k | (kStepBlock - 1), A.n_t - 1);
    const double dt_ref = A.in.t_arr[klast] - ta;
    const double dt = k < A.n_t ? A.in.t_arr[k] - ta : 0.0;
    const bool on = dt > 0.0;
    const int SM = A.S * A.M;
    double* o = A.steps + (size_t)slot * (1 + SM) * A.tf + k;
    const double u = (k == 0 || k == A.n_t - 1) ? 0.5 : 1.0;
    o[0] = on ? dt * (dt * dt) * A.in.cutw[k] * A.dt * u : 0.0;
    const double e = on && A.has_damp ? exp((dt_ref - dt) / A.damp) : 1.0;
    for (int q = 0; q < SM; ++q)
        o[(size_t)(1 + q) * A.tf] = on ? A.in.coeffs[q] * tpow(dt_ref / dt, A.in.powers[q]) * e : 0.0;
}

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

// The phi sums of one (pair, row) over a block of kStepBlock steps; lane l holds steps 4 l .. 4 l + 3 of it.
// EXACT: every patch and step by pow and exp as the reference forms them, for exponents and damping
// widths whose separated factors could leave the FP64 range (see direct_exact).
template <int G, bool EXACT>
__global__ void __launch_bounds__(32 * kDirWarps) k_direct_b(DirArgs A) {
    constexpr unsigned full = 0xffffffffu;
    constexpr int NS = kStepsPerLane;
    // per warp: the block's collisions added up by step, one row per weight
    __shared__ __align__(16) double s_acc[kDirWarps][G][kStepBlock];
    const int lane = threadIdx.x & 31;
    double(*acc)[kStepBlock] = s_acc[threadIdx.x >> 5];
    const int nkb = (A.k1 - A.k0 + kStepBlock - 1) / kStepBlock;
    const size_t wid = (size_t)blockIdx.x * kDirWarps + (threadIdx.x >> 5);
    if (wid >= A.n_fs * A.n_cos * nkb) return;
    const int kb = (int)(wid % nkb);
    const size_t row = wid / nkb;  // (pair, row)
    const int i = (int)(row % A.n_cos);
    const size_t fs = A.fs0 + row / A.n_cos;
    const int slot = (int)(fs % A.n_sel);
    const double ta = A.in.bub[(fs / A.n_sel) * A.n_tot + A.in.sel[slot]].t;
    const double* trow = A.in.tau + (fs * A.n_cos + i) * A.n_phi;
    const int kbase = A.k0 + kb * kStepBlock;
    const int klast = min(kbase + kStepBlock, A.k1) - 1;
    const double dt_first = A.in.t_arr[kbase] - ta, dt_last = A.in.t_arr[klast] - ta;
    const int SM = A.S * A.M;
    const double* steps = A.steps + (size_t)slot * (1 + SM) * A.tf + kbase + NS * lane;
    const bool live = dt_last > 0.0;
    double* out = A.B + row * (A.S * G) * A.tp + (kbase - A.k0) + NS * lane;
    // rows of B hold whole groups of 32 steps: a lane's four steps are all in or all out
    const bool store = kbase - A.k0 + NS * lane < A.tp;
    if (!live) {
        if (store)
            for (int col = 0; col < A.S * G; ++col)
#pragma unroll
                for (int m = 0; m < NS; m += 2)
                    *reinterpret_cast<double2*>(out + (size_t)col * A.tp + m) = make_double2(0.0, 0.0);
        return;
    }
    const double c = A.in.cos_t[i];
    // dphi, dcos with its end weight, 1 / (6 pi)
    const double rowf = A.dphi * A.dcos * ((i == 0 || i == A.n_cos - 1) ? 0.5 : 1.0) * (1.0 / (6.0 * CUDART_PI));
    double rw[G], quiet[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        rw[g] = row_weight<G>(c, g);
        quiet[g] = 0.0;
    }
    const double least = first_collision(trow, A.n_phi);
    if (!(least <= dt_first)) quiet_row<G>(A, c, quiet);
    double wk[NS];
    bool hits[NS];  // some patch has collided by this step
#pragma unroll
    for (int m = 0; m < NS; ++m) {
        const int k = kbase + NS * lane + m;
        wk[m] = k < A.k1 ? rowf * steps[m] : 0.0;
        hits[m] = least <= A.in.t_arr[min(k, klast)] - ta;
    }
    auto put = [&](int s, const double (&res)[NS][G]) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            double v[NS];
#pragma unroll
            for (int m = 0; m < NS; ++m) v[m] = wk[m] != 0.0 ? (hits[m] ? res[m][g] * rw[g] : quiet[g]) * wk[m] : 0.0;
            if (store) {
                double* o = out + (size_t)(s * G + g) * A.tp;
                *reinterpret_cast<double2*>(o) = make_double2(v[0], v[1]);
                *reinterpret_cast<double2*>(o + 2) = make_double2(v[2], v[3]);
            }
        }
    };
    if constexpr (EXACT) {
        double dta[NS];
#pragma unroll
        for (int m = 0; m < NS; ++m) dta[m] = A.in.t_arr[min(kbase + NS * lane + m, klast)] - ta;
        for (int s = 0; s < A.S; ++s) {
            double res[NS][G];
#pragma unroll
            for (int m = 0; m < NS; ++m)
#pragma unroll
                for (int g = 0; g < G; ++g) res[m][g] = 0.0;
            for (int j = 0; j < A.n_phi; ++j) {
                const double tj = trow[j];
                const double wj = (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0;
#pragma unroll
                for (int m = 0; m < NS; ++m) {
                    double f = 1.0;
                    if (tj > 0.0 && dta[m] >= tj) {
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
            put(s, res);
        }
    } else {
        const double inv_dt = 1.0 / A.dt;  // the estimate below is only a starting point
        // Adds the block's patches up: `base` (all lanes) the sum over the patches of state `pre` at the
        // block's first step (collided: P) or uncollided at its last (U), acc the patches colliding in
        // between, at their own step. 
        auto sweep = [&](bool collided, double p, double (&base)[G]) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                base[g] = 0.0;
#pragma unroll
                for (int m = 0; m < NS; ++m) acc[g][lane + 32 * m] = 0.0;
            }
            __syncwarp();
            for (int j0 = 0; j0 < A.n_phi; j0 += 32) {
                const int j = j0 + lane;
                const bool valid = j < A.n_phi;
                const double tj = valid ? trow[j] : 0.0;
                const bool col = tj > 0.0 && dt_last >= tj;   // collided at the block's last step
                const bool pre = tj > 0.0 && dt_first >= tj;  // ... and at its first
                const bool in = col && !pre;
                double v = valid ? ((j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0) : 0.0;
                if (collided) {
                    if (col) {
                        v *= tpow(tj / dt_last, p);
                        if (A.has_damp) v *= exp(-(dt_last - tj) / A.damp);
                    }
                }
                double x[G];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    x[g] = valid ? v * phi_weight<G>(A, j, g) : 0.0;
                    if (collided ? pre : !col) base[g] += x[g];
                }
                if (!__any_sync(full, in)) continue;
                int kj = 32 * NS + lane;  // position in the block of the first collided step
                if (in) {
                    const double est = ceil((ta + tj - A.in.t_arr[0]) * inv_dt);
                    int k = max(kbase, min(klast, (int)fmin(fmax(est, 0.0), 2e9)));
                    while (k > kbase && A.in.t_arr[k - 1] - ta >= tj) --k;
                    while (!(A.in.t_arr[k] - ta >= tj)) ++k;  // holds at klast at the latest
                    kj = k - kbase;
                }
                // patches of one step are added one after another, in lane order
                const unsigned same = __match_any_sync(full, kj);
                int rank = in ? __popc(same & ((1u << lane) - 1u)) : 32;
                for (int r = 0; __any_sync(full, rank >= r && rank < 32); ++r) {
                    if (rank == r) {
#pragma unroll
                        for (int g = 0; g < G; ++g) acc[g][kj] += x[g];
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int g = 0; g < G; ++g) base[g] += __shfl_xor_sync(full, base[g], o);
        };
        // uncollided sums: base plus the patches whose step comes later (a sum of what remains)
        double U[NS][G], base[G];
        sweep(false, 0.0, base);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            double v[NS], tot = 0.0;
#pragma unroll
            for (int m = 0; m < NS; ++m) v[m] = acc[g][NS * lane + m];
#pragma unroll
            for (int m = NS - 1; m >= 0; --m) {
                U[m][g] = tot;  // later steps of this lane
                tot += v[m];
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_down_sync(full, tot, o);
                if (lane + o < 32) tot += t;
            }
            double later = __shfl_down_sync(full, tot, 1);
            if (lane == 31) later = 0.0;
#pragma unroll
            for (int m = 0; m < NS; ++m) U[m][g] = base[g] + (later + U[m][g]);
        }
        __syncwarp();
        for (int s = 0; s < A.S; ++s) {
            double res[NS][G];
#pragma unroll
            for (int m = 0; m < NS; ++m)
#pragma unroll
                for (int g = 0; g < G; ++g) res[m][g] = U[m][g];
            for (int q = 0; q < A.M; ++q) {
                sweep(true, A.in.powers[s * A.M + q], base);
                double cm[NS];
#pragma unroll
                for (int m = 0; m < NS; ++m) cm[m] = steps[(size_t)(1 + s * A.M + q) * A.tf + m];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    double v[NS], tot = 0.0;
#pragma unroll
                    for (int m = 0; m < NS; ++m) {
                        tot += acc[g][NS * lane + m];
                        v[m] = tot;
                    }
                    double run = tot;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const double t = __shfl_up_sync(full, run, o);
                        if (lane >= o) run += t;
                    }
                    double before = __shfl_up_sync(full, run, 1);
                    if (lane == 0) before = 0.0;
                    // with nothing collided there is nothing to scale (cm may be huge there)
#pragma unroll
                    for (int m = 0; m < NS; ++m)
                        if (hits[m]) res[m][g] += cm[m] * (base[g] + (before + v[m]));
                }
                __syncwarp();
            }
            put(s, res);
        }
    }
}

constexpr double kTwinMax = 4.0e6;  // largest argument of the paired rows
static_assert(kTwinMax <= kPhaseMax, "the table's own range");

// Phase of one argument; BIG: arguments past kTwinMax (or not finite).
template <bool BIG>
__device__ __forceinline__ void phase_of(const double2* tab, double x, double& s, double& c) {
    if constexpr (BIG)
        sincos(x, &s, &c);
    else
        table_sincos(tab, x, s, c);
}

struct RowSumArgs {
    DirArgs d;
    int per_warp;     // spectrum: blocks of 32 steps taken in turn by one warp; integrand: bubbles of a part
    int n_parts;      // spectrum: blocks of 32 steps of the job
    int part0;        // spectrum: the first of this launch
    double2* partial; // spectrum: (pairs of the launch, n_parts, G, S, W); integrand: (bubble parts, G, S, W, n_t)
};

__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// Sums of N values over the 32 lanes, one result per lane: at each of the five exchanges a lane keeps
// half of its values and adds the other lane's (24 exchanges for 24 values instead of 120).
template <int N>
__device__ __forceinline__ double lane_sums(double (&v)[N]) {
    const int lane = threadIdx.x & 31;
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n == 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            continue;
        }
        const int half = (n + 1) / 2;
#pragma unroll
        for (int q = 0; q < N; ++q) {
            if (q >= half) break;
            const double up = q + half < n ? v[q + half] : 0.0;
            const bool upper = lane & o;
            const double got = __shfl_xor_sync(0xffffffffu, upper ? v[q] : up, o);
            v[q] = (upper ? up : v[q]) + got;
        }
        n = half;
    }
    return v[0];
}
// The index of the value that lane_sums leaves in this lane; -1: a copy or nothing.
template <int N>
__device__ __forceinline__ int lane_value(int lane) {
    int n = N, own = N, e = 0;  // values per lane (padded), this lane's own, the first of them
    for (int o = 16; o > 0; o >>= 1) {
        const bool upper = lane & o;
        if (n == 1) {
            if (upper) return -1;
            continue;
        }
        const int half = (n + 1) / 2;
        e += upper ? half : 0;
        own = upper ? own - half : min(own, half);
        if (own <= 0) return -1;
        n = half;
    }
    return e;
}

// Row pairs of one shared-memory stage: 8 KB with two columns, 12 KB with six.
template <int NC>
__host__ __device__ constexpr int stage_pairs() {
    return NC <= 2 ? 8 : 4;
}
constexpr int kRowStages = 3;

// NC columns from column c0 on, NW frequencies per warp, lane = step.  The block's warps share B: row
// pairs (i, n_cos - 1 - i) of the NC columns and 32 steps arrive in shared memory by asynchronous
// copies, three stages deep (from L1 and L2 directly the loads' latency was 70 % of the time: 2.09 ms
// against 0.34 ms of FP64 work for 4 frames of 64 bubbles, 64 rows, 256 steps, 64 w, 6 columns).
// Two blocks per SM for the spectrum (the integrand's accumulators take what registers they need).
template <int NC, int NW, bool BIG, bool PER_T>
__global__ void __launch_bounds__(32 * kDirWarps, PER_T ? 0 : 2) k_direct_a(RowSumArgs R, int G, int w_tiles) {
    constexpr int RP = stage_pairs<NC>();
    constexpr int kStageDoubles = RP * 2 * NC * 32;
    extern __shared__ __align__(16) double s_dyn[];
    double* s_b = s_dyn;                                 // [kRowStages][pair][2][NC][32]
    double* s_c = s_dyn + kRowStages * kStageDoubles;    // cos theta of the rows
    __shared__ double2 tab[kPhaseTable];
    const DirArgs& A = R.d;
    if constexpr (!BIG) phase_table_fill(tab);
    for (int q = threadIdx.x; q < A.n_cos; q += blockDim.x) s_c[q] = A.in.cos_t[q];
    const int lane = threadIdx.x & 31;
    // blocks of the same bubble and steps follow one another: they read the same B
    const int w_tile = blockIdx.x % w_tiles;
    const int unit_block = blockIdx.x / w_tiles;
    const int w0 = (w_tile * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * NW;
    const int cols = A.S * G, c0 = blockIdx.y * NC;
    const int nkc = (A.k1 - A.k0 + 31) >> 5;
    double wv[NW];
#pragma unroll
    for (int u = 0; u < NW; ++u) wv[u] = A.in.w[min(w0 + u, A.n_w - 1)];
    // The integrand sums over a part's bubbles per lane; the spectrum adds each unit up over the warp's lanes
    // (steps) at once and stores it, one value per lane (the register budget of two blocks per SM).  What is
    // added to what depends on neither the launch's pairs and steps nor the units of a warp, so a frame's
    // spectrum has the same bits alone and among others, whatever the scratch memory.
    constexpr int NV = 2 * NW * NC;
    double c_sum[PER_T ? NV : 1];
#pragma unroll
    for (int v = 0; v < (PER_T ? NV : 1); ++v) c_sum[v] = 0.0;
    const size_t W = A.n_w;
    auto place = [&](int e) {  // (G, S, W) index of value e / 2
        const int u = e / (2 * NC), col = c0 + (e / 2) % NC;
        return ((size_t)(col % G) * A.S + col / G) * W + w0 + u;
    };
    // units taken in turn.  Spectrum: step blocks [lo, hi) of one pair; integrand: pairs [lo, hi) at one step block
    const int n_grp = (nkc + R.per_warp - 1) / R.per_warp;
    size_t lo, hi, fixed;
    double2* o_part = R.partial;  // integrand: the part's array
    double* o_unit = nullptr;     // spectrum: where this lane's value of unit lo goes (null: it holds none)
    const size_t o_step = 2 * (size_t)cols * W;
    auto bubble = [&](size_t f) {
        const size_t fs = A.fs0 + f;
        return A.in.bub[(fs / A.n_sel) * A.n_tot + A.in.sel[fs % A.n_sel]];
    };
    D4 xa = D4{0.0, 0.0, 0.0, 0.0};
    double t = 0.0, dta = 0.0;
    if constexpr (PER_T) {
        fixed = unit_block % nkc;
        // this launch's bubbles of the part
        const size_t part = A.fs0 / R.per_warp + unit_block / nkc;
        lo = max(part * R.per_warp, A.fs0) - A.fs0;
        hi = min((part + 1) * R.per_warp, A.fs0 + A.n_fs) - A.fs0;
        o_part += part * cols * W * A.n_t + A.k0 + 32 * fixed + lane;
        if (lo + A.fs0 > part * R.per_warp && A.k0 + 32 * (int)fixed + lane < A.k1) {
            // the part was begun by an earlier launch
#pragma unroll
            for (int e = 0; e < NV; e += 2)
                if (w0 + e / (2 * NC) < A.n_w) {
                    const double2 v = o_part[place(e) * A.n_t];
                    c_sum[e] = v.x;
                    c_sum[e + 1] = v.y;
                }
        }
    } else {
        fixed = unit_block / n_grp;
        lo = (size_t)(unit_block % n_grp) * R.per_warp;
        hi = min(lo + R.per_warp, (size_t)nkc);
        const int e = lane_value<NV>(lane);
        if (e >= 0 && w0 + e / (2 * NC) < A.n_w)
            o_unit = reinterpret_cast<double*>(R.partial) + (fixed * R.n_parts + R.part0 + lo) * o_step + 2 * place(e) + (e & 1);
        // step blocks before the bubble nucleates hold nothing
        xa = bubble(fixed);
        for (; lo < hi && !(A.in.t_arr[min(A.k0 + 32 * (int)lo + 31, A.k1 - 1)] - xa.t > 0.0); ++lo)
            if (o_unit) {
                *o_unit = 0.0;
                o_unit += o_step;
            }
    }
    const size_t rstep = (size_t)cols * A.tp;
    const int n_pairs = (A.n_cos + 1) >> 1;
    const int per_unit = (n_pairs + RP - 1) / RP;
    const size_t n_stages = (hi - lo) * per_unit;
    auto load = [&](size_t q) {
        if (q < n_stages) {
            const size_t unit = lo + q / per_unit;
            const int p0 = (int)(q % per_unit) * RP;
            const size_t f = PER_T ? unit : fixed, b = PER_T ? fixed : unit;
            const double* src = A.B + f * A.n_cos * rstep + (size_t)c0 * A.tp + 32 * b;
            double* dst = s_b + (q % kRowStages) * kStageDoubles;
            for (int e = threadIdx.x; e < RP * 2 * NC * 16; e += blockDim.x) {
                const int line = e >> 4, at = (e & 15) * 2;  // line: (pair, side, column) of 32 steps
                const int n = line % NC, side = (line / NC) & 1, p = p0 + line / (2 * NC);
                if (p >= n_pairs) break;
                const int i = side ? A.n_cos - 1 - p : p;
                copy16_async(dst + line * 32 + at, src + i * rstep + (size_t)n * A.tp + at);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int q = 0; q < kRowStages - 1; ++q) load(q);
    double ar[NW][NC], ai[NW][NC];
    size_t unit = lo;
    int st = 0;  // stage within the unit
    for (size_t q = 0; q < n_stages; ++q) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRowStages - 2) : "memory");
        __syncthreads();  // stage q has landed for every thread, stage q - 1 is free
        load(q + kRowStages - 1);
        if (st == 0) {
            if constexpr (PER_T) xa = bubble(unit);
            t = A.in.t_arr[min(A.k0 + 32 * (int)(PER_T ? fixed : unit) + lane, A.k1 - 1)];
            dta = t - xa.t;
#pragma unroll
            for (int u = 0; u < NW; ++u)
#pragma unroll
                for (int n = 0; n < NC; ++n) ar[u][n] = ai[u][n] = 0.0;
        }
        const double* tile = s_b + (q % kRowStages) * kStageDoubles + lane;
        const int p1 = min(n_pairs, (st + 1) * RP);
        for (int p = st * RP; p < p1; ++p, tile += 2 * NC * 32) {
            const bool twin = p != A.n_cos - 1 - p;  // the middle row of an odd number stands alone
            double v0[NC], v1[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                v0[n] = tile[n * 32];
                v1[n] = twin ? tile[(NC + n) * 32] : 0.0;
            }
            const double m0 = -dta * s_c[p], m1 = -dta * s_c[A.n_cos - 1 - p];
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
        if (++st < per_unit) continue;
        st = 0;
        ++unit;
        const double tz = t - xa.z;
        double v[NV];
#pragma unroll
        for (int u = 0; u < NW; ++u) {
            double s0, q0;
            phase_of<BIG>(tab, __dmul_rn(wv[u], tz), s0, q0);
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                v[2 * (u * NC + n)] = ar[u][n] * q0 - ai[u][n] * s0;
                v[2 * (u * NC + n) + 1] = ar[u][n] * s0 + ai[u][n] * q0;
            }
        }
        if constexpr (PER_T) {
#pragma unroll
            for (int e = 0; e < NV; ++e) c_sum[e] += v[e];
        } else {
            const double total = lane_sums<NV>(v);
            if (o_unit) {
                *o_unit = total;
                o_unit += o_step;
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if constexpr (PER_T) {
        if (A.k0 + 32 * (int)fixed + lane >= A.k1) return;
#pragma unroll
        for (int e = 0; e < NV; e += 2)
            if (w0 + e / (2 * NC) < A.n_w) o_part[place(e) * A.n_t] = make_double2(c_sum[e], c_sum[e + 1]);
    }
}

// A pair's parts are added up as kSubSums sums over the parts s, s + kSubSums, ..., then in the order of s.  Single
// threads walking all parts took 2 to 4 us more of calls of 45 to 100 us: the loads of one batch wait for the last.
constexpr int kSubSums = 4;

// Sum s of a pair's n_parts values at p[part per], eight loads in flight (past the end zeros, which change no sum).
__device__ __forceinline__ double2 sub_sum(const double2* __restrict__ p, int s, int n_parts, size_t per) {
    constexpr int kBatch = 8;
    double2 v = make_double2(0.0, 0.0);
    for (int a = s; a < n_parts; a += kBatch * kSubSums) {
        double2 x[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int part = a + u * kSubSums;
            x[u] = part < n_parts ? p[part * per] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            v.x += x[u].x;
            v.y += x[u].y;
        }
    }
    return v;
}

// out[p][q] = the sum of pair p's parts at partial[p][part][q].
__global__ void k_direct_pairs(const double2* __restrict__ partial, int n_parts, size_t per, size_t n_pairs,
                               double2* __restrict__ out) {
    const size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= n_pairs * per) return;
    const double2* p = partial + at / per * (n_parts * per) + at % per;
    double2 sum = sub_sum(p, 0, n_parts, per);
#pragma unroll
    for (int s = 1; s < kSubSums; ++s) {
        const double2 v = sub_sum(p, s, n_parts, per);
        sum.x += v.x;
        sum.y += v.y;
    }
    out[at] = sum;
}

constexpr int kReduceRows = 32;
// Rows of threads that share a frame's n pairs: one a pair, as a power of two, up to 32.
int reduce_rows(size_t n) {
    int r = 1;
    while (r < kReduceRows && (size_t)r < n) r *= 2;
    return r;
}

// out[k][q] = the sum over frame k's n pairs of their parts' sums: blockDim.y strided rows of threads, then the rows
// in order (an order that depends on n and n_parts only).  ONE: there is one part a pair; otherwise a warp's lanes
// are kSubSums sums of 32 / kSubSums values.
template <bool ONE>
__global__ void __launch_bounds__(32 * kReduceRows)
    k_direct_reduce(const double2* __restrict__ partial, size_t n, int n_parts, size_t per, double2* __restrict__ out) {
    constexpr int NS = ONE ? 1 : kSubSums, NQ = 32 / NS;
    __shared__ double2 red[kReduceRows][NQ];
    const int ql = threadIdx.x % NQ, s = threadIdx.x / NQ;
    const size_t q = (size_t)blockIdx.x * NQ + ql;
    const size_t per_pair = n_parts * per;
    const double2* p = partial + blockIdx.y * n * per_pair + q;
    double2 acc = make_double2(0.0, 0.0);
    for (size_t a = threadIdx.y; a < n; a += blockDim.y) {
        double2 v = make_double2(0.0, 0.0);
        if (q < per) v = ONE ? p[a * per_pair] : sub_sum(p + a * per_pair, s, n_parts, per);
        double2 sum = v;
#pragma unroll
        for (int o = 1; o < NS; ++o) {
            sum.x += __shfl_sync(0xffffffffu, v.x, ql + o * NQ);
            sum.y += __shfl_sync(0xffffffffu, v.y, ql + o * NQ);
        }
        acc.x += sum.x;
        acc.y += sum.y;
    }
    if (s == 0) red[threadIdx.y][ql] = acc;  // (the other lanes' sums are not in this order)
    __syncthreads();
    if (threadIdx.y || s || q >= per) return;
    double2 sum = make_double2(0.0, 0.0);
    for (int y = 0; y < (int)blockDim.y; ++y) {
        sum.x += red[y][ql].x;
        sum.y += red[y][ql].y;
    }
    out[(size_t)blockIdx.y * per + q] = sum;
}

template <bool ONE>
void launch_reduce(const double2* partial, size_t n, int n_parts, size_t per, size_t frames, double2* out, cudaStream_t st) {
    constexpr size_t NQ = ONE ? 32 : 32 / kSubSums;
    const size_t gx = (per + NQ - 1) / NQ;
    if (gx > 0x7fffffffULL) throw Error{"direct kernel: too many outputs for one launch"};
    k_direct_reduce<ONE><<<dim3((unsigned)gx, (unsigned)frames), dim3(32, reduce_rows(n)), 0, st>>>(partial, n, n_parts, per,
                                                                                               out);
    CUDA_OK(cudaGetLastError());
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

// Arguments past kTwinMax: |w| times the largest time or position difference.
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
    return !(wmax * (tmax + xmax) < kTwinMax);
}

struct DirectPlan {
    int G;
    int nw, nc;          // frequencies per warp, columns per pass
    int nkc;             // blocks of 32 steps
    int per_warp;        // step blocks per warp
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

template <int G>
void launch_b(const DirArgs& A, bool exact, cudaStream_t st) {
    const size_t nkb = (A.k1 - A.k0 + kStepBlock - 1) / kStepBlock;
    const size_t blocks = (A.n_fs * A.n_cos * nkb + kDirWarps - 1) / kDirWarps;
    if (blocks > 0x7fffffffULL) throw Error{"direct kernel: too many (bubble, row, step) blocks for one launch"};
    if (exact)
        k_direct_b<G, true><<<(unsigned)blocks, 32 * kDirWarps, 0, st>>>(A);
    else
        k_direct_b<G, false><<<(unsigned)blocks, 32 * kDirWarps, 0, st>>>(A);
    CUDA_OK(cudaGetLastError());
}

// gx: (bubble, step block) units of the grid
template <int NC, int NW, bool PER_T>
void launch_a(const RowSumArgs& R, int G, size_t gx, bool big, cudaStream_t st) {
    const int groups = (R.d.n_w + NW - 1) / NW, warps = std::min(kDirWarps, groups);
    const int w_tiles = (groups + warps - 1) / warps;
    if (gx * w_tiles > 0x7fffffffULL) throw Error{"direct kernel: too many (bubble, step) blocks for one launch"};
    const dim3 grid((unsigned)(gx * w_tiles), (unsigned)(R.d.S * G / NC));
    const size_t smem = ((size_t)kRowStages * stage_pairs<NC>() * 2 * NC * 32 + R.d.n_cos) * sizeof(double);
    auto* kernel = big ? k_direct_a<NC, NW, true, PER_T> : k_direct_a<NC, NW, false, PER_T>;
    constexpr size_t most = kMaxBlockShared - kPhaseTable * sizeof(double2);
    if (smem > most) throw Error{"n_cos_thetax too large for the shared-memory layout"};
    allow_shared(kernel, most);
    kernel<<<grid, 32 * warps, smem, st>>>(R, G, w_tiles);
    CUDA_OK(cudaGetLastError());
}

// Step factors of the whole job (all steps, every radiating bubble).
void launch_steps(Device* dev, DirArgs& A) {
    A.tf = (A.n_t + kStepBlock - 1) / kStepBlock * kStepBlock;
    dev->fact_D.ensure((size_t)A.n_sel * (1 + A.S * A.M) * A.tf * sizeof(double));
    A.steps = (double*)dev->fact_D.p;
    const dim3 g((unsigned)(A.tf / kStepBlock), (unsigned)std::min(A.n_sel, 65535), (unsigned)(A.n_sel / 65535 + 1));
    if (g.z > 65535) throw Error{"too many radiating bubbles"};
    k_direct_steps<<<g, kStepBlock, 0, dev->stream>>>(A);
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

constexpr size_t kDirectBufferBytes = (size_t)1 << 30;   // B of one launch, at most
constexpr size_t kDirectSmallBytes = (size_t)1 << 28;    // ... taken without a look at the free memory
constexpr size_t kDirectPartialBytes = (size_t)1 << 28;  // partial sums of one launch (spectrum), of the job (integrand)
// Warps that the integrand's parts are cut for: 8 per scheduler of a B200.  A constant, so that the order of its sums
// depends on the job alone.
constexpr size_t kIntegrandWarps = 148 * 4 * 8;

// Steps and pairs of a launch whose B, `step_bytes` a step and pair, fits `limit`: whole step blocks of
// k_direct_b, one at least; all of a pair's steps before a second pair.
struct DirectRange {
    size_t steps, pairs;
};
DirectRange direct_range(size_t n_t, size_t pairs, size_t step_bytes, size_t limit) {
    DirectRange r;
    const size_t all = (n_t + kStepBlock - 1) / kStepBlock * kStepBlock;
    r.steps = std::min(all, std::max<size_t>(1, limit / (step_bytes * kStepBlock)) * kStepBlock);
    r.pairs = std::min(pairs, std::max<size_t>(1, limit / (step_bytes * r.steps)));
    if (r.steps < all) r.pairs = 1;
    return r;
}

// The largest range whose work arrays the device has room for: `reserve` allocates those of a range under a limit
// for B and says whether it could.  256 MiB serve a job that needs no more; a larger one, and one that they were
// refused, gets a third of the free memory up to 1 GiB (the query takes 67 us).
template <class F>
DirectRange reserve_range(const Device* dev, const SpectrumJob& job, size_t pairs, size_t step_bytes, F&& reserve) {
    auto third = [&]() -> size_t {
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return kDirectSmallBytes;
        return std::min((free_b + dev->beta.cap) / 3, kDirectBufferBytes);
    };
    size_t limit = kDirectSmallBytes;
    if (pairs * step_bytes * job.n_t > limit) limit = third();
    for (;;) {
        DirectRange r = direct_range(job.n_t, pairs, step_bytes, limit);
        if (reserve(r, limit)) return r;
        if (limit == 0) throw Error{"CUDA error: out of memory (work arrays of the direct kernel)"};
        limit = std::min(limit / 2, third());
    }
}

}  // namespace

// (the pairs' sums; the other work arrays are cut to size)
size_t direct_bytes_per_frame(const SpectrumJob& job) {
    return job.n_sel * (job.tensor ? 6 : 2) * job.n_sets * job.n_w * sizeof(double2);
}

uint64_t launch_direct(Device* dev, const SpectrumJob& job, const DirectInputs& in, size_t kn, double2* out) {
    const size_t pairs = kn * job.n_sel;
    const DirectPlan P = direct_plan(dev, job, pairs);
    const size_t cols = (size_t)P.G * job.n_sets, per = cols * job.n_w;
    const bool exact = direct_exact(job), big = direct_big(job);
    DirArgs A = direct_args(job, in);
    launch_steps(dev, A);
    uint64_t launches = 1;
    const size_t step_bytes = job.n_cos * cols * sizeof(double), part_bytes = P.nkc * per * sizeof(double2);
    const DirectRange r = reserve_range(dev, job, pairs, step_bytes, [&](DirectRange& q, size_t limit) {
        q.pairs = std::min(q.pairs, std::max<size_t>(1, std::min(limit, kDirectPartialBytes) / part_bytes));
        return (q.pairs == pairs || dev->fact_partial.try_ensure(pairs * per * sizeof(double2))) &&
               dev->partial.try_ensure(q.pairs * part_bytes) && dev->beta.try_ensure(q.pairs * step_bytes * q.steps);
    });
    A.B = (double*)dev->beta.p;
    // in several launches each pair's parts are added up before the next ones overwrite them
    const bool once = r.pairs == pairs;
    for (size_t f0 = 0; f0 < pairs; f0 += r.pairs) {
        A.fs0 = f0;
        A.n_fs = std::min(r.pairs, pairs - f0);
        for (size_t k0 = 0; k0 < job.n_t; k0 += r.steps) {
            A.k0 = (int)k0;
            A.k1 = (int)std::min(job.n_t, k0 + r.steps);
            A.tp = (A.k1 - A.k0 + 31) & ~31;
            if (job.tensor)
                launch_b<6>(A, exact, dev->stream);
            else
                launch_b<2>(A, exact, dev->stream);
            const RowSumArgs R{A, P.per_warp, P.nkc, (int)(k0 / 32), (double2*)dev->partial.p};
            const size_t groups = ((A.k1 - A.k0 + 31) / 32 + P.per_warp - 1) / P.per_warp;
            dispatch_a<false>(R, P, A.n_fs * groups, big, dev->stream);
            launches += 2;
        }
        if (!once) {
            const size_t n = A.n_fs * per;
            if ((n + 255) / 256 > 0x7fffffffULL) throw Error{"direct kernel: too many partial sums for one launch"};
            k_direct_pairs<<<(unsigned)((n + 255) / 256), 256, 0, dev->stream>>>(
                (const double2*)dev->partial.p, P.nkc, per, A.n_fs, (double2*)dev->fact_partial.p + f0 * per);
            CUDA_OK(cudaGetLastError());
            ++launches;
        }
    }
    if (once)
        launch_reduce<false>((const double2*)dev->partial.p, job.n_sel, P.nkc, per, kn, out, dev->stream);
    else
        launch_reduce<true>((const double2*)dev->fact_partial.p, job.n_sel, 1, per, kn, out, dev->stream);
    return launches + 1;
}

uint64_t launch_direct_integrand(Device* dev, const SpectrumJob& job, const DirectInputs& in, double2* out) {
    const size_t pairs = job.n_sel;
    DirectPlan P = direct_plan(dev, job, pairs);
    const size_t cols = (size_t)P.G * job.n_sets, per = cols * job.n_w * job.n_t;
    const bool exact = direct_exact(job), big = direct_big(job);
    // bubbles of a part: few enough for the chip to be full, as many as keep the parts' outputs small
    const size_t warps = ((job.n_w + P.nw - 1) / P.nw) * (cols / P.nc) * P.nkc;
    size_t parts = std::min(pairs, std::max<size_t>(1, (kIntegrandWarps + warps - 1) / warps));
    parts = std::min(parts, std::max<size_t>(1, kDirectPartialBytes / (per * sizeof(double2))));
    P.per_warp = (int)((pairs + parts - 1) / parts);
    parts = (pairs + P.per_warp - 1) / P.per_warp;
    if ((per + 31) / 32 > 0x7fffffffULL) throw Error{"direct kernel: integrand too large for one launch"};
    DirArgs A = direct_args(job, in);
    launch_steps(dev, A);
    uint64_t launches = 1;
    const size_t step_bytes = job.n_cos * cols * sizeof(double);
    dev->partial.ensure(parts * per * sizeof(double2));
    const DirectRange r = reserve_range(dev, job, pairs, step_bytes, [&](const DirectRange& q, size_t) {
        return dev->beta.try_ensure(q.pairs * step_bytes * q.steps);
    });
    A.B = (double*)dev->beta.p;
    for (size_t f0 = 0; f0 < pairs; f0 += r.pairs) {
        A.fs0 = f0;
        A.n_fs = std::min(r.pairs, pairs - f0);
        const size_t touched = (f0 + A.n_fs - 1) / P.per_warp - f0 / P.per_warp + 1;
        for (size_t k0 = 0; k0 < job.n_t; k0 += r.steps) {
            A.k0 = (int)k0;
            A.k1 = (int)std::min(job.n_t, k0 + r.steps);
            A.tp = (A.k1 - A.k0 + 31) & ~31;
            if (job.tensor)
                launch_b<6>(A, exact, dev->stream);
            else
                launch_b<2>(A, exact, dev->stream);
            const RowSumArgs R{A, P.per_warp, 0, 0, (double2*)dev->partial.p};
            dispatch_a<true>(R, P, touched * (size_t)(A.tp / 32), big, dev->stream);
            launches += 2;
        }
    }
    launch_reduce<true>((const double2*)dev->partial.p, parts, 1, per, 1, out, dev->stream);
    return launches + 1;
}

}  // namespace bgw
