// Factored spectrum kernels (FP64 and mixed precision).
//
// The reference accumulates, per bubble a, cos-theta row i and time t_k,
//   B_{s,g}(a,i,k) e^{-i w dt_k c_i} dc v_i  x  e^{i w (t_k - z_a)} u_k cut_k dt / (6 pi)
// (generalized_bulk_flow.rs:481-873).  The phase splits as
//   w [(t_k - z_a) - (t_k - t_a) c_i] = w t_k (1 - c_i) + w (t_a c_i - z_a),
// so for a fixed row i the time phase M_i[w, k] = e^{i w (1 - c_i) t_k} is the
// same for every bubble and every k-hat frame, and
//   C_{s,g}(w) = sum_i sum_a e^{i w (t_a c_i - z_a)} Y_i[w, (a,s,g)],
//   Y_i = M_i (W x T complex)  .  beta_i (T x columns real),
// a GEMM per row (columns = frame x bubble x set x {+,x}) followed by a
// per-(w, bubble) phase in the epilogue.
//
// beta comes from the collision structure without evaluating every patch at
// every t: with q_j = w_j g(phi_j) (g = cos 2phi, sin 2phi) and
//   f = sum_m a_m (tau_j / dt)^{p_m} exp(-(dt - tau_j) / width)   (collided),
//   dt^3 sum_j q_j f_j = dt^3 U(k) + sum_m a_m dt^{3-p_m} e^{-dt/width} Pm(k),
// where U(k) sums q_j over the patches not yet collided at step k and Pm(k)
// sums q_j tau_j^{p_m} e^{tau_j/width} over those already collided.  k_beta adds
// each collided patch to the first time step at which the reference's test
// (t_k - t_a) >= tau_j holds (exact FP64 comparisons) and forms Pm as running
// sums and U as backward sums of the remaining terms (total minus collided
// cancels catastrophically once most patches have collided).
//
// Kernels:
//   k_time_tables   per bubble and t: dt^3 and dt^{3-p} e^{-dt/width}
//   k_beta          per (frame, bubble, row): beta, as FP64 or FP32 values or as
//                   int8 digits with one scale per row (k_beta_sorted: the
//                   digits of calls whose masks the adjoint reads again)
//   k_gemm_fold     FP64 product over t, folded about the middle of the time grid
//   k_gemm          FP32 product over t in chunks of kKC, FP64 epilogue
//                   (spectrum_tc.cu: the int8 digits' tensor-core product)
//   k_reduce_tiles  deterministic sum of the column-tile partials per frame

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "bgw_internal.h"
#include "device_common.cuh"
#include "powers.cuh"
#include "spectrum_factored.cuh"
#include "spectrum_tc.cuh"
#include "tc_ptx.cuh"

namespace bgw {

constexpr int kKC = 32;          // time steps per GEMM k-tile
constexpr int kFold = 16;        // mixed: FP32 partial sums are folded into FP64 every kFold steps
constexpr int kWT = 64;          // frequencies per CTA
constexpr int kRows = 2 * kWT;   // GEMM rows: (Re, Im) of each frequency
constexpr int kThreads = 256;
constexpr int kTM = 8;           // register tile rows per thread (columns: TN = 8 FP32, 4 FP64)

// ---------------------------------------------------------------------------
// Place of step k in a row of the step factors and of k_beta's bins: within each block of 32 steps the first
// two of every four steps come first, so that lanes with four steps each read them as two 16-byte words
// without a bank conflict (or half a line) between them.
__host__ __device__ __forceinline__ int step_at(int k) {
    return (k & ~31) | ((k & 2) << 3) | ((k >> 1) & 14) | (k & 1);
}

// Step factors of a bubble, table row q over steps at ((slot (1 + SM) + q) tf + step_at(k)): row 0 the step weight
// (time cutoff x trapezoid end weight) times dt^3, row 1 + q the same times a_q dt^{3-p_q} e^{-dt/width};
// zero where dt <= 0 and past n_t (tf is n_t rounded up to whole blocks of 32 steps).
__global__ void k_time_tables(const D4* __restrict__ bub, const uint32_t* __restrict__ sel, int n_sel,
                              const double* __restrict__ t_arr, int n_t, int tf, const double* __restrict__ powers,
                              const double* __restrict__ coeffs, const double* __restrict__ cutw, int SM,
                              int has_damp, double damp, double* __restrict__ D, int* __restrict__ kfirst) {
    const int slot = blockIdx.x;
    const int k = blockIdx.y * blockDim.x + threadIdx.x;
    if (slot >= n_sel || k >= tf || sel[slot] == kNoSlot) return;
    const double ta = bub[sel[slot]].t;
    const double dt = k < n_t ? t_arr[k] - ta : 0.0;
    double* row = D + (size_t)slot * (1 + SM) * tf + step_at(k);
    const bool on = dt > 0.0;
    const double wk = k < n_t ? cutw[k] * ((k == 0 || k == n_t - 1) ? 0.5 : 1.0) : 0.0;
    const double d3 = on ? dt * (dt * dt) : 0.0;
    row[0] = wk * d3;
    const double e = has_damp ? exp(-dt / damp) : 1.0;
    for (int q = 0; q < SM; ++q)
        row[(size_t)(1 + q) * tf] = d3 != 0.0 ? wk * coeffs[q] * (pow(dt, 3.0 - powers[q]) * e) : 0.0;
    if (k >= n_t) return;
    // first active step (t_a <= t_k and dt > 0): monotone in k
    if (on && (k == 0 || !(t_arr[k - 1] - ta > 0.0))) kfirst[slot] = k;
    if (k == n_t - 1 && !on) kfirst[slot] = n_t;
}

// Per (bubble, block of 32 steps): the least and the largest D_q(k) of each
// table row over the block's steps (one warp, a lane each), stored as (min, max)
// pairs.
__global__ void k_time_maxima(const double* __restrict__ D, int n_sel, int tf, int nblk, int Q,
                              double* __restrict__ Dmax) {
    const long wid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long)n_sel * nblk) return;
    const int slot = (int)(wid / nblk), b = (int)(wid % nblk);
    for (int q = 0; q < Q; ++q) {
        const double v = D[((size_t)slot * Q + q) * tf + (b << 5) + lane];
        double lo = v, hi = v;
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            Dmax[((size_t)wid * Q + q) * 2] = lo;
            Dmax[((size_t)wid * Q + q) * 2 + 1] = hi;
        }
    }
}

// ---------------------------------------------------------------------------
// k_beta: one warp per row (frame, slot, i).  The row's collided patches
// become events at the first step k_j with (t_k - t_a) >= tau_j (exact FP64
// comparisons, GBF:405).  Before the row's first event and after its last the
// collided sums Pm and the uncollided sums U are constant ("quiet" steps, two
// sets of constants); in between the steps are formed in segments of 128, from
// the first event's block of 32 on: every event's weights are added to its
// step's bin in shared memory (events of one step one after another, in lane
// order), and warp scans, lane = 4 consecutive steps, give Pm(k) as a prefix and
// U(k) as a suffix sum -- both are sums of the terms they stand for, never
// differences (a difference cancels catastrophically once most patches have
// collided).  At 192 phi patches and 1024 steps a row's events span about two
// blocks, so one segment holds them.
// beta(k) = rf_i u_k cut_k [dt^3 U(k) + sum_m a_m dt^{3-p_m} e^{-dt/w} Pm(k)]
// is written to beta[frame][i][col][k], col = slot*2S + 2s + g.
//
// What bounds it: issue and shared memory.  Sorting the events into blocks and again into steps,
// with totals and scans over every block, took two thirds of 62.8 ms for 8
// frames of 4096 bubbles x 192 rows; the digits and stores of the quiet steps a
// quarter.  Now 38.8 ms there (the 51 GB of digits and 10 GB of delays alone:
// 9.3 ms at the measured copy rate), and 1.42 ms in FP64 for 4 frames of 512
// bubbles x 128 rows x 512 steps (2.19).  Issue and the shared-memory pipe are
// each 62 % busy; with the steps of a block in order (two-way bank conflicts)
// and the delays' two steps read one after the other it took 47 ms.
struct BetaArgs {
    const double* tau;     // (kn, n_sel, n_cos*n_phi)
    const D4* bub;         // bubbles (frame 0; times are frame independent)
    const uint32_t* sel;
    int n_sel, n_cos, n_phi, n_t, S, M;
    const double* t_arr;
    const double* cutw;
    const double* cos_t;
    const double* cos2;
    const double* sin2;
    const double* powers;  // (S*M)
    const double* coeffs;  // (S*M)
    const double* D;       // (n_sel, 1+S*M, tf) step factors
    int tf;
    int has_damp;
    double damp;
    double dphi, dcos, dt;
    long n_rows;           // kn * n_sel * n_cos
    int nblk;              // ceil(n_t / 32)
    long cols_pad;         // columns per (frame, i): tiles_per_frame * tile_cols
    int tile_cols;         // columns of one GEMM tile
    int bpt;               // bubbles per tile
    int t_pad;             // row length of beta
    int keep;              // event segments whose bins a warp holds at once
    int per_warp;          // doubles of shared memory per warp
    int per_warp_bytes;    // the same of k_beta_sorted, in bytes
    int tiles;             // column tiles per frame (int8 digit layout)
    double* scale;         // int8 digit layout: (kn, n_sel, n_cos) row scales, max |beta| of the row
    const double* Dmax;    // int8 digit layout: (n_sel, nblk, 1+S*M, 2) least and largest D over each block's steps
};

constexpr size_t kBetaShared = 220 * 1024;  // shared memory of k_beta's blocks on an SM, at most
constexpr int kSegBlocks = 4;              // blocks of 32 steps in an event segment
constexpr int kSeg = 32 * kSegBlocks;

__device__ __forceinline__ void copy8_async(double* smem, const double* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// warps of a block, and blocks per SM: 24 warps at 80 registers with one term, 16 at 128 with two
__host__ __device__ constexpr int beta_warps(int SMC) { return SMC == 1 ? 8 : 4; }
__host__ __device__ constexpr int beta_blocks(int SMC) { return SMC == 1 ? 3 : SMC == 2 ? 4 : SMC <= 4 ? 3 : 2; }
// With two terms and more a warp takes every so-manieth row and fetches the next one's delays while it
// works (16 or 8 warps do not hide them: 564 against 760 us for 6 frames of 101 bubbles, 4 terms); with one
// term the loop's registers spill (67 against 47 ms for 8 frames of 4096 bubbles).
__host__ __device__ constexpr int beta_rows_held(int SMC) { return SMC == 1 ? 1 : 2; }
template <class Real, int SMC>
__global__ void __launch_bounds__(32 * beta_warps(SMC), beta_blocks(SMC)) k_beta(BetaArgs A, Real* __restrict__ beta) {
    extern __shared__ __align__(16) double sm_beta[];
    constexpr bool kI8 = std::is_same<Real, int8_t>::value, kLoop = SMC > 1;
    constexpr int NQ = 2 + 2 * SMC;  // weights of an event: cos, sin; then cos and sin times each term's factor
    constexpr unsigned full = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NB = A.nblk;
    // Lane l holds the patches [c l, c l + c): neighbouring patches collide at the same or the next step,
    // so most of a step's events are added up in registers before they reach its bin.  Their rows in shared
    // memory have an odd pitch (no bank conflicts).
    const int c_pat = (A.n_phi + 31) >> 5, pitch = c_pat | 1;
    double2* s_wgt = reinterpret_cast<double2*>(sm_beta);                       // [32 pitch] weights, block's own
    double* base_w = sm_beta + 64 * pitch + (size_t)warp * A.per_warp;
    double* bins = base_w;                                                   // [keep][NQ][kSeg]
    double* s_const = bins + (size_t)A.keep * NQ * kSeg;                     // [4 + 2 SMC] quiet constants
    double* s_tau = s_const + 4 + 2 * SMC;                                   // [rows held][32 pitch] delays
    int* s_kj = reinterpret_cast<int*>(s_tau + beta_rows_held(SMC) * 32 * pitch);  // [32 pitch] first collided steps
    for (int j = threadIdx.x; j < A.n_phi; j += blockDim.x) {
        const double wj = (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0;
        s_wgt[j / c_pat * pitch + j % c_pat] = make_double2(wj * A.cos2[j], wj * A.sin2[j]);
    }
    auto beta_row = [&](long row, const double* s_tau) {
    const int slot = (int)((row / A.n_cos) % A.n_sel);
    if (A.sel[slot] == kNoSlot) return;  // a padding slot of a batched job: its columns are never read
    const int i = (int)(row % A.n_cos);
    const long frame = row / ((long)A.n_cos * A.n_sel);
    const double ta = A.bub[A.sel[slot]].t;
    const double inv_dt = 1.0 / A.dt;  // the estimate below is only a starting point
    constexpr int kNever = 0x7fffffff;
    // first k with (t_k - t_a) >= tau_j: arithmetic estimate, then exact comparisons (the predicate is
    // monotone in k) settle the boundary; the two steps they read first are loaded ahead
    auto guess = [&](double tj) -> int {
        const double est = ceil((ta + tj - A.t_arr[0]) * inv_dt);
        return est < 0.0 ? 0 : (est > (double)A.n_t ? A.n_t : (int)est);
    };
    auto settle = [&](double tj, int lo, double below, double here) -> int {
        if (!(tj > 0.0)) return kNever;
        if ((lo > 0 && below - ta >= tj) || (lo < A.n_t && !(here - ta >= tj))) {
            while (lo > 0 && A.t_arr[lo - 1] - ta >= tj) --lo;
            while (lo < A.n_t && !(A.t_arr[lo] - ta >= tj)) ++lo;
        }
        return lo < A.n_t ? lo : kNever;
    };
    int k_lo = kNever, k_hi = -1;
    const int n_own = max(0, min(c_pat, A.n_phi - lane * c_pat));  // this lane's patches
    const int own = lane * pitch;
    for (int m = 0; m < n_own; m += 2) {  // two patches' loads in flight
        const bool two = m + 1 < n_own;
        const double tj = s_tau[own + m], tj2 = two ? s_tau[own + m + 1] : 0.0;
        const int lo = guess(tj), lo2 = guess(tj2);
        const double below = __ldg(A.t_arr + max(lo - 1, 0)), here = __ldg(A.t_arr + min(lo, A.n_t - 1));
        const double below2 = __ldg(A.t_arr + max(lo2 - 1, 0)), here2 = __ldg(A.t_arr + min(lo2, A.n_t - 1));
        const int kj = settle(tj, lo, below, here), kj2 = settle(tj2, lo2, below2, here2);
        s_kj[own + m] = kj;
        if (two) s_kj[own + m + 1] = kj2;
        k_lo = min(k_lo, min(kj, kj2));
        if (kj != kNever) k_hi = max(k_hi, kj);
        if (kj2 != kNever) k_hi = max(k_hi, kj2);
    }
    k_lo = __reduce_min_sync(full, k_lo);
    k_hi = __reduce_max_sync(full, k_hi);
    // event segments: blocks [b_ev, b_ev + 4 n_seg); without events none, and every block is "before"
    const int b_ev = k_hi < 0 ? NB : k_lo >> 5;
    const int n_seg = k_hi < 0 ? 0 : ((k_hi >> 5) - b_ev) / kSegBlocks + 1;
    const int b_aft = min(NB, b_ev + kSegBlocks * n_seg);
    const double ci = A.cos_t[i];
    const double vi = (i == 0 || i == A.n_cos - 1) ? 0.5 : 1.0;
    const double rf = (0.5 * (1.0 - ci * ci) * A.dphi) * (A.dcos * vi) * A.dt * (1.0 / (6.0 * CUDART_PI));
    const double* Dslot = A.D + (size_t)slot * (1 + SMC) * A.tf;
    // constants of the quiet steps: uncollided sums before (0, 1) and after (2, 3) the events, collided sums
    // after them (4 ..); held in shared memory
    if (n_seg == 0) {
        double u0 = 0.0, u1 = 0.0;
        for (int m = 0; m < n_own; ++m) {
            u0 += s_wgt[own + m].x;
            u1 += s_wgt[own + m].y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            u0 += __shfl_xor_sync(full, u0, o);
            u1 += __shfl_xor_sync(full, u1, o);
        }
        if (lane < 4 + 2 * SMC) s_const[lane] = lane == 0 ? u0 : lane == 1 ? u1 : 0.0;
        __syncwarp();
    }
    const int at4 = step_at(4 * lane);  // the lane's four steps of a segment: at4, at4 + 1, at4 + 16, at4 + 17
    auto four = [&](const double* p, double (&v)[4]) {
        const double2 lo = reinterpret_cast<const double2*>(p + at4)[0], hi = reinterpret_cast<const double2*>(p + at4)[8];
        v[0] = lo.x;
        v[1] = lo.y;
        v[2] = hi.x;
        v[3] = hi.y;
    };
    // The running sums of segment g into bins w: rows 0, 1 the uncollided sums U after each step, the
    // others the collided sums Pm up to it (lane: steps 4 lane .. 4 lane + 3).
    auto form = [&](int g, double* w) {
        const int s0 = (b_ev + g * kSegBlocks) << 5, s1 = s0 + kSeg;
        double2* wz = reinterpret_cast<double2*>(w);
        for (int q = lane; q < NQ * kSeg / 2; q += 32) wz[q] = make_double2(0.0, 0.0);
        __syncwarp();
        double base[NQ];  // uncollided after the segment, collided before it
#pragma unroll
        for (int q = 0; q < NQ; ++q) base[q] = 0.0;
        double run[NQ];  // the lane's current run of patches with one collision step
        int k_run = -1;
        for (int m = 0; m <= c_pat; ++m) {
            const int kj = m < n_own ? s_kj[own + m] : kNever;
            const bool flush = k_run >= 0 && kj != k_run;
            if (__any_sync(full, flush)) {
                const unsigned same = __match_any_sync(full, flush ? k_run : -1 - lane);
                const int rank = flush ? __popc(same & ((1u << lane) - 1u)) : -1;
                const int rounds = __reduce_max_sync(full, rank);
                for (int r = 0; r <= rounds; ++r) {
                    if (rank == r) {
                        double* e = w + step_at(k_run - s0);
#pragma unroll
                        for (int q = 0; q < NQ; ++q) e[q * kSeg] += run[q];
                    }
                    __syncwarp();
                }
                if (flush) k_run = -1;
            }
            if (m >= n_own) continue;
            double x[NQ];
            const double2 wg = s_wgt[own + m];
            x[0] = wg.x;
            x[1] = wg.y;
            if (kj >= s1) {
                base[0] += x[0];
                base[1] += x[1];
                continue;
            }
            const double tj = s_tau[own + m];
            const double ed = A.has_damp ? exp(tj / A.damp) : 1.0;
#pragma unroll
            for (int t = 0; t < SMC; ++t) {
                const double f = tpow(tj, A.powers[t]) * ed;
                x[2 + 2 * t] = x[0] * f;
                x[3 + 2 * t] = x[1] * f;
            }
            if (kj < s0) {
#pragma unroll
                for (int q = 2; q < NQ; ++q) base[q] += x[q];
            } else if (k_run < 0) {
                k_run = kj;
#pragma unroll
                for (int q = 0; q < NQ; ++q) run[q] = x[q];
            } else {
#pragma unroll
                for (int q = 0; q < NQ; ++q) run[q] += x[q];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < NQ; ++q) base[q] += __shfl_xor_sync(full, base[q], o);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            double2* e = reinterpret_cast<double2*>(w + q * kSeg + at4);
            const double2 lo = e[0], hi = e[8];
            if (q < 2) {  // the sum of the later steps' events
                const double v2 = hi.y, v1 = hi.x + v2, v0 = lo.y + v1;
                double run = lo.x + v0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double t = __shfl_down_sync(full, run, o);
                    if (lane + o < 32) run += t;
                }
                double later = __shfl_down_sync(full, run, 1);
                if (lane == 31) later = 0.0;
                later += base[q];
                e[0] = make_double2(v0 + later, v1 + later);
                e[8] = make_double2(v2 + later, later);
                if (g == 0 && lane == 0) s_const[q] = run + base[q];
                if (g == n_seg - 1 && lane == 0) s_const[2 + q] = base[q];
            } else {  // this step's and the earlier ones'
                const double v0 = lo.x, v1 = v0 + lo.y, v2 = v1 + hi.x, v3 = v2 + hi.y;
                double run = v3;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double t = __shfl_up_sync(full, run, o);
                    if (lane >= o) run += t;
                }
                double before = __shfl_up_sync(full, run, 1);
                if (lane == 0) before = 0.0;
                before += base[q];
                e[0] = make_double2(v0 + before, v1 + before);
                e[8] = make_double2(v2 + before, v3 + before);
                if (g == n_seg - 1 && lane == 31) s_const[2 + q] = run + base[q];
            }
        }
        __syncwarp();
    };
    // table row q at the lane's four steps of the blocks from b on
    auto factors = [&](int q, int b, double (&v)[4]) {
        const double2* d = reinterpret_cast<const double2*>(Dslot + (size_t)q * A.tf + (b << 5) + at4);
        const double2 lo = __ldg(d), hi = __ldg(d + 8);
        v[0] = lo.x;
        v[1] = lo.y;
        v[2] = hi.x;
        v[3] = hi.y;
    };
    // beta of set s at the lane's steps of segment g from its bins
    auto seg_values = [&](int g, const double* w, int s, double (&xc)[4], double (&xs)[4]) {
        const int b = b_ev + g * kSegBlocks;
        const bool on = b + (lane >> 3) < NB;
        double d[4] = {0.0, 0.0, 0.0, 0.0}, c[4], e[4];
        if (on) factors(0, b, d);
        four(w, c);
        four(w + kSeg, e);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            xc[m] = d[m] * c[m];
            xs[m] = d[m] * e[m];
        }
        const int t0 = s * A.M, t1 = t0 + A.M;
#pragma unroll
        for (int t = 0; t < SMC; ++t) {
            if (SMC > 1 && (t < t0 || t >= t1)) continue;
            if (on) factors(1 + t, b, d);
            four(w + (2 + 2 * t) * kSeg, c);
            four(w + (3 + 2 * t) * kSeg, e);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                xc[m] = fma(d[m], c[m], xc[m]);
                xs[m] = fma(d[m], e[m], xs[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            xc[m] *= rf;
            xs[m] *= rf;
        }
    };
    const long col = (long)(slot / A.bpt) * A.tile_cols + (long)(slot % A.bpt) * 2 * A.S;
    const int nbase = (slot % A.bpt) * 2 * A.S;
    double vmax = 0.0;
    if constexpr (kI8) {
        // Digits (streaming stores: the GEMM reads them back from DRAM), lane = 4 steps of 4 blocks:
        // the packed digits of 4 steps are transposed in registers, so that a store instruction
        // fills whole 32-byte rows of the blocks.
        int8_t* blk_row = reinterpret_cast<int8_t*>(beta) +
                          (((size_t)frame * A.n_cos + i) * A.tiles + slot / A.bpt) * (size_t)NB * kI8BlockSet;
        const int s4 = (lane & 7) * 4;
        auto put = [&](int b, int s, uint32_t (&pc)[4], uint32_t (&ps)[4]) {
            uint32_t wc[4], ws[4];
            i8_transpose4(pc[0], pc[1], pc[2], pc[3], wc);
            i8_transpose4(ps[0], ps[1], ps[2], ps[3], ws);
            int8_t* blk = blk_row + (size_t)(b + (lane >> 3)) * kI8BlockSet;
            // two lanes hold 8 steps of both columns: the even one stores the first column's, the odd one the
            // second's (8 lanes of a block are here together).  Four 8-byte stores for eight of 4 bytes: 38.8
            // against 39.8 ms for 8 frames of 4096 bubbles x 192 rows.
            const bool odd = lane & 1;
            const unsigned eight = 0xffu << (lane & 24);
            blk += i8_swz(nbase + 2 * s + (odd ? 1 : 0), s4 & ~7);
#pragma unroll
            for (int d = 0; d < kI8Slices; ++d) {
                const uint32_t other = __shfl_xor_sync(eight, odd ? wc[d] : ws[d], 1);
                __stcs(reinterpret_cast<uint2*>(blk + d * kI8Block),
                       odd ? make_uint2(other, ws[d]) : make_uint2(wc[d], other));
            }
        };
        // Turns 0 .. n_seg - 1 form the event segments (their values stay in the set's own bins), turn
        // n_seg finds the scale and writes the quiet steps' digits, the others write the segments'
        // (formed again where there are more than the warp holds).
        double inv = 0.0;
        for (int turn = 0; turn <= 2 * n_seg; ++turn) {
            if (turn == n_seg) {
                // The row's scale is max |beta| over its steps and columns, found exactly without forming
                // every value: the event segments' are formed; a quiet block's beta = rf (D0(k) U + sum_m
                // Dm(k) Pm) is bounded by interval arithmetic over the per-block ranges of the step
                // factors, and such blocks are formed in decreasing order of their bound until no bound
                // exceeds the largest value found (most often one block: the last one, where dt^3 peaks).
                const double* Dmx = A.Dmax + (size_t)slot * NB * (1 + SMC) * 2;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(full, vmax, o));
                for (int bc = 0; bc < NB; bc += 32) {
                    const int bl = bc + lane;
                    double bnd = -1.0;  // this lane's block's bound (-1: none or in a segment)
                    if (bl < NB && (bl < b_ev || bl >= b_aft)) {
                        const bool aft = bl >= b_aft;
                        const double* mx = Dmx + (size_t)bl * (1 + SMC) * 2;
                        auto term = [&](double dlo, double dhi, double c, double& lo, double& hi, double& sa) {
                            const double p0 = dlo * c, p1 = dhi * c;
                            lo += fmin(p0, p1);
                            hi += fmax(p0, p1);
                            sa += fmax(fabs(dlo), fabs(dhi)) * fabs(c);
                        };
                        for (int s2 = 0; s2 < A.S; ++s2) {
                            const int t0 = s2 * A.M, t1 = t0 + A.M;
#pragma unroll
                            for (int g = 0; g < 2; ++g) {
                                double lo = 0.0, hi = 0.0, sa = 0.0;
                                term(mx[0], mx[1], s_const[aft ? 2 + g : g], lo, hi, sa);
                                if (aft) {
#pragma unroll
                                    for (int q = 0; q < SMC; ++q)
                                        if (SMC == 1 || (q >= t0 && q < t1))
                                            term(mx[2 + 2 * q], mx[3 + 2 * q], s_const[4 + 2 * q + g], lo, hi, sa);
                                }
                                // relative and absolute margins cover the rounding of these sums and of
                                // the values themselves (a few ulp of the summed magnitudes)
                                bnd = fmax(bnd, (fmax(fabs(lo), fabs(hi)) * (1.0 + 1e-12) + 1e-13 * sa) * rf);
                            }
                        }
                    }
                    for (;;) {
                        double bb = bnd;
                        int bi = lane;
                        for (int o = 16; o > 0; o >>= 1) {
                            const double ob = __shfl_xor_sync(full, bb, o);
                            const int oi = __shfl_xor_sync(full, bi, o);
                            if (ob > bb || (ob == bb && oi < bi)) {
                                bb = ob;
                                bi = oi;
                            }
                        }
                        // Every remaining bound is covered once no bound exceeds vmax (1 + 1e-10): a value up
                        // to that much above the scale still maps to |x F| <= F + 0.22, which rounds into the
                        // digit range.  (Without the slack, blocks whose values all equal the maximum, as after
                        // the last collision with powers = 3, would each be formed.)
                        if (!(bb > vmax * (1.0 + 1e-10))) break;
                        {
                            const int b = bc + bi;
                            const bool aft = b >= b_aft;
                            const double* d = Dslot + (b << 5) + lane;  // the block's steps in any order
                            const double d0 = d[0];
                            double m = 0.0;
                            for (int s2 = 0; s2 < A.S; ++s2) {
                                const int t0 = s2 * A.M, t1 = t0 + A.M;
                                double xc = d0 * s_const[aft ? 2 : 0], xs = d0 * s_const[aft ? 3 : 1];
#pragma unroll
                                for (int q = 0; q < SMC; ++q) {
                                    if (!aft || (SMC > 1 && (q < t0 || q >= t1))) continue;
                                    const double dq = d[(size_t)(1 + q) * A.tf];
                                    xc = fma(dq, s_const[4 + 2 * q], xc);
                                    xs = fma(dq, s_const[5 + 2 * q], xs);
                                }
                                m = fmax(m, fmax(fabs(xc), fabs(xs)));
                            }
                            m *= rf;
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(full, m, o));
                            vmax = fmax(vmax, m);
                        }
                        if (lane == bi) bnd = -1.0;
                    }
                }
                if (lane == 0) A.scale[row] = vmax;
                inv = vmax > 0.0 ? 1.0 / vmax : 0.0;
                // quiet steps: the constants with the scale (and F) folded in
                const double rinv = rf * inv;
                auto quiet = [&](int b_lo, int b_hi, bool aft) {
                    const double* U = s_const + (aft ? 2 : 0);
                    const double Uc = rinv * U[0], Us = rinv * U[1];
                    const bool none = U[0] == 0.0 && U[1] == 0.0;  // every patch has collided
                    double P[2 * SMC];
#pragma unroll
                    for (int q = 0; q < 2 * SMC; ++q) P[q] = rinv * s_const[4 + q];
                    for (int b = b_lo; b < b_hi; b += kSegBlocks) {
                        if (b + (lane >> 3) >= b_hi) continue;
                        for (int s = 0; s < A.S; ++s) {
                            const int t0 = s * A.M, t1 = t0 + A.M;
                            double xc[4] = {0.0, 0.0, 0.0, 0.0}, xs[4] = {0.0, 0.0, 0.0, 0.0}, d[4];
                            if (!none) {
                                factors(0, b, d);
#pragma unroll
                                for (int m = 0; m < 4; ++m) {
                                    xc[m] = d[m] * Uc;
                                    xs[m] = d[m] * Us;
                                }
                            }
                            if (aft) {
#pragma unroll
                                for (int t = 0; t < SMC; ++t) {
                                    if (SMC > 1 && (t < t0 || t >= t1)) continue;
                                    factors(1 + t, b, d);
#pragma unroll
                                    for (int m = 0; m < 4; ++m) {
                                        xc[m] = fma(d[m], P[2 * t], xc[m]);
                                        xs[m] = fma(d[m], P[2 * t + 1], xs[m]);
                                    }
                                }
                            }
                            uint32_t pc[4], ps[4];
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                pc[m] = i8_digits(xc[m]);
                                ps[m] = i8_digits(xs[m]);
                            }
                            put(b, s, pc, ps);
                        }
                    }
                };
                quiet(0, min(b_ev, NB), false);
                quiet(b_aft, NB, true);
                continue;
            }
            const int g = turn < n_seg ? turn : 2 * n_seg - turn;  // then from the last: it is still held
            double* w = bins + (size_t)(g % A.keep) * NQ * kSeg;
            const bool kept = turn > n_seg && g >= n_seg - A.keep;  // its values are still in its bins
            if (!kept) form(g, w);
            for (int s = 0; s < A.S; ++s) {
                double xc[4], xs[4];
                double2* e = reinterpret_cast<double2*>(w + (2 + 2 * s * A.M) * kSeg + at4);
                double2* f = e + kSeg / 2;
                if (kept) {
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        xc[2 * m] = e[8 * m].x;
                        xc[2 * m + 1] = e[8 * m].y;
                        xs[2 * m] = f[8 * m].x;
                        xs[2 * m + 1] = f[8 * m].y;
                    }
                } else {
                    seg_values(g, w, s, xc, xs);
                }
                if (turn < n_seg) {
#pragma unroll
                    for (int m = 0; m < 4; ++m) vmax = fmax(vmax, fmax(fabs(xc[m]), fabs(xs[m])));
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        e[8 * m] = make_double2(xc[2 * m], xc[2 * m + 1]);
                        f[8 * m] = make_double2(xs[2 * m], xs[2 * m + 1]);
                    }
                } else {
                    uint32_t pc[4], ps[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        pc[m] = i8_digits(xc[m] * inv);
                        ps[m] = i8_digits(xs[m] * inv);
                    }
                    const int b = b_ev + g * kSegBlocks;
                    if (b + (lane >> 3) < NB) put(b, s, pc, ps);
                }
            }
            __syncwarp();
        }
    } else {
        for (int g = 0; g < n_seg; ++g) {
            form(g, bins);
            for (int s = 0; s < A.S; ++s) {
                double xc[4], xs[4];
                seg_values(g, bins, s, xc, xs);
                Real* o = beta + (((size_t)frame * A.n_cos + i) * A.cols_pad + col + 2 * s) * A.t_pad;
                const int k = ((b_ev + g * kSegBlocks) << 5) + 4 * lane;
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (k + m < A.t_pad) {
                        o[k + m] = (Real)xc[m];
                        o[A.t_pad + k + m] = (Real)xs[m];
                    }
            }
            __syncwarp();
        }
        auto quiet = [&](int b_lo, int b_hi, bool aft) {
            const double* U = s_const + (aft ? 2 : 0);
            for (int b = b_lo; b < b_hi; b += kSegBlocks) {
                if (b + (lane >> 3) >= b_hi) continue;
                for (int s = 0; s < A.S; ++s) {
                    const int t0 = s * A.M, t1 = t0 + A.M;
                    double xc[4], xs[4], d[4];
                    factors(0, b, d);
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        xc[m] = d[m] * U[0];
                        xs[m] = d[m] * U[1];
                    }
                    if (aft) {
#pragma unroll
                        for (int t = 0; t < SMC; ++t) {
                            if (SMC > 1 && (t < t0 || t >= t1)) continue;
                            factors(1 + t, b, d);
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                xc[m] = fma(d[m], s_const[4 + 2 * t], xc[m]);
                                xs[m] = fma(d[m], s_const[5 + 2 * t], xs[m]);
                            }
                        }
                    }
                    Real* o = beta + (((size_t)frame * A.n_cos + i) * A.cols_pad + col + 2 * s) * A.t_pad;
                    const int k = (b << 5) + 4 * lane;
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (k + m < A.t_pad) {
                            o[k + m] = (Real)(rf * xc[m]);
                            o[A.t_pad + k + m] = (Real)(rf * xs[m]);
                        }
                }
            }
        };
        quiet(0, min(b_ev, NB), false);
        quiet(b_aft, NB, true);
    }
    };
    auto fetch = [&](long r, double* dst) {  // a row's delays, all in flight at once
        if (r < A.n_rows) {
            const double* src = A.tau + (size_t)r * A.n_phi;
            for (int j = lane; j < A.n_phi; j += 32) copy8_async(dst + j / c_pat * pitch + j % c_pat, src + j);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const long row0 = (long)blockIdx.x * (blockDim.x >> 5) + warp;
    const long n_warps = (long)gridDim.x * (blockDim.x >> 5);
    fetch(row0, s_tau);
    double* s_next = s_tau + (kLoop ? 32 * pitch : 0);
    __syncthreads();
    for (long row = row0; row < A.n_rows; row += n_warps) {
    if constexpr (kLoop) {
        fetch(row + n_warps, s_next);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncwarp();
    beta_row(row, s_tau);
    if constexpr (!kLoop) break;
    double* t = s_tau;
    s_tau = s_next;
    s_next = t;
    __syncwarp();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <class Real, int SMC>
static void launch_beta_smc(const BetaArgs& B, Real* out, size_t smem, int n_sm, int warps, cudaStream_t st) {
    allow_shared(k_beta<Real, SMC>, kBetaShared);
    // three blocks per SM need the largest shared-memory carveout; without the preference the
    // driver may pick a smaller one (two blocks per SM) depending on the kernels run before
    CUDA_OK(cudaFuncSetAttribute(k_beta<Real, SMC>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared));
    const long blocks = (B.n_rows + warps - 1) / warps;
    if (blocks > 0x7fffffffL) throw Error{"too many (bubble, row) pairs for one launch"};
    int per_sm = 1;
    if (SMC > 1) CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_beta<Real, SMC>, 32 * warps, smem));
    const long grid = SMC > 1 ? std::min(blocks, (long)n_sm * std::max(1, per_sm)) : blocks;
    k_beta<Real, SMC><<<(unsigned)grid, 32 * warps, smem, st>>>(B, out);
}

template <class Real>
static void launch_beta(int SM, const BetaArgs& B, Real* out, size_t smem, int n_sm, int warps,
                        cudaStream_t st) {
    switch (SM) {
        case 1: launch_beta_smc<Real, 1>(B, out, smem, n_sm, warps, st); break;
        case 2: launch_beta_smc<Real, 2>(B, out, smem, n_sm, warps, st); break;
        case 3: launch_beta_smc<Real, 3>(B, out, smem, n_sm, warps, st); break;
        case 4: launch_beta_smc<Real, 4>(B, out, smem, n_sm, warps, st); break;
        case 5: launch_beta_smc<Real, 5>(B, out, smem, n_sm, warps, st); break;
        case 6: launch_beta_smc<Real, 6>(B, out, smem, n_sm, warps, st); break;
        case 7: launch_beta_smc<Real, 7>(B, out, smem, n_sm, warps, st); break;
        case 8: launch_beta_smc<Real, 8>(B, out, smem, n_sm, warps, st); break;
        default: throw Error{"at most 8 (set, term) pairs in the factored kernels"};
    }
}

// The int8 digits of a forward call whose masks are kept for the adjoint, with every sum in the order in
// which the events are sorted: by block of 32 steps, then by step, then by patch.  The mixed adjoint's FP32
// products turn a change of the spectrum in its last bits into one of 1e-8 in the gradients (measured with
// k_beta's order: 1.8e-8 on 256 bubbles, 32 k-hat), so its forward keeps this order although k_beta takes
// 3.5 ms where this kernel takes 4.4.
template <int SMC>
__global__ void __launch_bounds__(256, 3) k_beta_sorted(BetaArgs A, int8_t* __restrict__ beta) {
    extern __shared__ __align__(16) unsigned char sm_b[];
    constexpr int NQ = 2 + 2 * SMC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= A.n_rows) return;
    const int NB = A.nblk;
    const int EV = A.n_phi;  // event capacity: one event per patch at most
    unsigned char* base = sm_b + (size_t)warp * A.per_warp_bytes;
    double* evq = reinterpret_cast<double*>(base);             // [NQ][n_phi]: weight q of event e at q * n_phi + e
    double* btot = evq + (size_t)A.n_phi * NQ;                  // [NQ][NB] block totals
    double* uend = btot + (size_t)NQ * NB;                      // [NB][2] uncollided after block
    double* pbeg = uend + 2 * NB;                               // [NB][2 SMC] collided before block
    int* boff = reinterpret_cast<int*>(pbeg + (size_t)2 * SMC * NB);  // [NB+1]
    int* brun = boff + NB + 1;                                  // [NB]
    uint8_t* evs = reinterpret_cast<uint8_t*>(brun + NB);       // [n_phi + 4] step of each event within its block
    // a crowded event block's per-step counts and running offsets [2][32], and its events in step order [n_phi]
    int* scnt = reinterpret_cast<int*>(evs + ((A.n_phi + 4 + 3) & ~3));
    uint16_t* sperm = reinterpret_cast<uint16_t*>(scnt + 64);
    const int slot = (int)((row / A.n_cos) % A.n_sel);
    if (A.sel[slot] == kNoSlot) return;  // a padding slot of a batched job: its columns are never read
    const int i = (int)(row % A.n_cos);
    const long frame = row / ((long)A.n_cos * A.n_sel);
    const double* trow = A.tau + (size_t)row * A.n_phi;
    // The delays of patches j = lane + 32 jj, jj < kMaxJ, are loaded first, all at once (one
    // memory latency for the row), and kept for both passes over the patches.
    constexpr int kMaxJ = 6;
    double tj_c[kMaxJ];
#pragma unroll
    for (int jj = 0; jj < kMaxJ; ++jj) {
        const int j = 32 * jj + lane;
        tj_c[jj] = j < A.n_phi ? __ldcs(trow + j) : 0.0;
    }
    const double ta = A.bub[A.sel[slot]].t;
    const unsigned full = 0xffffffffu;
    const double inv_dt = 1.0 / A.dt;  // the estimate below is only a starting point
    auto block_of = [&](int j, double tj, int& kj) -> int {
        kj = A.n_t;
        if (j >= A.n_phi) return -2;  // not a patch
        if (!(tj > 0.0)) return -1;    // never collides
        // first k with (t_k - t_a) >= tau_j: arithmetic estimate, then exact
        // comparisons (the predicate is monotone in k) settle the boundary
        const double est = ceil((ta + tj - A.t_arr[0]) * inv_dt);
        int lo = est < 0.0 ? 0 : (est > (double)A.n_t ? A.n_t : (int)est);
        while (lo > 0 && A.t_arr[lo - 1] - ta >= tj) --lo;
        while (lo < A.n_t && !(A.t_arr[lo] - ta >= tj)) ++lo;
        kj = lo;
        return lo < A.n_t ? lo >> 5 : -1;
    };
    for (int b = lane; b < NB; b += 32) boff[b] = 0;
    __syncwarp();
    // pass 1: events per block; never-colliding weights (lane sums, fixed-order reduction).
    // The first collided step of patches j = lane + 32 jj, jj < kMaxJ, is kept for pass 2.
    int kj_c[kMaxJ], b_c[kMaxJ];
    double nc = 0.0, ns = 0.0;
    auto pass1 = [&](int j, int b) {
        if (b == -1) {
            const double wj = (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0;
            nc += wj * A.cos2[j];
            ns += wj * A.sin2[j];
        }
        const unsigned m = __match_any_sync(full, b);
        if (b >= 0 && lane == __ffs(m) - 1) boff[b] += __popc(m);
        __syncwarp();
    };
#pragma unroll
    for (int jj = 0; jj < kMaxJ; ++jj) {
        if (32 * jj >= A.n_phi) break;
        const int j = 32 * jj + lane;
        kj_c[jj] = 0;
        b_c[jj] = block_of(j, tj_c[jj], kj_c[jj]);
        pass1(j, b_c[jj]);
    }
    for (int j0 = 32 * kMaxJ; j0 < A.n_phi; j0 += 32) {
        int kj;
        const int j = j0 + lane;
        const int b = block_of(j, j < A.n_phi ? trow[j] : 0.0, kj);
        pass1(j, b);
    }
    for (int o = 16; o > 0; o >>= 1) {
        nc += __shfl_down_sync(full, nc, o);
        ns += __shfl_down_sync(full, ns, o);
    }
    // block counts -> first event of each block: an exclusive warp scan over 32 blocks at a time
    {
        int carry = 0;
        for (int bc = 0; bc < NB; bc += 32) {
            const int b = bc + lane;
            const int c = b < NB ? boff[b] : 0;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(full, incl, o);
                if (lane >= o) incl += t;
            }
            if (b < NB) {
                boff[b] = carry + incl - c;
                brun[b] = carry + incl - c;
            }
            carry += __shfl_sync(full, incl, 31);
        }
        __syncwarp();
        if (lane == 0) boff[NB] = carry;
    }
    __syncwarp();
    // pass 2: scatter events (stable in j within a block)
    const unsigned lt = (1u << lane) - 1u;
    auto pass2 = [&](int j, double tj, int kj, int b) {
        const unsigned m = __match_any_sync(full, b);
        int pos = 0;
        if (b >= 0) pos = brun[b] + __popc(m & lt);
        __syncwarp();
        if (b >= 0 && lane == __ffs(m) - 1) brun[b] += __popc(m);
        __syncwarp();
        if (b >= 0) {
            evs[pos] = (uint8_t)(kj & 31);
            const double wj = (j == 0 || j == A.n_phi - 1) ? 0.5 : 1.0;
            const double qc = wj * A.cos2[j], qs = wj * A.sin2[j];
            double* q = evq + pos;
            q[0] = qc;
            q[EV] = qs;
            const double ed = A.has_damp ? exp(tj / A.damp) : 1.0;
#pragma unroll
            for (int t = 0; t < SMC; ++t) {
                const double f = tpow(tj, A.powers[t]) * ed;
                q[(2 + 2 * t) * EV] = qc * f;
                q[(3 + 2 * t) * EV] = qs * f;
            }
        }
    };
#pragma unroll
    for (int jj = 0; jj < kMaxJ; ++jj) {
        if (32 * jj >= A.n_phi) break;
        pass2(32 * jj + lane, tj_c[jj], kj_c[jj], b_c[jj]);
    }
    for (int j0 = 32 * kMaxJ; j0 < A.n_phi; j0 += 32) {
        int kj;
        const int j = j0 + lane;
        const double tj = j < A.n_phi ? trow[j] : 0.0;
        const int b = block_of(j, tj, kj);
        pass2(j, tj, kj, b);
    }
    __syncwarp();
    // block totals of every weight: the lanes take a block's events in strides
    // of 32 and a butterfly reduction adds the lane sums (a fixed order for a
    // given event count); then the collided sums before each block (exclusive
    // prefix over blocks) and the uncollided sums after each block (exclusive
    // suffix plus the never-colliding weights), as warp scans over lanes = blocks
    for (int b = lane; b < NB; b += 32)
        if (boff[b] == boff[b + 1]) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) btot[(size_t)q * NB + b] = 0.0;
        }
    for (int bc = 0; bc < NB; bc += 32) {
        const int bl = bc + lane;
        for (unsigned h = __ballot_sync(full, bl < NB && boff[bl] != boff[bl + 1]); h; h &= h - 1) {
            const int b = bc + __ffs(h) - 1;
            double t[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) t[q] = 0.0;
            for (int e = boff[b] + lane; e < boff[b + 1]; e += 32) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) t[q] += evq[(size_t)q * EV + e];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) t[q] += __shfl_xor_sync(full, t[q], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) btot[(size_t)q * NB + b] = t[q];
            }
        }
    }
    __syncwarp();
    {
        double carry[2 * SMC];
#pragma unroll
        for (int q = 0; q < 2 * SMC; ++q) carry[q] = 0.0;
        for (int bc = 0; bc < NB; bc += 32) {
            const int b = bc + lane;
            double v[2 * SMC];
#pragma unroll
            for (int q = 0; q < 2 * SMC; ++q) v[q] = b < NB ? btot[(size_t)(2 + q) * NB + b] : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                for (int q = 0; q < 2 * SMC; ++q) {
                    const double u = __shfl_up_sync(full, v[q], o);
                    if (lane >= o) v[q] += u;
                }
            }
#pragma unroll
            for (int q = 0; q < 2 * SMC; ++q) {
                double ex = __shfl_up_sync(full, v[q], 1);
                if (lane == 0) ex = 0.0;
                if (b < NB) pbeg[(size_t)b * 2 * SMC + q] = carry[q] + ex;
                carry[q] += __shfl_sync(full, v[q], 31);
            }
        }
        // the never-colliding sums were reduced into lane 0
        double cc = __shfl_sync(full, nc, 0), cs = __shfl_sync(full, ns, 0);
        for (int bc = ((NB - 1) >> 5) << 5; bc >= 0; bc -= 32) {
            const int b = bc + lane;
            double vc = b < NB ? btot[b] : 0.0, vs = b < NB ? btot[(size_t)NB + b] : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double uc = __shfl_down_sync(full, vc, o), us = __shfl_down_sync(full, vs, o);
                if (lane + o < 32) {
                    vc += uc;
                    vs += us;
                }
            }
            double xc = __shfl_down_sync(full, vc, 1), xs = __shfl_down_sync(full, vs, 1);
            if (lane == 31) xc = xs = 0.0;
            if (b < NB) {
                uend[2 * b] = cc + xc;
                uend[2 * b + 1] = cs + xs;
            }
            cc += __shfl_sync(full, vc, 0);
            cs += __shfl_sync(full, vs, 0);
        }
    }
    __syncwarp();
    // pass 3.  Blocks holding events ("event blocks") are formed one at a time
    // with lane = step: each lane sums the events at its own step (their block
    // offsets are compared four at a time as bytes), then warp scans give the
    // collided sums up to and the uncollided sums after every step.  Blocks
    // without events have constant sums: each lane forms 4 consecutive steps,
    // 8 lanes a block, 4 such blocks at a time.  The digits need the row's
    // scale, max |beta| over its steps and columns, first.
    const double ci = A.cos_t[i];
    const double vi = (i == 0 || i == A.n_cos - 1) ? 0.5 : 1.0;
    const double rf = (0.5 * (1.0 - ci * ci) * A.dphi) * (A.dcos * vi) * A.dt * (1.0 / (6.0 * CUDART_PI));
    const double* Dslot = A.D + (size_t)slot * (1 + SMC) * A.tf;
    const int nbase = (slot % A.bpt) * 2 * A.S;
    int8_t* blk_row = beta + (((size_t)frame * A.n_cos + i) * A.tiles + slot / A.bpt) * (size_t)NB * kI8BlockSet;
    // beta of coefficient set s at step k from the sums there: the table row
    // holds the step weight times dt^3 and times a_m dt^{3-p_m} e^{-dt/w}
    auto value = [&](int k, int s, const double* P, double Uc, double Us, double mul, double& xc, double& xs) {
        double g[1 + SMC];
#pragma unroll
        for (int q = 0; q < 1 + SMC; ++q) g[q] = __ldg(Dslot + (size_t)q * A.tf + step_at(min(k, A.n_t - 1)));
        double vc = g[0] * Uc, vs = g[0] * Us;
        const int t0 = s * A.M, t1 = t0 + A.M;  // the terms of set s
#pragma unroll
        for (int t = 0; t < SMC; ++t) {
            if (t < t0 || t >= t1) continue;
            vc += g[1 + t] * P[2 * t];
            vs += g[1 + t] * P[2 * t + 1];
        }
        const double r = k < A.n_t ? mul : 0.0;
        xc = r * vc;
        xs = r * vs;
    };
    // Collided sums through step (b << 5) + lane and uncollided sums after it, for
    // block b, lane = step (the whole warp calls it with the same b).
    auto step_sums = [&](int b, double (&P)[2 * SMC], double& Uc, double& Us) {
        const int e0 = boff[b], e1 = boff[b + 1];
        if (e0 == e1) {  // a block without events: constant sums
#pragma unroll
            for (int q = 0; q < 2 * SMC; ++q) P[q] = pbeg[(size_t)b * 2 * SMC + q];
            Uc = uend[2 * b];
            Us = uend[2 * b + 1];
            return;
        }
        double dq[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) dq[q] = 0.0;
        if (e1 - e0 > 32) {
            // Many events: the block's events are counting-sorted by their step (stable in event
            // order; ranks within 32 events from __match_any groups), then each lane adds the
            // events of its own step in event order.
            int* run = scnt + 32;
            scnt[lane] = 0;
            __syncwarp();
            for (int r0 = e0; r0 < e1; r0 += 32) {
                const int e = r0 + lane;
                const int se = e < e1 ? (int)evs[e] : 32 + lane;
                const unsigned m = __match_any_sync(full, se);
                if (e < e1 && lane == __ffs(m) - 1) scnt[se] += __popc(m);
                __syncwarp();
            }
            const int c = scnt[lane];
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(full, incl, o);
                if (lane >= o) incl += t;
            }
            const int ex = incl - c;  // first position of this lane's step
            run[lane] = ex;
            __syncwarp();
            const unsigned lt = (1u << lane) - 1u;
            for (int r0 = e0; r0 < e1; r0 += 32) {
                const int e = r0 + lane;
                const bool v = e < e1;
                const int se = v ? (int)evs[e] : 32 + lane;
                const unsigned m = __match_any_sync(full, se);
                if (v) sperm[run[se] + __popc(m & lt)] = (uint16_t)e;
                __syncwarp();
                if (v && lane == __ffs(m) - 1) run[se] += __popc(m);
                __syncwarp();
            }
            for (int r = 0; r < c; ++r) {
                const double* qe = evq + sperm[ex + r];
#pragma unroll
                for (int q = 0; q < NQ; ++q) dq[q] += qe[(size_t)q * EV];
            }
            __syncwarp();
        } else {
            const uint32_t pat = 0x01010101u * (uint32_t)lane;
            for (int e4 = e0 & ~3; e4 < e1; e4 += 4) {
                uint32_t eq = __vcmpeq4(*reinterpret_cast<const uint32_t*>(evs + e4), pat);
                if (e4 < e0) eq &= 0xffffffffu << (8 * (e0 - e4));
                if (e1 - e4 < 4) eq &= (1u << (8 * (e1 - e4))) - 1u;
                while (eq) {
                    const int by = (__ffs(eq) - 1) >> 3;
                    eq &= ~(0xffu << (8 * by));
                    const double* qe = evq + (e4 + by);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) dq[q] += qe[(size_t)q * EV];
                }
            }
        }
        // collided sums through this step (inclusive scan), uncollided after it (suffix scan)
        double uc = dq[0], us = dq[1];
#pragma unroll
        for (int q = 0; q < 2 * SMC; ++q) P[q] = dq[2 + q];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int q = 0; q < 2 * SMC; ++q) {
                const double v = __shfl_up_sync(full, P[q], o);
                if (lane >= o) P[q] += v;
            }
            const double vc = __shfl_down_sync(full, uc, o), vs = __shfl_down_sync(full, us, o);
            if (lane + o < 32) {
                uc += vc;
                us += vs;
            }
        }
        // uncollided after this step: the next step's inclusive suffix sum
        Uc = __shfl_down_sync(full, uc, 1);
        Us = __shfl_down_sync(full, us, 1);
        if (lane == 31) Uc = Us = 0.0;
        Uc += uend[2 * b];
        Us += uend[2 * b + 1];
#pragma unroll
        for (int q = 0; q < 2 * SMC; ++q) P[q] = pbeg[(size_t)b * 2 * SMC + q] + P[q];
    };
    // The row's scale is max |beta| over its steps and columns, found exactly without
    // forming every value.
    // (a) Every event block is formed once (lane = step) and its 2S values are kept for the
    //     digits: a block of at least 32 events in its own weight slots (plane 2s + g, slots
    //     boff[b] + lane; its weights are not read again), smaller blocks in the block-total
    //     table while it has room (the rest are formed again in (c)).
    // (b) In a block without events U and Pm are constant, so beta = rf (D0(k) U + sum_m Dm(k)
    //     Pm) is bounded by interval arithmetic over the per-block ranges of the time table;
    //     such blocks are formed (lane = step) in decreasing order of their bound until no
    //     bound exceeds the largest value found (most often one block: the last one, where
    //     dt^3 peaks).
    // (c) Digits of every block.
    double vmax = 0.0;
    const double* Dmx = A.Dmax + (size_t)slot * NB * (1 + SMC) * 2;
    int* where = brun;  // per event block: -1 not kept, -2 own slots, c >= 0 table slot c
    const int n_tab = (NQ * NB) / (64 * A.S);
    int used_tab = 0;
    auto kept = [&](int b, int& stride) -> double* {
        const int w = where[b];
        if (w == -2) {
            stride = EV;
            return evq + boff[b];
        }
        stride = 32;
        return w >= 0 ? btot + (size_t)w * 64 * A.S : nullptr;
    };
    for (int bc = 0; bc < NB; bc += 32) {
        const int bl = bc + lane;
        for (unsigned h = __ballot_sync(full, bl < NB && boff[bl] != boff[bl + 1]); h; h &= h - 1) {
            const int b = bc + __ffs(h) - 1;
            double P[2 * SMC], Uc, Us;
            step_sums(b, P, Uc, Us);
            const int k = (b << 5) + lane;
            const int code = boff[b + 1] - boff[b] >= 32 ? -2 : (used_tab < n_tab ? used_tab++ : -1);
            __syncwarp();
            if (lane == 0) where[b] = code;
            __syncwarp();
            int stride = 0;
            double* dst = kept(b, stride);
            for (int s2 = 0; s2 < A.S; ++s2) {
                double xc, xs;
                value(k, s2, P, Uc, Us, rf, xc, xs);
                vmax = fmax(vmax, fmax(fabs(xc), fabs(xs)));
                if (dst) {
                    dst[(size_t)(2 * s2) * stride + lane] = xc;
                    dst[(size_t)(2 * s2 + 1) * stride + lane] = xs;
                }
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(full, vmax, o));
    for (int bc = 0; bc < NB; bc += 32) {
        const int bl = bc + lane;
        double bnd = -1.0;  // this lane's block's bound (-1: none or an event block)
        if (bl < NB && boff[bl] == boff[bl + 1]) {
            // beta of set s, column g lies in rf (D0 [U] + sum_m Dm [Pm]) with D in [min, max]
            // over the block and U, Pm the block's constants
            const double* mx = Dmx + (size_t)bl * (1 + SMC) * 2;
            auto term = [&](double dlo, double dhi, double c, double& lo, double& hi, double& sa) {
                const double p0 = dlo * c, p1 = dhi * c;
                lo += fmin(p0, p1);
                hi += fmax(p0, p1);
                sa += fmax(fabs(dlo), fabs(dhi)) * fabs(c);
            };
            for (int s2 = 0; s2 < A.S; ++s2) {
                const int t0 = s2 * A.M, t1 = t0 + A.M;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    double lo = 0.0, hi = 0.0, sa = 0.0;
                    term(mx[0], mx[1], uend[2 * bl + g], lo, hi, sa);
#pragma unroll
                    for (int q = 0; q < SMC; ++q)
                        if (q >= t0 && q < t1)
                            term(mx[2 + 2 * q], mx[3 + 2 * q], pbeg[(size_t)bl * 2 * SMC + 2 * q + g], lo, hi, sa);
                    // relative and absolute margins cover the rounding of these sums and of
                    // the values themselves (a few ulp of the summed magnitudes)
                    bnd = fmax(bnd, (fmax(fabs(lo), fabs(hi)) * (1.0 + 1e-12) + 1e-13 * sa) * rf);
                }
            }
        }
        for (;;) {
            double bb = bnd;
            int bi = lane;
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(full, bb, o);
                const int oi = __shfl_xor_sync(full, bi, o);
                if (ob > bb || (ob == bb && oi < bi)) {
                    bb = ob;
                    bi = oi;
                }
            }
            // Every remaining bound is covered once no bound exceeds vmax (1 + 1e-10): a value up
            // to that much above the scale still maps to |x F| <= F + 0.22, which rounds into the
            // digit range.  (Without the slack, blocks whose values all equal the maximum, as after
            // the last collision with powers = 3, would each be formed.)
            if (!(bb > vmax * (1.0 + 1e-10))) break;
            {
                const int b = bc + bi, k = (b << 5) + lane;
                const double* P = pbeg + (size_t)b * 2 * SMC;
                const double Uc = uend[2 * b], Us = uend[2 * b + 1];
                double m = 0.0;
                for (int s2 = 0; s2 < A.S; ++s2) {
                    double xc, xs;
                    value(k, s2, P, Uc, Us, rf, xc, xs);
                    m = fmax(m, fmax(fabs(xc), fabs(xs)));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(full, m, o));
                vmax = fmax(vmax, m);
            }
            if (lane == bi) bnd = -1.0;
        }
    }
    if (lane == 0) A.scale[row] = vmax;
    const double inv = vmax > 0.0 ? 1.0 / vmax : 0.0;
    const double rinv = rf * inv;
    // digits (streaming stores: the GEMM reads them back from DRAM).  Event blocks: lane = step; a
    // quad of lanes transposes its packed digit
    // words so that lane 4q + d holds digit d of steps 4q .. 4q + 3.  Blocks without
    // events: 4 steps per lane (8 lanes a block, 4 blocks at a time), transposed in
    // registers.  Either way a store instruction fills whole 32-byte rows of the blocks.
    const bool odd = lane & 1, hi = lane & 2;
    auto quad_transpose = [&](uint32_t p) {
        const uint32_t t1 = __shfl_xor_sync(full, p, 1);
        p = __byte_perm(p, t1, odd ? 0x3715 : 0x6240);
        const uint32_t t2 = __shfl_xor_sync(full, p, 2);
        return __byte_perm(p, t2, hi ? 0x3276 : 0x5410);
    };
    const int dg = lane & 3, s4 = (lane >> 2) * 4;
    for (int bc = 0; bc < NB; bc += 32) {
        const int bl = bc + lane;
        const bool has = bl < NB && boff[bl] != boff[bl + 1];
        const unsigned ev_blocks = __ballot_sync(full, has);
        unsigned quiet = __ballot_sync(full, bl < NB && !has);
        for (unsigned h = ev_blocks; h; h &= h - 1) {
            const int b = bc + __ffs(h) - 1;
            const int k = (b << 5) + lane;
            int stride = 0;
            const double* src = kept(b, stride);
            double P[2 * SMC], Uc = 0.0, Us = 0.0;
            if (!src) step_sums(b, P, Uc, Us);
            int8_t* blk = blk_row + (size_t)b * kI8BlockSet + dg * kI8Block;
            for (int s2 = 0; s2 < A.S; ++s2) {
                double xc, xs;
                if (src) {
                    xc = src[(size_t)(2 * s2) * stride + lane];
                    xs = src[(size_t)(2 * s2 + 1) * stride + lane];
                } else {
                    value(k, s2, P, Uc, Us, rf, xc, xs);
                }
                const uint32_t wc = quad_transpose(i8_digits(xc * inv));
                const uint32_t ws = quad_transpose(i8_digits(xs * inv));
                __stcs(reinterpret_cast<unsigned int*>(blk + i8_swz(nbase + 2 * s2, s4)), wc);
                __stcs(reinterpret_cast<unsigned int*>(blk + i8_swz(nbase + 2 * s2 + 1, s4)), ws);
            }
        }
        const int sub = lane >> 3, s0 = (lane & 7) * 4;
        while (quiet) {
            unsigned t = quiet;
            for (int g = 0; g < sub && t; ++g) t &= t - 1;
            const int b = t ? bc + __ffs(t) - 1 : -1;
            for (int g = 0; g < 4 && quiet; ++g) quiet &= quiet - 1;
            if (b < 0) continue;
            const int k0 = (b << 5) + s0;
            // the block's constant sums, with rf / scale folded in: 1 + SMC products per
            // value (steps past n_t, in the last block only, go through value())
            const bool tail = k0 + 4 > A.n_t;
            double P[2 * SMC];
#pragma unroll
            for (int q = 0; q < 2 * SMC; ++q) P[q] = rinv * pbeg[(size_t)b * 2 * SMC + q];
            const double Uc = rinv * uend[2 * b], Us = rinv * uend[2 * b + 1];
            const double* Db = Dslot + step_at(k0);
            int8_t* blk = blk_row + (size_t)b * kI8BlockSet;
            for (int s2 = 0; s2 < A.S; ++s2) {
                uint32_t pc[4], ps[4];
                const int t0 = s2 * A.M, t1 = t0 + A.M;  // the terms of set s2
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    double xc, xs;
                    if (tail) {
                        value(k0 + m, s2, P, Uc, Us, 1.0, xc, xs);
                    } else {
                        double g[1 + SMC];
#pragma unroll
                        for (int q = 0; q < 1 + SMC; ++q) g[q] = __ldg(Db + (size_t)q * A.tf + (m & 1) + 8 * (m & 2));
                        xc = g[0] * Uc;
                        xs = g[0] * Us;
#pragma unroll
                        for (int q = 0; q < SMC; ++q) {
                            if (SMC > 1 && (q < t0 || q >= t1)) continue;
                            xc = fma(g[1 + q], P[2 * q], xc);
                            xs = fma(g[1 + q], P[2 * q + 1], xs);
                        }
                    }
                    pc[m] = i8_digits(xc);
                    ps[m] = i8_digits(xs);
                }
                uint32_t wc[4], ws[4];
                i8_transpose4(pc[0], pc[1], pc[2], pc[3], wc);
                i8_transpose4(ps[0], ps[1], ps[2], ps[3], ws);
                const int oc = i8_swz(nbase + 2 * s2, s0), os = i8_swz(nbase + 2 * s2 + 1, s0);
#pragma unroll
                for (int d = 0; d < kI8Slices; ++d) {
                    __stcs(reinterpret_cast<unsigned int*>(blk + d * kI8Block + oc), wc[d]);
                    __stcs(reinterpret_cast<unsigned int*>(blk + d * kI8Block + os), ws[d]);
                }
            }
        }
    }
}

template <int SMC>
static void launch_sorted_smc(BetaArgs& B, int8_t* out, cudaStream_t st) {
    const int NQ = 2 + 2 * SMC, n_phi = B.n_phi;
    size_t pw = (size_t)n_phi * NQ * sizeof(double) + 2 * (size_t)NQ * B.nblk * sizeof(double) +
                (2 * (size_t)B.nblk + 1) * sizeof(int) + (((size_t)n_phi + 4 + 3) & ~(size_t)3) + 64 * sizeof(int) +
                (size_t)n_phi * sizeof(uint16_t);
    pw = (pw + 15) & ~(size_t)15;
    B.per_warp_bytes = (int)pw;
    constexpr size_t most = 200 * 1024;
    const int warps = (int)std::min<size_t>(8, most / pw);
    if (warps < 1) throw Error{"n_phi too large for the beta kernel"};
    const size_t smem = (size_t)warps * pw;
    allow_shared(k_beta_sorted<SMC>, most);
    CUDA_OK(cudaFuncSetAttribute(k_beta_sorted<SMC>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared));
    k_beta_sorted<SMC><<<(unsigned)((B.n_rows + warps - 1) / warps), warps * 32, smem, st>>>(B, out);
}

static void launch_sorted(int SM, BetaArgs& B, int8_t* out, cudaStream_t st) {
    switch (SM) {
        case 1: return launch_sorted_smc<1>(B, out, st);
        case 2: return launch_sorted_smc<2>(B, out, st);
        case 3: return launch_sorted_smc<3>(B, out, st);
        case 4: return launch_sorted_smc<4>(B, out, st);
        case 5: return launch_sorted_smc<5>(B, out, st);
        case 6: return launch_sorted_smc<6>(B, out, st);
        case 7: return launch_sorted_smc<7>(B, out, st);
        default: return launch_sorted_smc<8>(B, out, st);
    }
}

// ---------------------------------------------------------------------------
struct FactArgs {
    const D4* bub;  // rotated frames (kn, n_tot)
    size_t n_tot;
    const uint32_t* sel;
    int n_sel;
    int n_cos, n_t, n_w;
    int S;
    const double* t_arr;
    const double* w;
    const double* cos_t;
    const int* kfirst;     // (n_sel)
    const void* beta;      // (kn, n_cos, cols_pad, t_pad) Real
    long cols_pad;
    int t_pad;
    double dt;
    int bpt;               // bubbles per column tile
    int tiles_per_frame;
    double2* partial;      // (kn, tiles_per_frame, 2, S, W)
};

// One CTA per (64-frequency tile, column tile), looping over the rows i.
// Thread (ty, tx) of 16 x 16 owns rows ty*8 .. ty*8+7 (frequencies ty*4 .. +3,
// Re/Im interleaved) and TN columns in two groups of TN/2: tx*TN/2 + u and
// COLS/2 + tx*TN/2 + u, so that consecutive threads read consecutive 16-byte
// words of a beta-tile row (no shared-memory bank conflicts).
template <int TN, int COLS>
__device__ __forceinline__ int thread_col(int tx, int u) {
    return u < TN / 2 ? tx * (TN / 2) + u : COLS / 2 + tx * (TN / 2) + (u - TN / 2);
}

constexpr int kGemmTN = 8, kGemmCols = 16 * kGemmTN, kGemmBS = kGemmCols + 4;  // (padded row of the beta tile)

__global__ void __launch_bounds__(kThreads, 1) k_gemm(FactArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int TN = kGemmTN, COLS = kGemmCols, BS = kGemmBS;
    constexpr int VEC = 4;                                         // elements per 16-byte load
    constexpr int NPRE = COLS * kKC / VEC / kThreads;              // 16-byte loads per thread per tile
    float* Msm = reinterpret_cast<float*>(smem);                   // [kKC][kRows]
    float* Bsm = Msm + kKC * kRows;                                // [kKC][BS]
    double* Pn_re = reinterpret_cast<double*>(Bsm + kKC * BS);      // [kKC][kWT]
    double* Pn_im = Pn_re + kKC * kWT;
    double* anc = Pn_im + kKC * kWT;                               // [2][kWT]
    double2* red = reinterpret_cast<double2*>(anc + 2 * kWT);       // [kThreads][4][2S]
    double2* Cacc = red + kThreads * 4 * 2 * A.S;                  // [kWT][2S]
    int* binfo = reinterpret_cast<int*>(Cacc + kWT * 2 * A.S);      // [bpt]: slot or -1
    double* bt = reinterpret_cast<double*>(binfo + 64);            // [bpt] t_a
    double* bz = bt + 64;                                          // [bpt] z_a

    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;
    const int w0 = blockIdx.x * kWT;
    const int frame = blockIdx.y / A.tiles_per_frame;
    const int tile = blockIdx.y % A.tiles_per_frame;
    const int cpb = 2 * A.S;  // columns per bubble
    const D4* B = A.bub + (size_t)frame * A.n_tot;
    const float* beta = static_cast<const float*>(A.beta);

    if (tid < 64) {
        const int slot = tile * A.bpt + tid;
        const bool ok = tid < A.bpt && slot < A.n_sel && A.sel[slot] != kNoSlot;
        binfo[tid] = ok ? slot : -1;
        if (ok) {
            const D4 xa = B[A.sel[slot]];
            bt[tid] = xa.t;
            bz[tid] = xa.z;
        }
    }
    for (int q = tid; q < kWT * cpb; q += kThreads) Cacc[q] = make_double2(0.0, 0.0);
    __syncthreads();
    int kstart = A.n_t;
    for (int b = 0; b < A.bpt; ++b)
        if (binfo[b] >= 0) kstart = min(kstart, A.kfirst[binfo[b]]);
    const int c_start = kstart / kKC;
    const int n_chunks = (A.n_t + kKC - 1) / kKC;
    const long col0 = (long)tile * COLS;

    for (int i = 0; i < A.n_cos; ++i) {
        const double ci = A.cos_t[i];
        const double one_m_c = 1.0 - ci;
        for (int q = tid; q < kKC * kWT; q += kThreads) {
            const int n = q / kWT, wl = q % kWT;
            const int wi = w0 + wl;
            double sn = 0.0, cs = 1.0;
            if (wi < A.n_w) phase<float>(A.w[wi] * one_m_c * (n * A.dt), sn, cs);
            Pn_re[q] = cs;
            Pn_im[q] = sn;
        }
        const float* bi = beta + (((size_t)frame * A.n_cos + i) * A.cols_pad + col0) * A.t_pad;
        // 16-byte loads of the beta tile: column q / (kKC/VEC), steps VEC*(q % (kKC/VEC)) ...
        float4 pre[NPRE];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int v = 0; v < NPRE; ++v) {
                const int q = tid + v * kThreads;
                const int col = q / (kKC / VEC), n = (q % (kKC / VEC)) * VEC;
                const int k = k0 + n;  // t_pad is a multiple of VEC: a load is all in or all out
                if (k < A.t_pad) pre[v] = __ldg(reinterpret_cast<const float4*>(bi + (size_t)col * A.t_pad + k));
                else pre[v] = float4{};
            }
        };
        double acc[kTM][TN];
#pragma unroll
        for (int r = 0; r < kTM; ++r)
#pragma unroll
            for (int u = 0; u < TN; ++u) acc[r][u] = 0.0;
        if (c_start < n_chunks) fetch(c_start * kKC);
        __syncthreads();

        for (int ch = c_start; ch < n_chunks; ++ch) {
            const int k0 = ch * kKC;
            if (tid < kWT) {
                const int wi = w0 + tid;
                double sn = 0.0, cs = 0.0;
                if (wi < A.n_w) phase<float>(A.w[wi] * one_m_c * A.t_arr[k0], sn, cs);
                anc[tid] = cs;
                anc[kWT + tid] = sn;
            }
#pragma unroll
            for (int v = 0; v < NPRE; ++v) {
                const int q = tid + v * kThreads;
                const int col = q / (kKC / VEC), n = (q % (kKC / VEC)) * VEC;
                const float* pv = reinterpret_cast<const float*>(&pre[v]);
#pragma unroll
                for (int e = 0; e < VEC; ++e) Bsm[(n + e) * BS + col] = pv[e];
            }
            __syncthreads();
            for (int q = tid; q < kKC * kWT; q += kThreads) {
                const int n = q / kWT, wl = q % kWT;
                const double ar = anc[wl], ai = anc[kWT + wl];
                const double pr = Pn_re[q], pi = Pn_im[q];
                const bool valid = k0 + n < A.n_t;
                Msm[n * kRows + 2 * wl] = valid ? (float)(ar * pr - ai * pi) : 0.0f;
                Msm[n * kRows + 2 * wl + 1] = valid ? (float)(ar * pi + ai * pr) : 0.0f;
            }
            __syncthreads();
            if (ch + 1 < n_chunks) fetch(k0 + kKC);  // in flight during the GEMM below
#pragma unroll 1
            for (int n0 = 0; n0 < kKC; n0 += kFold) {
                float cacc[kTM][TN];
#pragma unroll
                for (int r = 0; r < kTM; ++r)
#pragma unroll
                    for (int u = 0; u < TN; ++u) cacc[r][u] = 0.0f;
#pragma unroll
                for (int n = n0; n < n0 + kFold; ++n) {
                    float a[kTM], bb[TN];
                    const float4* ap = reinterpret_cast<const float4*>(Msm + n * kRows + ty * kTM);
                    const float4 b0 = *reinterpret_cast<const float4*>(Bsm + n * BS + tx * (TN / 2));
                    const float4 b1 = *reinterpret_cast<const float4*>(Bsm + n * BS + COLS / 2 + tx * (TN / 2));
#pragma unroll
                    for (int r = 0; r < kTM / 4; ++r) {
                        const float4 v = ap[r];
                        a[4 * r] = v.x;
                        a[4 * r + 1] = v.y;
                        a[4 * r + 2] = v.z;
                        a[4 * r + 3] = v.w;
                    }
                    bb[0] = b0.x;
                    bb[1] = b0.y;
                    bb[2] = b0.z;
                    bb[3] = b0.w;
                    bb[4] = b1.x;
                    bb[5] = b1.y;
                    bb[6] = b1.z;
                    bb[7] = b1.w;
#pragma unroll
                    for (int r = 0; r < kTM; ++r)
#pragma unroll
                        for (int u = 0; u < TN; ++u) cacc[r][u] = fmaf(a[r], bb[u], cacc[r][u]);
                }
#pragma unroll
                for (int r = 0; r < kTM; ++r)
#pragma unroll
                    for (int u = 0; u < TN; ++u) acc[r][u] += (double)cacc[r][u];
            }
            __syncthreads();
        }
        // epilogue: per thread, C_{s,g}(w) partials of its columns in fixed order
        // partials in structure-of-arrays order red[(q*cpb + sg)*kThreads + tid]
        for (int q = 0; q < 4 * cpb; ++q) red[(size_t)q * kThreads + tid] = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < kTM / 2; ++q) {
            const int wl = ty * (kTM / 2) + q;
            const int wi = w0 + wl;
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                const int col = thread_col<TN, COLS>(tx, u);
                const int b = col / cpb;
                if (b >= A.bpt || binfo[b] < 0 || wi >= A.n_w) continue;
                double sn, cs;
                phase<float>(A.w[wi] * (bt[b] * ci - bz[b]), sn, cs);
                const double yr = acc[2 * q][u], yi = acc[2 * q + 1][u];
                double2& d = red[(size_t)(q * cpb + (col % cpb)) * kThreads + tid];
                d.x += cs * yr - sn * yi;
                d.y += cs * yi + sn * yr;
            }
        }
        __syncthreads();
        for (int q = tid; q < kWT * cpb; q += kThreads) {
            const int wl = q / cpb, sg = q % cpb;
            const int tyw = wl / (kTM / 2), qq = wl % (kTM / 2);
            double2 sum = Cacc[q];
            for (int t = 0; t < 16; ++t) {
                const double2 v = red[(size_t)(qq * cpb + sg) * kThreads + tyw * 16 + t];
                sum.x += v.x;
                sum.y += v.y;
            }
            Cacc[q] = sum;
        }
        __syncthreads();
    }
    for (int q = tid; q < kWT * cpb; q += kThreads) {
        const int wl = q / cpb, sg = q % cpb;
        const int s = sg >> 1, g = sg & 1;
        const int wi = w0 + wl;
        if (wi >= A.n_w) continue;
        const size_t o = ((((size_t)frame * A.tiles_per_frame + tile) * 2 + g) * A.S + s) * A.n_w + wi;
        A.partial[o] = Cacc[q];
    }
}

// FP64: the same product folded about the middle of the time grid.  Steps hi = h0 + d and lo = l0 - d lie
// symmetrically about t_mid, so with theta_d = w (1 - c_i) (t_hi - t_lo) / 2
//   sum_k e^{i w (1 - c_i) t_k} beta_k = e^{i w (1 - c_i) t_mid} [ sum_d cos theta_d (beta_hi + beta_lo)
//                                                             + i sum_d sin theta_d (beta_hi - beta_lo) ]:
// one real product per (frequency, pair) for each of Re and Im where the plain form has one per step, and
// the middle phase goes into the epilogue's.  What bounds it: FP64 FMAs (half of the plain form's; 9.2 ms
// before, of which 4.1 at the FP64 peak, for 4 frames of 512 bubbles x 128 rows x 512 steps x 128 w).  The
// rows are split over CTAs, 8 rows each at least: a small call had 16 CTAs (1.7 ms for 8 frames of 48
// bubbles).  Now 5.05 ms for the former.  The split depends on the grid alone, so that a realization's sums do not depend on its batch.
constexpr int kFoldTN = 4, kFoldCols = 16 * kFoldTN, kFoldBS = kFoldCols + 2;

struct FoldSmem {  // doubles
    static constexpr int m = 0;                                // [kKC][kRows]
    static constexpr int e = m + kKC * kRows;                  // [kKC][kFoldBS]
    static constexpr int o = e + kKC * kFoldBS;
    static constexpr int p_re = o + kKC * kFoldBS;             // [kKC][kWT]
    static constexpr int p_im = p_re + kKC * kWT;
    static constexpr int anc = p_im + kKC * kWT;               // [2][kWT]
    static constexpr int main = anc + 2 * kWT;
};
static int fold_work(int S) { return std::max(FoldSmem::main, kThreads * 4 * 2 * S * 2); }  // or the epilogue's partials
static size_t fold_smem_bytes(int S) {
    return ((size_t)fold_work(S) + kWT * 2 * S * 2 + 2 * 64) * sizeof(double) + 64 * sizeof(int);
}
static int fold_row_parts(int n_cos) { return std::max(1, std::min(16, n_cos / 8)); }

// e^{i w (t_a c - z_a + (1 - c) t_mid)} with the argument's roundings made good to first order: this phase
// multiplies a whole row, where the plain form's time phases each had a rounding of their own.
__device__ __forceinline__ void middle_phase(double w, double ta, double za, double c, double t_mid, double& s, double& co) {
    const double d = __dsub_rn(1.0, c), ed = __dsub_rn(__dsub_rn(1.0, d), c);
    const double p = __dmul_rn(ta, c), ep = fma(ta, c, -p);
    const double q = __dmul_rn(d, t_mid), eq = fma(d, t_mid, -q);
    // two-sums of p - za and of that + q
    const double u = __dsub_rn(p, za), bu = __dsub_rn(p, u);
    const double eu = __dadd_rn(__dsub_rn(p, __dadd_rn(u, bu)), __dsub_rn(bu, za));
    const double v = __dadd_rn(u, q), bv = __dsub_rn(v, u);
    const double ev = __dadd_rn(__dsub_rn(u, __dsub_rn(v, bv)), __dsub_rn(q, bv));
    const double x = __dmul_rn(w, v);
    const double e = fma(w, ((ep + eq) + (eu + ev)) + ed * t_mid, fma(w, v, -x));
    double sn, cs;
    sincos(x, &sn, &cs);
    s = fma(e, cs, sn);
    co = fma(-e, sn, cs);
}

__global__ void __launch_bounds__(kThreads, 1) k_gemm_fold(FactArgs A, int work) {
    extern __shared__ __align__(16) double fsm[];
    double* Msm = fsm + FoldSmem::m;
    double* Esm = fsm + FoldSmem::e;
    double* Osm = fsm + FoldSmem::o;
    double* Pn_re = fsm + FoldSmem::p_re;
    double* Pn_im = fsm + FoldSmem::p_im;
    double* anc = fsm + FoldSmem::anc;
    double2* red = reinterpret_cast<double2*>(fsm);            // [4 cpb][kThreads], between the rows' products
    double2* Cacc = reinterpret_cast<double2*>(fsm + work);    // [kWT][2S]
    double* bt = fsm + work + kWT * 2 * A.S * 2;               // [64] t_a
    double* bz = bt + 64;                                      // [64] z_a
    int* binfo = reinterpret_cast<int*>(bz + 64);              // [64]: slot or -1
    constexpr int TN = kFoldTN, COLS = kFoldCols, BS = kFoldBS;
    constexpr int NPRE = COLS * kKC / kThreads;

    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;
    const int w0 = blockIdx.x * kWT;
    const int frame = blockIdx.y / A.tiles_per_frame;
    const int tile = blockIdx.y % A.tiles_per_frame;
    const int part = blockIdx.z, parts = gridDim.z;
    const int cpb = 2 * A.S;
    const D4* B = A.bub + (size_t)frame * A.n_tot;
    const double* beta = static_cast<const double*>(A.beta);

    if (tid < 64) {
        const int slot = tile * A.bpt + tid;
        const bool ok = tid < A.bpt && slot < A.n_sel && A.sel[slot] != kNoSlot;
        binfo[tid] = ok ? slot : -1;
        if (ok) {
            const D4 xa = B[A.sel[slot]];
            bt[tid] = xa.t;
            bz[tid] = xa.z;
        }
    }
    for (int q = tid; q < kWT * cpb; q += kThreads) Cacc[q] = make_double2(0.0, 0.0);
    __syncthreads();
    int kstart = A.n_t;
    for (int b = 0; b < A.bpt; ++b)
        if (binfo[b] >= 0) kstart = min(kstart, A.kfirst[binfo[b]]);
    // pairs d: hi = h0 + d, lo = l0 - d (an odd grid's middle step is its own pair, d = 0)
    const int h0 = A.n_t >> 1, l0 = (A.n_t - 1) >> 1;
    const int n_pairs = A.n_t - h0;
    const double t_mid = 0.5 * (A.t_arr[h0] + A.t_arr[l0]);
    const int c_start = max(0, kstart - h0) / kKC;
    const int n_chunks = kstart < A.n_t ? (n_pairs + kKC - 1) / kKC : 0;
    const long col0 = (long)tile * COLS;
    const int lane = tid & 31, wp = tid >> 5;

    for (int i = A.n_cos * part / parts; i < A.n_cos * (part + 1) / parts; ++i) {
        const double ci = A.cos_t[i];
        const double one_m_c = 1.0 - ci;
        for (int q = tid; q < kKC * kWT; q += kThreads) {
            const int n = q / kWT, wl = q % kWT;
            const int wi = w0 + wl;
            double sn = 0.0, cs = 1.0;
            if (wi < A.n_w) phase<double>(A.w[wi] * one_m_c * (n * A.dt), sn, cs);
            Pn_re[q] = cs;
            Pn_im[q] = sn;
        }
        const double* bi = beta + (((size_t)frame * A.n_cos + i) * A.cols_pad + col0) * A.t_pad;
        // a warp's lanes take 32 consecutive pairs of one column: both halves are read in whole lines
        double hi[NPRE], lo[NPRE];
        auto fetch = [&](int d0) {
            const int d = d0 + lane;
            const bool in = d < n_pairs;
#pragma unroll
            for (int v = 0; v < NPRE; ++v) {
                const double* c = bi + (size_t)(wp + 8 * v) * A.t_pad;
                hi[v] = in ? __ldg(c + h0 + d) : 0.0;
                lo[v] = in && h0 + d != l0 - d ? __ldg(c + l0 - d) : 0.0;
            }
        };
        double acc[kTM][TN];
#pragma unroll
        for (int r = 0; r < kTM; ++r)
#pragma unroll
            for (int u = 0; u < TN; ++u) acc[r][u] = 0.0;
        if (c_start < n_chunks) fetch(c_start * kKC);
        __syncthreads();

        for (int ch = c_start; ch < n_chunks; ++ch) {
            const int d0 = ch * kKC;
            if (tid < kWT) {
                const int wi = w0 + tid;
                double sn = 0.0, cs = 0.0;
                if (wi < A.n_w) phase<double>(A.w[wi] * one_m_c * (0.5 * (A.t_arr[h0 + d0] - A.t_arr[l0 - d0])), sn, cs);
                anc[tid] = cs;
                anc[kWT + tid] = sn;
            }
#pragma unroll
            for (int v = 0; v < NPRE; ++v) {
                Esm[lane * BS + wp + 8 * v] = hi[v] + lo[v];
                // (the middle step of an odd grid has no sine)
                Osm[lane * BS + wp + 8 * v] = hi[v] - lo[v];
            }
            __syncthreads();
            for (int q = tid; q < kKC * kWT; q += kThreads) {
                const int n = q / kWT, wl = q % kWT;
                const double ar = anc[wl], ai = anc[kWT + wl];
                const double pr = Pn_re[q], pi = Pn_im[q];
                const bool valid = d0 + n < n_pairs;
                *reinterpret_cast<double2*>(Msm + n * kRows + 2 * wl) =
                    valid ? make_double2(ar * pr - ai * pi, ar * pi + ai * pr) : make_double2(0.0, 0.0);
            }
            __syncthreads();
            if (ch + 1 < n_chunks) fetch(d0 + kKC);  // in flight during the products below
#pragma unroll 4
            for (int n = 0; n < kKC; ++n) {
                const double2* ap = reinterpret_cast<const double2*>(Msm + n * kRows + ty * kTM);
                const double* ep = Esm + n * BS + tx * (TN / 2);
                const double* op = Osm + n * BS + tx * (TN / 2);
                const double2 e0 = *reinterpret_cast<const double2*>(ep), e1 = *reinterpret_cast<const double2*>(ep + COLS / 2);
                const double2 o0 = *reinterpret_cast<const double2*>(op), o1 = *reinterpret_cast<const double2*>(op + COLS / 2);
                const double e[TN] = {e0.x, e0.y, e1.x, e1.y}, o[TN] = {o0.x, o0.y, o1.x, o1.y};
#pragma unroll
                for (int r = 0; r < kTM / 2; ++r) {
                    const double2 a = ap[r];  // cos, sin of frequency ty * 4 + r
#pragma unroll
                    for (int u = 0; u < TN; ++u) {
                        acc[2 * r][u] = fma(a.x, e[u], acc[2 * r][u]);
                        acc[2 * r + 1][u] = fma(a.y, o[u], acc[2 * r + 1][u]);
                    }
                }
            }
            __syncthreads();
        }
        // epilogue: per thread, C_{s,g}(w) partials of its columns in fixed order, in structure-of-arrays
        // order red[(q*cpb + sg)*kThreads + tid]
        for (int q = 0; q < 4 * cpb; ++q) red[(size_t)q * kThreads + tid] = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < kTM / 2; ++q) {
            const int wl = ty * (kTM / 2) + q;
            const int wi = w0 + wl;
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                const int col = thread_col<TN, COLS>(tx, u);
                const int b = col / cpb;
                if (b >= A.bpt || binfo[b] < 0 || wi >= A.n_w) continue;
                double sn, cs;
                middle_phase(A.w[wi], bt[b], bz[b], ci, t_mid, sn, cs);
                const double yr = acc[2 * q][u], yi = acc[2 * q + 1][u];
                double2& d = red[(size_t)(q * cpb + (col % cpb)) * kThreads + tid];
                d.x += cs * yr - sn * yi;
                d.y += cs * yi + sn * yr;
            }
        }
        __syncthreads();
        for (int q = tid; q < kWT * cpb; q += kThreads) {
            const int wl = q / cpb, sg = q % cpb;
            const int tyw = wl / (kTM / 2), qq = wl % (kTM / 2);
            double2 sum = Cacc[q];
            for (int t = 0; t < 16; ++t) {
                const double2 v = red[(size_t)(qq * cpb + sg) * kThreads + tyw * 16 + t];
                sum.x += v.x;
                sum.y += v.y;
            }
            Cacc[q] = sum;
        }
        __syncthreads();
    }
    for (int q = tid; q < kWT * cpb; q += kThreads) {
        const int wl = q / cpb, sg = q % cpb;
        const int s = sg >> 1, g = sg & 1;
        const int wi = w0 + wl;
        if (wi >= A.n_w) continue;
        const size_t at = ((((size_t)frame * A.tiles_per_frame + tile) * parts + part) * 2 + g) * A.S + s;
        A.partial[at * A.n_w + wi] = Cacc[q];
    }
}

__global__ void k_reduce_tiles(const double2* __restrict__ partial, int tiles, size_t per, int kn,
                               double2* __restrict__ out) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (q >= per || k >= kn) return;
    double2 acc = make_double2(0.0, 0.0);
    const double2* p = partial + (size_t)k * tiles * per + q;
    for (int t = 0; t < tiles; ++t) {
        const double2 v = p[(size_t)t * per];
        acc.x += v.x;
        acc.y += v.y;
    }
    out[(size_t)k * per + q] = acc;
}

// Batched jobs: frame k of realization r is the sum of its own column tiles'
// partials, in the order of k_reduce_tiles (tiles, then row parts).
__global__ void k_reduce_real(const double2* __restrict__ partial, const uint32_t* __restrict__ real_tiles,
                              int tiles_per_frame, int parts, size_t per, int kn, size_t n_k, size_t k0,
                              double2* __restrict__ out) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    const int r = blockIdx.z;
    if (q >= per || k >= kn) return;
    double2 acc = make_double2(0.0, 0.0);
    const double2* p = partial + (size_t)k * tiles_per_frame * parts * per + q;
    for (size_t t = (size_t)real_tiles[r] * parts; t < (size_t)real_tiles[r + 1] * parts; ++t) {
        const double2 v = p[t * per];
        acc.x += v.x;
        acc.y += v.y;
    }
    out[((size_t)r * n_k + k0 + k) * per + q] = acc;
}

// ---------------------------------------------------------------------------
static size_t gemm_smem_bytes(int S) {
    size_t b = (size_t)kKC * kRows * sizeof(float) + (size_t)kKC * kGemmBS * sizeof(float);
    b = (b + 15) & ~(size_t)15;
    b += 2 * (size_t)kKC * kWT * sizeof(double);   // step table
    b += 2 * (size_t)kWT * sizeof(double);         // anchors
    b += (size_t)kThreads * 4 * 2 * S * sizeof(double2);  // epilogue partials
    b += (size_t)kWT * 2 * S * sizeof(double2);    // C accumulator
    b += 64 * sizeof(int) + 2 * 64 * sizeof(double);
    return b;
}

struct FactGeom {
    int bpt, tiles_per_frame, t_pad, nblk, tile_cols;
    long cols_pad;
};

// real_size: 8 (FP64 GEMM, 64-column tiles), 4 (FP32 GEMM) or 1 (int8 tensor-core GEMM), 128-column tiles
static FactGeom fact_geom(const SpectrumJob& job, size_t real_size) {
    FactGeom g;
    const int S = (int)job.n_sets;
    const int cols = real_size == 8 ? 64 : 128;
    g.tile_cols = cols;
    g.bpt = std::min(64, cols / (2 * S));
    g.tiles_per_frame = (int)((job.n_sel + g.bpt - 1) / g.bpt);
    g.cols_pad = (long)g.tiles_per_frame * cols;  // every tile is `cols` wide; unused columns stay zero
    const int align = real_size == 4 ? 4 : 2;
    g.t_pad = (int)((job.n_t + align - 1) / align * align);
    g.nblk = (int)((job.n_t + 31) / 32);
    return g;
}

// Sums the column-tile partials of kn frames: per frame (single job) or per
// (realization, frame) (batched job).
static uint64_t reduce_tiles(Device* dev, const SpectrumJob& job, const double2* partial, int tiles_per_frame,
                             int parts, size_t per, size_t k0, size_t kn, double2* out, const uint32_t* real_tiles) {
    if (job.n_real > 0) {
        if (job.n_real > 65535) throw Error{"too many realizations in one batched call"};
        dim3 gr((unsigned)((per + 255) / 256), (unsigned)kn, (unsigned)job.n_real);
        k_reduce_real<<<gr, 256, 0, dev->stream>>>(partial, real_tiles, tiles_per_frame, parts, per, (int)kn,
                                                   job.n_k, k0, out);
    } else {
        dim3 gr((unsigned)((per + 255) / 256), (unsigned)kn);
        k_reduce_tiles<<<gr, 256, 0, dev->stream>>>(partial, tiles_per_frame * parts, per, (int)kn, out + k0 * per);
    }
    CUDA_OK(cudaGetLastError());
    return 1;
}

template <class Real>
static uint64_t launch_typed(Device* dev, const SpectrumJob& job, const D4* bub_frames, const uint32_t* sel,
                             const double* tau, const double* cos_t, const double* sin2, const double* cos2,
                             const double* coeffs, const double* powers, const double* t_arr, const double* cutw,
                             const double* w, size_t k0, size_t kn, double2* out, const uint32_t* real_tiles,
                             cudaEvent_t* ev3) {
    const int S = (int)job.n_sets, M = (int)job.n_terms, SM = S * M;
    const int n_t = (int)job.n_t, n_cos = (int)job.n_cos, n_phi = (int)job.n_phi, n_w = (int)job.n_w;
    const int n_sel = (int)job.n_sel;
    constexpr bool tc = std::is_same<Real, int8_t>::value;
    if (SM > 8 || 2 * S > (sizeof(Real) == 8 ? 64 : 128))
        throw Error{"the factored kernels support at most 8 (set, term) pairs; use the fp64_direct kernel"};
    if (job.has_damping) {
        const double span = job.t_arr[job.n_t - 1] - job.t_arr[0] + 4.0;
        if (!(std::fabs(span / job.damping) < 600.0))
            throw Error{"damping width too small for the factored kernels (exp overflow); use fp64_direct"};
    }
    const FactGeom G = fact_geom(job, sizeof(Real));
    uint64_t launches = 0;
    // per-bubble time tables (frame independent)
    const int tf = G.nblk * 32;
    dev->fact_D.ensure((size_t)n_sel * tf * (1 + SM) * sizeof(double));
    dev->fact_kfirst.ensure((size_t)n_sel * sizeof(int));
    if ((n_t + 127) / 128 > 65535) throw Error{"too many time steps for the time-table grid"};
    {
        dim3 g((unsigned)n_sel, (unsigned)((tf + 127) / 128));
        k_time_tables<<<g, 128, 0, dev->stream>>>(bub_frames, sel, n_sel, t_arr, n_t, tf, powers, coeffs, cutw, SM,
                                                  job.has_damping ? 1 : 0, job.damping, (double*)dev->fact_D.p,
                                                  (int*)dev->fact_kfirst.p);
        CUDA_OK(cudaGetLastError());
        ++launches;
    }
    // beta
    record_event(dev, ev3[0]);
    const int nkb = G.nblk;
    const size_t beta_elems = tc ? (size_t)kn * n_cos * G.tiles_per_frame * nkb * kI8BlockSet
                                 : (size_t)kn * n_cos * G.cols_pad * G.t_pad;
    if (tc) {
        // row scales, and the per-block maxima of the time table that bound them
        dev->beta_scale.ensure((size_t)kn * n_sel * n_cos * sizeof(double));
        dev->fact_Dmax.ensure((size_t)n_sel * nkb * (1 + SM) * 2 * sizeof(double));
        const long warps = (long)n_sel * nkb;
        k_time_maxima<<<(unsigned)((warps + 7) / 8), 256, 0, dev->stream>>>((const double*)dev->fact_D.p, n_sel, tf,
                                                                            nkb, 1 + SM, (double*)dev->fact_Dmax.p);
        CUDA_OK(cudaGetLastError());
        ++launches;
    }
    dev->beta.ensure(beta_elems * sizeof(Real));
    if ((long)n_sel * 2 * S != G.cols_pad) {  // unused tile columns must read as zero
        // padding columns of the last tile are read by the GEMM: keep them zero
        CUDA_OK(cudaMemsetAsync(dev->beta.p, 0, beta_elems * sizeof(Real), dev->stream));
    }
    {
        BetaArgs B;
        B.tau = tau;
        B.bub = bub_frames;
        B.sel = sel;
        B.n_sel = n_sel;
        B.n_cos = n_cos;
        B.n_phi = n_phi;
        B.n_t = n_t;
        B.S = S;
        B.M = M;
        B.t_arr = t_arr;
        B.cutw = cutw;
        B.cos_t = cos_t;
        B.cos2 = cos2;
        B.sin2 = sin2;
        B.powers = powers;
        B.coeffs = coeffs;
        B.D = (const double*)dev->fact_D.p;
        B.tf = tf;
        B.has_damp = job.has_damping ? 1 : 0;
        B.damp = job.damping;
        B.dphi = 2.0 * M_PI / (double)n_phi;
        B.dcos = 2.0 / (double)(n_cos - 1);
        B.dt = job.dt;
        B.n_rows = (long)kn * n_sel * n_cos;
        B.nblk = G.nblk;
        B.cols_pad = G.cols_pad;
        B.tile_cols = G.tile_cols;
        B.bpt = G.bpt;
        B.t_pad = G.t_pad;
        // shared memory of a warp: a segment's bins (a second segment's too while the blocks still fit an
        // SM), the quiet constants, the row's delays and steps; of the block: the weights
        const size_t pitch = (((size_t)n_phi + 31) / 32) | 1;
        const size_t bins = (size_t)(2 + 2 * SM) * kSeg;
        const size_t others = 4 + 2 * (size_t)SM + beta_rows_held(SM) * 32 * pitch + 16 * pitch;
        const size_t blocks_sm = beta_blocks(SM), most = beta_warps(SM);
        B.keep = tc && blocks_sm * (64 * pitch + most * (2 * bins + others)) * sizeof(double) <= kBetaShared ? 2 : 1;
        const size_t per_warp = (B.keep * bins + others + 1) & ~(size_t)1;
        B.per_warp = (int)per_warp;
        B.tiles = G.tiles_per_frame;
        B.scale = tc ? (double*)dev->beta_scale.p : nullptr;
        B.Dmax = tc ? (const double*)dev->fact_Dmax.p : nullptr;
        bool sorted = false;
        if constexpr (tc) sorted = job.keep_masks;
        if (sorted) {
            if constexpr (tc) launch_sorted(SM, B, (int8_t*)dev->beta.p, dev->stream);
        } else {
            const size_t room = kBetaShared / sizeof(double);
            if (64 * pitch + per_warp > room) throw Error{"n_phi too large for the beta kernel"};
            const int warps = (int)std::min<size_t>(most, (room - 64 * pitch) / per_warp);
            const size_t smem = (64 * pitch + warps * per_warp) * sizeof(double);
            launch_beta<Real>(SM, B, (Real*)dev->beta.p, smem, dev->n_sm, warps, dev->stream);
        }
        CUDA_OK(cudaGetLastError());
        ++launches;
    }
    // GEMM + epilogue
    record_event(dev, ev3[1]);
    FactArgs A;
    A.bub = bub_frames;
    A.n_tot = job.n_tot;
    A.sel = sel;
    A.n_sel = n_sel;
    A.n_cos = n_cos;
    A.n_t = n_t;
    A.n_w = n_w;
    A.S = S;
    A.t_arr = t_arr;
    A.w = w;
    A.cos_t = cos_t;
    A.kfirst = (const int*)dev->fact_kfirst.p;
    A.beta = dev->beta.p;
    A.cols_pad = G.cols_pad;
    A.t_pad = G.t_pad;
    A.dt = job.dt;
    A.bpt = G.bpt;
    A.tiles_per_frame = G.tiles_per_frame;
    const size_t per = (size_t)2 * S * n_w;
    // tensor-core path: each column tile's CTAs split the cos-theta rows so that
    // the grid fills whole waves of one CTA per SM
    constexpr bool fold = std::is_same<Real, double>::value;
    const int row_parts =
        fold ? fold_row_parts(n_cos)
        : !tc ? 1
              : job.row_parts > 0 ? std::min(std::min(job.row_parts, 16), n_cos)
                                  : tc_row_parts((size_t)((n_w + 63) / 64) * kn * G.tiles_per_frame, n_cos, dev->n_sm);
    // (the launch shape's row parts are the tensor-core GEMM's)
    dev->last_row_parts = tc ? row_parts : 1;
    dev->fact_partial.ensure((size_t)kn * G.tiles_per_frame * row_parts * per * sizeof(double2));
    A.partial = (double2*)dev->fact_partial.p;
    if constexpr (tc) {
        // time-phase digits: frame independent, built by the first launch chunk of each call
        // (0.8 ms at config 3) and reused by the others
        const int n_wt = (n_w + 63) / 64;
        const size_t atab_bytes = (size_t)n_cos * n_wt * nkb * kI8BlockSet;
        if (!dev->tc_atab_valid || dev->tc_atab.cap < atab_bytes) {
            dev->tc_atab.ensure(atab_bytes);
            launch_tc_phase_table(w, cos_t, t_arr, n_cos, n_w, n_t, (int8_t*)dev->tc_atab.p, dev->stream);
            ++launches;
            dev->tc_atab_valid = true;
        }
        TcArgs T;
        T.bub = bub_frames;
        T.n_tot = job.n_tot;
        T.sel = sel;
        T.n_sel = n_sel;
        T.n_cos = n_cos;
        T.n_t = n_t;
        T.n_w = n_w;
        T.S = S;
        T.w = w;
        T.cos_t = cos_t;
        T.kfirst = (const int*)dev->fact_kfirst.p;
        T.atab = (const int8_t*)dev->tc_atab.p;
        T.btab = (const int8_t*)dev->beta.p;
        T.bscale = (const double*)dev->beta_scale.p;
        T.n_wt = n_wt;
        T.nkb = nkb;
        T.bpt = G.bpt;
        T.tiles_per_frame = G.tiles_per_frame;
        T.row_parts = row_parts;
        T.stages = job.gemm_stages > 0 ? job.gemm_stages : 4;
        dev->last_gemm_stages = T.stages;
        T.partial = A.partial;
        T.err = reinterpret_cast<unsigned int*>(static_cast<unsigned char*>(dev->counters.p) + 8);
        launch_gemm_tc(T, kn, dev->stream);
        ++launches;
        record_event(dev, ev3[2]);
        launches += reduce_tiles(dev, job, A.partial, G.tiles_per_frame, row_parts, per, k0, kn, out, real_tiles);
        return launches;
    } else {
        const size_t smem = fold ? fold_smem_bytes(S) : gemm_smem_bytes(S);
        // (the folded product's layout has room for 6 sets; more than 4 were always refused in FP64)
        if (smem > kMaxBlockShared || (fold && S > 4))
            throw Error{"too many coefficient sets for the factored kernel's shared memory"};
        const size_t gy = (size_t)kn * G.tiles_per_frame;
        if (gy > 65535) throw Error{"too many column tiles in one k-hat chunk"};
        const dim3 grid((unsigned)((n_w + kWT - 1) / kWT), (unsigned)gy, (unsigned)row_parts);
        if constexpr (fold) {
            allow_shared(k_gemm_fold, kMaxBlockShared);
            k_gemm_fold<<<grid, kThreads, smem, dev->stream>>>(A, fold_work(S));
        } else {
            allow_shared(k_gemm, kMaxBlockShared);
            k_gemm<<<grid, kThreads, smem, dev->stream>>>(A);
        }
        CUDA_OK(cudaGetLastError());
        ++launches;
        record_event(dev, ev3[2]);
        launches += reduce_tiles(dev, job, A.partial, G.tiles_per_frame, row_parts, per, k0, kn, out, real_tiles);
        return launches;
    }
}

uint64_t launch_factored(Device* dev, const SpectrumJob& job, const D4* bub_frames, const uint32_t* sel,
                         const double* tau, const double* cos_t, const double* sin2, const double* cos2,
                         const double* coeffs, const double* powers, const double* t_arr, const double* cutw,
                         const double* w, size_t k0, size_t kn, double2* out, const uint32_t* real_tiles,
                         cudaEvent_t* ev3) {
    if (job.kernel == BGWX_KERNEL_MIXED)
        return launch_typed<int8_t>(dev, job, bub_frames, sel, tau, cos_t, sin2, cos2, coeffs, powers, t_arr, cutw, w,
                                    k0, kn, out, real_tiles, ev3);
    if (job.kernel == BGWX_KERNEL_MIXED_SIMT)
        return launch_typed<float>(dev, job, bub_frames, sel, tau, cos_t, sin2, cos2, coeffs, powers, t_arr, cutw, w,
                                   k0, kn, out, real_tiles, ev3);
    return launch_typed<double>(dev, job, bub_frames, sel, tau, cos_t, sin2, cos2, coeffs, powers, t_arr, cutw, w, k0,
                                kn, out, real_tiles, ev3);
}

size_t factored_bubbles_per_tile(const SpectrumJob& job) {
    const size_t real = job.kernel == BGWX_KERNEL_MIXED        ? 1
                        : job.kernel == BGWX_KERNEL_MIXED_SIMT ? sizeof(float)
                                                               : sizeof(double);
    return (size_t)fact_geom(job, real).bpt;
}

int factored_auto_row_parts(const Device* dev, const SpectrumJob& job, size_t kn) {
    if (job.kernel != BGWX_KERNEL_MIXED) return 1;
    const FactGeom G = fact_geom(job, 1);
    return tc_row_parts((size_t)((job.n_w + 63) / 64) * kn * G.tiles_per_frame, (int)job.n_cos, dev->n_sm);
}

size_t factored_bytes_per_frame(const SpectrumJob& job) {
    const size_t real = job.kernel == BGWX_KERNEL_MIXED        ? 1
                        : job.kernel == BGWX_KERNEL_MIXED_SIMT ? sizeof(float)
                                                               : sizeof(double);
    const FactGeom G = fact_geom(job, real);
    // int8 tensor-core path: the digit block sets and one FP64 scale per (bubble, row)
    const size_t beta = job.kernel == BGWX_KERNEL_MIXED
                            ? (size_t)job.n_cos * G.tiles_per_frame * G.nblk * kI8BlockSet +
                                  (size_t)job.n_sel * job.n_cos * sizeof(double)
                            : (size_t)job.n_cos * G.cols_pad * G.t_pad * real;
    // partials: up to 16 row parts per column tile on the tensor-core and the FP64 path
    const size_t parts = job.kernel == BGWX_KERNEL_MIXED_SIMT ? 1 : 16;
    return beta + (size_t)G.tiles_per_frame * parts * 2 * job.n_sets * job.n_w * sizeof(double2);
}

}  // namespace bgw
