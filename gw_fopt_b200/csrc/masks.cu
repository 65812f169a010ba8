// First-collider search with per-bubble candidate lists (exact).
//
// For interior bubble a and a collider c with Delta = x_c - x_a (t, x, y, z),
// the collision delay along any direction x-hat = (1, n) is
//   tau_c(n) = s_c / (2 d_c),  s_c = -dt^2 + |dx|^2,  d_c = -dt + dx.n,
// and because d_c <= D_c = |dx| - dt and s_c = D_c (|dx| + dt),
//   tau_c(n) >= key_c = (|dx| + dt) / 2        for every n with d_c > 0.
// k_neighbors builds, once per radiating bubble (frame independent, the keys
// are rotation invariant), the list of the colliders with the smallest keys
// (radix select on the float keys, then a bitonic sort by (key, index)),
// kmax = a lower bound of every key outside the list, and
//   rho1 = max_c (dt^2 + |dx|^2) / D_c,  rho2 = max_c (|dt| + |dx|) / D_c.
//
// k_masks_list then decides each direction exactly as the reference
// (generalized_bulk_flow.rs:127-206, 1003-1018) does -- the unique b passing
// check(b, c) against every c, or None -- but evaluates only what can matter:
//   1. argmin m of tau over the list in key order, stopping once
//      key > tau_best (1 + 1e-12): no later collider can have a smaller tau;
//   2. check(m, c) for the listed c with key_c <= theta_m, where
//        theta_m = tau_m (1 + 1e-12) + 64 u (A_m rho1 + Q_m rho2) / d_m
//      (u = 2^-53).  The rounding error of the reference's check expression is
//      below 20 u (A_m Q_c + A_c Q_m) while its exact value is at least
//      2 d_m D_c (key_c - tau_m), so every c with key_c > theta_m passes in
//      floating point as well and needs no evaluation;
//   3. if m fails, the passer (if any) is one of the c that m failed against
//      (r(c, m) = -r(m, c) exactly in IEEE arithmetic); each is verified the
//      same way.
// Patch lists.  Almost every direction is decided without steps 1-3, from the fact that a collider's
// inverse delay is linear in the direction: 1 / (2 tau_c) = d_c / s_c = (dx.n - dt) / s_c, so the first
// collider is the largest of a few linear forms.  A warp takes an item, a small patch of the sphere inside
// a cap about its middle direction.  Over the cap d_c lies in [D-, D+], so every collider with D- > 0
// bounds the first collision by s_c / (2 D-); with T the least of these, a collider with
//   s_c / 2 - T max(D+, 0) > 1e-9 (Q_c + A_c)
// passes every check against a candidate with tau_m <= T: the check's exact value is at least
// 2 d_m (s_c / 2 - tau_m max(D+, 0)) and its rounding error below 20 u (A_m Q_c + A_c Q_m), which the
// margin covers for every candidate with max(A_m, Q_m) / d_m <= 4e5.  The others (about 7 of the 25 to 55
// entries whose key is small enough) are kept per warp as FP32 forms
//   g_e(n) = dx.n / s - dt / s + w_e,   w_e = 32 2^-24 L1_e / s,
// and one pass per direction finds the largest and the second largest g.  With m the largest,
// g_second < g_m - 2 w_m certifies check(m, e) for every e: w is more than three times the FP32 error
// 9 2^-24 L1 / s of a form, and the reference's own rounding is far below that.  Ties to within FP32 (2.5
// directions in 1e5) are decided by the reference's expression.  A patch that keeps too many colliders
// (towards the corners of the box, where the first collision is late) is halved, and at one tile of 32
// directions the pass runs over the whole list.  What is still open (a near-lightlike first
// collider, an unlisted first collider, one of the conditions above broken) takes steps 1-3 in a second kernel.
// What bounds it: issue (77 % of the slots); per direction about 9 instructions per entry and 100 more,
// per list about 400.  8 frames of 4096 bubbles x 192 x 192 directions: 13.7 ms (40.4 ms with a walk down
// the rows, each direction's candidate verified in FP64 against every entry with a smaller key); 32 frames
// of 256 bubbles x 64 x 64: 0.73 ms (2.26).
//
// Whenever a bound reaches past the list (or the list has no candidate and is
// not complete) the direction falls back to the exhaustive scan over all
// colliders.  Colliders with a near-lightlike interval (D_c tiny) are kept in
// a small always-checked set; too many of them make the bubble use the
// exhaustive scan for every direction.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "bgw_internal.h"
#include "device_common.cuh"
#include "masks.cuh"

namespace bgw {

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ bool check_pt(const D4& dba, double nb, const D4& dca, const D4& x) {
    const double nc = mdot(dca, dca);
    D4 cv;
    cv.t = dsub(dmul(dba.t, nc), dmul(dca.t, nb));
    cv.x = dsub(dmul(dba.x, nc), dmul(dca.x, nb));
    cv.y = dsub(dmul(dba.y, nc), dmul(dca.y, nb));
    cv.z = dsub(dmul(dba.z, nc), dmul(dca.z, nb));
    return mdot(cv, x) > 0.0;
}

// check(b, c) with both Minkowski norms precomputed (same values as check_pt).
__device__ __forceinline__ bool check_pre(const D4& dba, double nb, const D4& dca, double nc, const D4& x) {
    D4 cv;
    cv.t = dsub(dmul(dba.t, nc), dmul(dca.t, nb));
    cv.x = dsub(dmul(dba.x, nc), dmul(dca.x, nb));
    cv.y = dsub(dmul(dba.y, nc), dmul(dca.y, nb));
    cv.z = dsub(dmul(dba.z, nc), dmul(dca.z, nb));
    return mdot(cv, x) > 0.0;
}

// Exhaustive decision for one direction, by a whole warp (all 32 lanes call it
// with the same arguments).  It returns what the sequential procedure returns:
// the argmin of tau in collider order (first index on ties), checked against
// every collider; when it fails, the first of its failures (in collider order)
// that passes every check, or the reference loop (GBF:162-199) when it failed
// more than kMaxFail times.  Lanes take colliders lane, lane + 32, ...; a
// check over all colliders is the AND of the lanes' checks, so its order does
// not matter.
__device__ __forceinline__ double tau_of(const D4& dba, const D4& x, bool& ok) {
    const double dot = mdot(dba, x);
    ok = false;
    double tau = CUDART_INF;
    if (dot > 1e-10) {
        tau = __ddiv_rn(mdot(dba, dba), dmul(2.0, dot));
        ok = tau > 0.0;
    }
    return tau;
}

// true when check(b, c) passes for every collider c other than a and b
__device__ bool warp_all_pass(const D4* __restrict__ B, size_t n_tot, uint32_t a, size_t b, const D4& xa,
                              const D4& dba, double nb, const D4& x) {
    const unsigned full = 0xffffffffu;
    for (size_t base = 0; base < n_tot; base += 32) {
        const size_t c = base + (threadIdx.x & 31);
        bool pass = true;
        if (c < n_tot && c != a && c != b) pass = check_pt(dba, nb, dsub4(B[c], xa), x);
        if (!__all_sync(full, pass)) return false;
    }
    return true;
}

__device__ long exhaustive_warp(const D4* __restrict__ B, size_t n_tot, uint32_t a, const D4& xa, const D4& x) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // 1. argmin: lane-local first minimum, then the (tau, index) minimum over lanes
    double bt = CUDART_INF;
    long bi = -1;
    for (size_t b = lane; b < n_tot; b += 32) {
        if (b == a) continue;
        bool ok;
        const double tau = tau_of(dsub4(B[b], xa), x, ok);
        if (ok && tau < bt) {
            bt = tau;
            bi = (long)b;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double t2 = __shfl_xor_sync(full, bt, o);
        const long i2 = __shfl_xor_sync(full, bi, o);
        if (i2 >= 0 && (bi < 0 || t2 < bt || (t2 == bt && i2 < bi))) {
            bt = t2;
            bi = i2;
        }
    }
    if (bi < 0) return -1;
    const long best = bi;
    // 2. check the argmin against every collider; keep its first kMaxFail failures
    const D4 dm = dsub4(B[best], xa);
    const double nm = mdot(dm, dm);
    long my_fail = -1;  // lane f holds failure f
    int nfail = 0;
    for (size_t base = 0; base < n_tot; base += 32) {
        const size_t c = base + lane;
        bool fail = false;
        if (c < n_tot && c != a && (long)c != best) fail = !check_pt(dm, nm, dsub4(B[c], xa), x);
        unsigned m = __ballot_sync(full, fail);
        while (m && nfail < kMaxFail) {
            const int bit = __ffs(m) - 1;
            m &= m - 1;
            if (lane == nfail) my_fail = (long)(base + bit);
            ++nfail;
        }
        nfail += __popc(m);
    }
    if (nfail == 0) return best;
    if (nfail > kMaxFail) {
        // the reference loop (GBF:162-199): candidates in collider order with tau below the current result's
        long r = -1;
        double rt = CUDART_INF;
        for (size_t base = 0; base < n_tot; base += 32) {
            const size_t b = base + lane;
            bool ok = false;
            double tau = CUDART_INF;
            if (b < n_tot && b != a) {
                // the reference's skips: dot <= 1e-10, tau <= 0 (NaN goes on, as there)
                const D4 dba = dsub4(B[b], xa);
                const double dot = mdot(dba, x);
                if (!(dot <= 1e-10)) {
                    tau = __ddiv_rn(mdot(dba, dba), dmul(2.0, dot));
                    ok = !(tau <= 0.0);
                }
            }
            unsigned m = __ballot_sync(full, ok);
            while (m) {
                const int bit = __ffs(m) - 1;
                m &= m - 1;
                const double tb = __shfl_sync(full, tau, bit);
                if (tb >= rt) continue;
                const size_t cb = base + bit;
                const D4 dba = dsub4(B[cb], xa);
                if (warp_all_pass(B, n_tot, a, cb, xa, dba, mdot(dba, dba), x)) {
                    r = (long)cb;
                    rt = tb;
                }
            }
        }
        return r;
    }
    // 3. the first failure (in collider order) that passes every check
    for (int f = 0; f < nfail; ++f) {
        const long c = __shfl_sync(full, my_fail, f);
        const D4 dc = dsub4(B[c], xa);
        bool ok;
        tau_of(dc, x, ok);
        if (!ok) continue;
        if (warp_all_pass(B, n_tot, a, (size_t)c, xa, dc, mdot(dc, dc), x)) return c;
    }
    return -1;
}

// ------------------------------------------------------------ k_neighbors
__device__ __forceinline__ void collider_bounds(const D4& d, double& key, double& D, double& Q, double& A) {
    const double dx = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
    key = fmax(0.5 * (dx + d.t), 0.0);
    D = dx - d.t;
    Q = d.t * d.t + dx * dx;
    A = fabs(d.t) + dx;
}

// One block per radiating bubble.  The colliders are read once: their float keys (rounded down) stay in
// shared memory (up to n_cache of them; the others are formed again) for the three passes of the radix
// select, and the rho bounds and outliers are taken on the way.  Reading them in every pass, and one thread
// walking the 2048 bins, took 1.9 ms for 4096 bubbles among 28672 (L2 bandwidth) and 168 us for 256 among
// 1792 (the walk); now 1.25 ms there.
template <int NT>
__global__ void __launch_bounds__(NT)
    k_neighbors(const D4* __restrict__ bub, size_t n_int, size_t n_tot, const uint32_t* __restrict__ sel,
                const uint2* __restrict__ ranges, unsigned n_cache, NbList* __restrict__ out) {
    extern __shared__ unsigned s_fb[];  // [n_cache]
    __shared__ unsigned hist[2048];
    __shared__ unsigned s_prefix, s_mask, s_need, s_count, s_nout;
    __shared__ double s_key[kList];
    __shared__ int s_idx[kList];
    __shared__ double s_r1[NT / 32], s_r2[NT / 32];
    __shared__ unsigned s_sum[NT / 32];
    const int slot = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t a = sel[slot];
    NbList* L = out + slot;
    if (a >= n_int) {  // not an interior bubble: marked, never dereferenced
        if (tid == 0) L->count = -1;
        return;
    }
    if (ranges) {  // several realizations: this slot's colliders are its own realization's rows
        const uint2 r = ranges[slot];
        bub += r.x;
        n_tot = r.y;
        a -= r.x;
    }
    const D4 xa = bub[a];
    const unsigned n = (unsigned)n_tot;
    const bool complete = n - 1 <= (unsigned)kList;  // colliders other than a
    if (tid == 0) {
        s_prefix = 0;
        s_mask = 0;
        s_need = kList;  // rank of the cut value (1-based)
        s_count = 0;
        s_nout = 0;
    }
    for (int q = tid; q < 2048; q += NT) hist[q] = 0;
    __syncthreads();
    constexpr unsigned kSelf = 0xffffffffu;  // above every key
    auto fbits = [&](unsigned c, double& key, double& D, double& Q, double& A) -> unsigned {
        collider_bounds(dsub4(bub[c], xa), key, D, Q, A);
        return c == a ? kSelf : __float_as_uint(__double2float_rd(key));
    };
    auto fkey = [&](unsigned c) -> unsigned {
        double key, D, Q, A;
        return c < n_cache ? s_fb[c] : fbits(c, key, D, Q, A);
    };
    // first pass: keys, the first histogram, rho bounds; near-lightlike colliders are kept aside
    double r1 = 0.0, r2 = 0.0;
    for (unsigned c = tid; c < n; c += NT) {
        double key, D, Q, A;
        const unsigned v = fbits(c, key, D, Q, A);
        if (c < n_cache) s_fb[c] = v;
        if (v == kSelf) continue;
        if (!complete) atomicAdd(&hist[v >> 21], 1u);
        if (D > 1e-6 * A) {
            r1 = fmax(r1, Q / D);
            r2 = fmax(r2, A / D);
        } else {
            const unsigned pos = atomicAdd(&s_nout, 1u);
            if (pos < (unsigned)kMaxOutliers) L->outlier[pos] = (int)c;
        }
    }
    unsigned cut = kSelf;  // list = {c : fkey(c) < cut}
    if (!complete) {
        const int shifts[3] = {21, 10, 0};
        const unsigned widths[3] = {11, 11, 10};
        for (int p = 0; p < 3; ++p) {
            const unsigned dmask = (1u << widths[p]) - 1u;
            if (p > 0) {
                for (int q = tid; q < 2048; q += NT) hist[q] = 0;
                __syncthreads();
                const unsigned pre = s_prefix, pm = s_mask;
                for (unsigned c = tid; c < n; c += NT) {
                    const unsigned v = fkey(c);
                    if (v != kSelf && (v & pm) == pre) atomicAdd(&hist[(v >> shifts[p]) & dmask], 1u);
                }
            }
            __syncthreads();
            // the bin that holds rank s_need: thread t sums NB bins from NB t on, block scan of the sums
            constexpr int NB = 2048 / NT;
            unsigned own[NB], sum = 0;
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                own[q] = hist[NB * tid + q];
                sum += own[q];
            }
            unsigned incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) s_sum[warp] = incl;
            __syncthreads();
            unsigned before = incl - sum;
            for (int w = 0; w < warp; ++w) before += s_sum[w];
            const unsigned need = s_need, pre = s_prefix, pm = s_mask;
            __syncthreads();
            if (before < need && need <= before + sum) {  // one thread
                unsigned acc = before;
                bool found = false;
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    if (!found && acc + own[q] >= need) {
                        s_need = need - acc;
                        s_prefix = pre | ((unsigned)(NB * tid + q) << shifts[p]);
                        found = true;
                    }
                    acc += own[q];
                }
                s_mask = pm | (dmask << shifts[p]);
            }
            __syncthreads();
        }
        cut = s_prefix;  // the kList-th smallest float key (bits)
    } else {
        __syncthreads();
    }
    // collect the list (unordered), then sort by (key, index)
    for (unsigned c = tid; c < n; c += NT) {
        if (fkey(c) < cut) {  // (a itself has the largest)
            double key, D, Q, A;
            collider_bounds(dsub4(bub[c], xa), key, D, Q, A);
            const unsigned pos = atomicAdd(&s_count, 1u);
            if (pos < (unsigned)kList) {
                s_key[pos] = key;
                s_idx[pos] = (int)c;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        r1 = fmax(r1, __shfl_xor_sync(0xffffffffu, r1, o));
        r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    }
    if (lane == 0) {
        s_r1[warp] = r1;
        s_r2[warp] = r2;
    }
    __syncthreads();
    const int count = (int)min(s_count, (unsigned)kList);
    int sorted = 32;  // the sort's length: the next power of two
    while (sorted < count) sorted <<= 1;
    for (int q = count + tid; q < sorted; q += NT) {
        s_key[q] = CUDART_INF;
        s_idx[q] = 0x7fffffff;
    }
    __syncthreads();
    // bitonic sort
    for (int size = 2; size <= sorted; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int q = tid; q < sorted; q += NT) {
                const int p = q ^ stride;
                if (p > q) {
                    const bool up = (q & size) == 0;
                    const double kq = s_key[q], kp = s_key[p];
                    const int iq = s_idx[q], ip = s_idx[p];
                    const bool gt = kq > kp || (kq == kp && iq > ip);
                    if (gt == up) {
                        s_key[q] = kp;
                        s_key[p] = kq;
                        s_idx[q] = ip;
                        s_idx[p] = iq;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int q = tid; q < count; q += NT) {
        L->key[q] = s_key[q];
        L->idx[q] = s_idx[q];
    }
    if (tid == 0) {
        double m1 = 0.0, m2 = 0.0;
        for (int q = 0; q < NT / 32; ++q) {
            m1 = fmax(m1, s_r1[q]);
            m2 = fmax(m2, s_r2[q]);
        }
        L->rho1 = m1 * (1.0 + 1e-12);
        L->rho2 = m2 * (1.0 + 1e-12);
        L->count = count;
        L->kmax = complete ? CUDART_INF : (double)__uint_as_float(cut);
        const unsigned no = s_nout;
        L->n_outliers = no <= (unsigned)kMaxOutliers ? (int)no : -1;
    }
}

// Float keys of up to 32768 colliders stay in shared memory (128 KB; with several realizations, whose
// counts are below the total, up to 8192).  Above 8192 only one block fits an SM: 1024 threads then.
static void launch_neighbors(const D4* bub, size_t n_int, size_t n_tot, const uint32_t* sel, const uint2* ranges,
                             size_t n_sel, NbList* lists, cudaStream_t st) {
    if (n_sel > 0x7fffffffULL) throw Error{"too many radiating bubbles"};
    if (n_tot > 0x7fffffffULL) throw Error{"too many bubbles"};
    constexpr unsigned few = 8192, most = 32768;
    const unsigned n_cache = (unsigned)std::min<size_t>(n_tot, ranges ? few : most);
    const size_t smem = n_cache * sizeof(unsigned);
    auto* kernel = n_cache > few ? k_neighbors<1024> : k_neighbors<256>;
    allow_shared(kernel, (n_cache > few ? most : few) * sizeof(unsigned));
    kernel<<<(unsigned)n_sel, n_cache > few ? 1024 : 256, smem, st>>>(bub, n_int, n_tot, sel, ranges, n_cache, lists);
    CUDA_OK(cudaGetLastError());
}

// ------------------------------------------------------------ k_masks_list
// Shared memory of a block: the candidate list of its radiating bubble (direction independent, with the
// reference's operations), the warps' patch lists and what the slow path needs.
struct MaskBlock {
    D4 pos[kList];       // Delta = x_c - x_a of each listed collider
    double nrm[kList];   // its Minkowski norm
    double key[kList];
    int idx[kList];
    // in FP32, over s: the form's coefficients dx / s and -dt / s + w; |dx| / s, 2 w, the margin
    // 1e-9 (Q + A) / s, and the largest delay for which step 0 may decide for the collider
    float4 form[kList], fval[kList];
    // each warp's patch list: forms and list positions
    float4 pform[kMaskListThreads / 32][kPatchList];
    int ppos[kMaskListThreads / 32][kPatchList];
    D4 opos[kMaxOutliers];
    double onrm[kMaxOutliers];
    int oidx[kMaxOutliers];
    const D4* B;         // the frame's bubbles (of the slot's realization)
    size_t n_tot;
    uint32_t a;          // radiating bubble
    int n, no;           // listed colliders, outliers (-1: too many)
    D4 xa;
    double kmax, rho1, rho2;
    bool big;            // a listed Delta too large for the candidate filter's margin
    bool no_patch;       // no patch lists: that, outliers, or a listed |dx| whose square leaves the FP32 range
    unsigned next;       // the block's work queue of items
    unsigned open;       // directions were left open
};

// Direction-independent part of the verification bound of a collider (see decide_slow).
__device__ __forceinline__ double theta_slope(const MaskBlock& S, const D4& dc, double nrm) {
    const double dx = sqrt(dc.x * dc.x + dc.y * dc.y + dc.z * dc.z);
    const double A = fabs(dc.t) + dx, Q = dc.t * dc.t + dx * dx;
    return nrm > 0.0 ? 2.0 * (64.0 * 1.1102230246251565e-16) * (A * S.rho1 + Q * S.rho2) / nrm : CUDART_INF;
}

// Steps 1-3 for one direction.  Returns the first collider (-1: none) and its delay; `full`: only the
// exhaustive scan decides.
__device__ long decide_slow(const MaskBlock& S, const D4& x, double& res_tau, bool& full) {
    constexpr int kBatch = 2;
    const int n = S.n, no = S.no;
    const double kmax = S.kmax;
    long result = -1;
    res_tau = 0.0;
    full = no < 0 || S.big;

    // Approximate Minkowski product with the direction (FMA chain): within
    // 4.01 u L1(d) of the exact value, since |x_i| <= 1.
    auto adot = [&](const D4& p) { return fma(p.z, x.z, fma(p.y, x.y, fma(p.x, x.x, -(p.t * x.t)))); };

    // Verifies candidate c (Delta dc, norm nc) against the list up to key theta and the
    // outliers.  check(c, e) is the sign of the reference's expression V_ref; the filter value
    //   V = fma(ne, adot(c), -(nc adot(e)))
    // is within 6.03 u S of the exact value and V_ref within 6.01 u S, where
    // S = |ne| L1(c) + |nc| L1(e); |V| > 32 u S (plus an underflow guard) fixes
    // the sign, otherwise the reference's expression is evaluated.  The bound is taken as
    // 32 u max(L1(c), |nc|) (|ne| + L1(e)) >= 32 u S: looser, which only sends a few more
    // values near zero to the exact evaluation.  c is the candidate's collider index, cpos its
    // list position (the list holds each collider once).
    auto verify = [&](int c, int cpos, const D4& dc, double nc, double theta, int* fails, int& nfail) -> bool {
        const double dotc = adot(dc);
        const double l1c = fabs(dc.t) + fabs(dc.x) + fabs(dc.y) + fabs(dc.z);
        const double mc = 32.0 * 1.1102230246251565e-16 * fmax(l1c, fabs(nc));
        bool ok = true;
        // entries in batches of kBatch: their filter values are independent
        // (instruction-level parallelism); decisions are taken in list order
        bool done = false;
        for (int e0 = 0; e0 < n && !done; e0 += kBatch) {
            double vb[kBatch], bb[kBatch], kb[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int e = min(e0 + j, n - 1);
                kb[j] = S.key[e];
                const D4 pe = S.pos[e];
                const double ns = S.nrm[e];
                vb[j] = fma(ns, dotc, -(nc * adot(pe)));
                bb[j] = fma(fabs(ns) + (fabs(pe.t) + fabs(pe.x) + fabs(pe.y) + fabs(pe.z)), mc, 1e-300);
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int e = e0 + j;
                if (e >= n || kb[j] > theta) {
                    done = true;
                    break;
                }
                if (e == cpos) continue;
                bool pass;
                if (vb[j] > bb[j]) pass = true;
                else if (vb[j] < -bb[j]) pass = false;
                else pass = check_pre(dc, nc, S.pos[e], S.nrm[e], x);
                if (!pass) {
                    ok = false;
                    if (fails) {
                        if (nfail < kMaxFail) fails[nfail] = e;
                        ++nfail;
                    } else {
                        return false;
                    }
                }
            }
        }
        for (int e = 0; e < no; ++e) {
            const int ce = S.oidx[e];
            if (ce == c) continue;
            bool in_list = false;  // already checked above when listed with key <= theta
            for (int q = 0; q < n && S.key[q] <= theta; ++q) in_list |= (S.idx[q] == ce);
            if (in_list) continue;
            if (!check_pre(dc, nc, S.opos[e], S.onrm[e], x)) {
                ok = false;
                if (!fails) return false;
                nfail = kMaxFail + 1;  // outliers are resolved by the exhaustive path
            }
        }
        return ok;
    };
    // The verification bound of listed candidate e with delay tau: theta = tau (1 + 1e-12) +
    // 64 u (A rho1 + Q rho2) / dot with 1 / dot = 2 tau / nrm (the 1e-12 relative slack covers the few
    // roundings of this form)
    auto theta_of = [&](int e, double tau) { return tau * ((1.0 + 1e-12) + theta_slope(S, S.pos[e], S.nrm[e])); };


    if (!full) {
        // 1. a candidate: the approximate argmin of tau = nrm / (2 dot) in key order
        //    (quotients compared by cross-multiplication), stopping once key exceeds
        //    the best quotient with a margin.  Any candidate serves: steps 2-3 decide
        //    exactly whatever it is; the exact argmin only keeps step 3 idle.
        double bn = 0.0, bd = 0.0;  // best quotient bn / bd, bd > 0
        int bi = -1;
        bool ended = true, stop = false;
        for (int e0 = 0; e0 < n && !stop; e0 += kBatch) {
            double kb[kBatch], nb[kBatch], db[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int e = min(e0 + j, n - 1);
                kb[j] = S.key[e];
                nb[j] = S.nrm[e];
                db[j] = 2.0 * adot(S.pos[e]);
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                if (e0 + j >= n) break;
                if (bi >= 0 && kb[j] * bd > bn * (1.0 + 1e-11)) {
                    ended = false;
                    stop = true;
                    break;
                }
                // every collider of the exact test (dot > 1e-10, nrm > 0) has den > 0 here,
                // since the block's L1 norms keep 4.01 u L1 below 1e-10
                if (db[j] > 0.0 && nb[j] > 0.0 && (bi < 0 || nb[j] * bd < bn * db[j])) {
                    bn = nb[j];
                    bd = db[j];
                    bi = e0 + j;
                }
            }
        }
        double best = CUDART_INF, dotm = 0.0;
        if (bi >= 0) {
            // the candidate's tau with the reference's operations (compute_delta_tab)
            dotm = mdot(S.pos[bi], x);
            if (dotm > 1e-10) best = __ddiv_rn(S.nrm[bi], dmul(2.0, dotm));
            if (!(dotm > 1e-10) || !(best > 0.0)) full = true;  // not a collider by the exact test
        }
        if (!full && ended && !(kmax > best * (1.0 + 1e-11))) full = !(bi < 0 && kmax == CUDART_INF);
        if (!full && bi >= 0) {
            // 2. verify the candidate
            const D4 dm = S.pos[bi];
            const double nm = S.nrm[bi];
            const double th = theta_of(bi, best);
            if (!(th < kmax)) {
                full = true;
            } else {
                int fails[kMaxFail];
                int nfail = 0;
                if (verify(S.idx[bi], bi, dm, nm, th, fails, nfail)) {
                    result = S.idx[bi];
                    res_tau = best;
                } else if (nfail > kMaxFail) {
                    full = true;
                } else {
                    // 3. the passer, if any, is among the failures
                    for (int f = 0; f < nfail && result < 0 && !full; ++f) {
                        const int e = fails[f];
                        const D4 dc = S.pos[e];
                        const double dot = mdot(dc, x);
                        if (!(dot > 1e-10)) continue;
                        const double nc = S.nrm[e];
                        const double tau = __ddiv_rn(nc, dmul(2.0, dot));
                        if (!(tau > 0.0)) continue;
                        const double thf = theta_of(e, tau);
                        if (!(thf < kmax)) {
                            full = true;
                            break;
                        }
                        int dummy = 0;
                        if (verify(S.idx[e], e, dc, nc, thf, nullptr, dummy)) {
                            result = S.idx[e];
                            res_tau = tau;
                        }
                    }
                }
            }
        }
    }
    return result;
}

// Arguments of the two search kernels.
struct MaskArgs {
    const D4* bub;            // frames (kn, n_tot)
    size_t n_int, n_tot;
    const uint32_t* sel;
    const uint2* ranges;
    size_t n_sel;
    const NbList* lists;
    const D4* dirs;           // (n_rows, n_cols)
    const double* cosphi;     // GRID: per column
    const double* sinphi;
    int n_rows, n_cols;
    unsigned n_split;         // blocks per (bubble, frame)
    int rows_per_item, lane_cols;
    double* tau;
    int32_t* codes;           // may be null
    unsigned* open;           // per block: it left directions open (null: unknown)
    unsigned long long* counters;
};

// A delay that k_masks_list leaves for k_masks_rest (a decided one is positive or zero).
constexpr double kOpenTau = -1.0;

// Gathers a block's candidate list; false for a slot that radiates nothing.
__device__ __forceinline__ bool mask_block_fill(const MaskArgs& A, MaskBlock& S, int k, size_t slot) {
    const uint32_t a0 = A.sel[slot];
    const NbList* L = A.lists + slot;
    const int n = L->count;
    if (a0 >= A.n_int || n < 0) return false;
    const D4* B = A.bub + (size_t)k * A.n_tot;
    uint32_t a = a0;
    size_t n_tot = A.n_tot;
    if (A.ranges) {  // several realizations: this slot's colliders are its own realization's rows
        const uint2 r = A.ranges[slot];
        B += r.x;
        n_tot = r.y;
        a -= r.x;
    }
    const D4 xa = B[a];
    const int no = L->n_outliers;
    if (threadIdx.x == 0) {
        S.B = B;
        S.n_tot = n_tot;
        S.a = a;
        S.n = n;
        S.no = no;
        S.xa = xa;
        S.kmax = L->kmax;
        S.rho1 = L->rho1;
        S.rho2 = L->rho2;
        S.big = false;
        S.no_patch = no < 0;
        S.open = 0;
        S.next = 0;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < no; q += kMaskListThreads) {
        S.oidx[q] = L->outlier[q];
        const D4 dc = dsub4(B[L->outlier[q]], xa);
        S.opos[q] = dc;
        S.onrm[q] = mdot(dc, dc);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += kMaskListThreads) {
        const int c = L->idx[q];
        S.idx[q] = c;
        S.key[q] = L->key[q];
        const D4 dc = dsub4(B[c], xa);
        S.pos[q] = dc;
        const double nrm = mdot(dc, dc);
        S.nrm[q] = nrm;
        const double dx = sqrt(dc.x * dc.x + dc.y * dc.y + dc.z * dc.z);
        const double A1 = fabs(dc.t) + dx, Q = dc.t * dc.t + dx * dx;
        float4 f = make_float4(0.0f, 0.0f, 0.0f, CUDART_INF_F), v = make_float4(0.0f, CUDART_INF_F, CUDART_INF_F, 0.0f);
        bool aside = false;  // an outlier is checked by itself
        for (int e = 0; e < no; ++e) aside |= c == S.oidx[e];
        if (aside) {
            f.w = -CUDART_INF_F;
        } else if (nrm > 0.0) {  // any other collider keeps a form that is largest, which leaves the direction open
            const double inv = 1.0 / nrm, l1 = fabs(dc.t) + fabs(dc.x) + fabs(dc.y) + fabs(dc.z);
            const double w = 32.0 * 5.9604644775390625e-08 * l1 * inv, slope = theta_slope(S, dc, nrm);
            f = make_float4((float)(dc.x * inv), (float)(dc.y * inv), (float)(dc.z * inv), (float)(w - dc.t * inv));
            // max(A, Q) / d = 2 tau max(A, Q) / n <= 4e5, and theta < kmax (1e-6: these bounds' rounding).
            // A patch list ends at keys above T (1 + 1e-5), so theta = tau (1 + 1e-12 + slope) must not reach
            // further: only near-lightlike colliders have a slope of 1e-5 (most are below 1e-8), and the
            // directions that they decide take steps 1-3
            const double top = fmin(2e5 * nrm / fmax(A1, Q), S.kmax / (1.0 + 1e-12 + slope));
            v = make_float4((float)(dx * inv), __double2float_ru(2.0 * w), __double2float_ru(1e-9 * (A1 + Q) * inv),
                            slope < 9e-6 ? __double2float_rd((1.0 - 1e-6) * top) : 0.0f);
        }
        S.form[q] = f;
        S.fval[q] = v;
        if (!(fabs(dc.t) + fabs(dc.x) + fabs(dc.y) + fabs(dc.z) < 1e5)) S.big = S.no_patch = true;  // every writer: true
        if (dx > 0.0 && dx < 1e-15) S.no_patch = true;
    }
    __syncthreads();
    return true;
}

__device__ __forceinline__ int32_t mask_code(const MaskArgs& A, long result) {
    return result < 0 ? -1 : ((size_t)result < A.n_int ? (int32_t)result : -((int32_t)(result - A.n_int) + 2));
}

// A patch list's largest forms tie to within their FP32 error: the largest is checked against those it is
// not certified against with the reference's expression, and if it fails one of them, that one the same
// way.  Returns the list position of the collider that passes, -1: not decided here.
__device__ __noinline__ int resolve_tie(const MaskBlock& S, const float4* pform, const int* ppos, int n_patch,
                                        int best, D4 x) {
    const float xf = (float)x.x, yf = (float)x.y, zf = (float)x.z;
    for (int round = 0; round < 3; ++round) {
        const int q = ppos[best];
        const float4 fb = pform[best];
        const float cut = fmaf(fb.z, zf, fmaf(fb.y, yf, fmaf(fb.x, xf, fb.w))) - S.fval[q].y;
        const D4 dq = S.pos[q];
        const double nq = S.nrm[q];
        int fail = -1;
        for (int e = 0; e < n_patch && fail < 0; ++e) {
            const float4 f = pform[e];
            if (e == best || fmaf(f.z, zf, fmaf(f.y, yf, fmaf(f.x, xf, f.w))) < cut) continue;
            if (!check_pre(dq, nq, S.pos[ppos[e]], S.nrm[ppos[e]], x)) fail = e;
        }
        if (fail < 0) return q;
        best = fail;
    }
    return -1;
}

__device__ __noinline__ bool passes_outliers(const MaskBlock& S, int q, D4 x) {
    bool ok = true;
    for (int e = 0; e < S.no; ++e)
        if (S.oidx[e] != S.idx[q]) ok &= check_pre(S.pos[q], S.nrm[q], S.opos[e], S.onrm[e], x);
    return ok;
}

// Step 0 for every direction.  One block per (radiating bubble, range of its items, frame): the candidate
// list is gathered into shared memory once, then every warp takes items independently.  Directions that
// step 0 does not decide are marked and left to k_masks_rest: with steps 1-3 in this kernel (150 registers)
// it had 16 warps per SM and an issue slot in 2.5 used.
//
// GRID: the directions are the grid's, (1, s_i cos phi_j, s_i sin phi_j, c_i) with phi_0 = 0, and are formed
// from the rows' s_i and c_i (the table's first column) and the columns' cos phi_j and sin phi_j with the
// table's own products.  Read as they are, 32 bytes a direction (and again for the cap), they made L1 the
// bound of fine grids: 86 % busy, 0.96 ms for 2 frames of 512 bubbles x 192 x 192 directions.
template <bool GRID>
__global__ void __launch_bounds__(kMaskListThreads, kMaskBlocks) k_masks_list(MaskArgs A) {
    extern __shared__ __align__(16) unsigned char smem_mask[];
    MaskBlock& S = *reinterpret_cast<MaskBlock*>(smem_mask);
    const size_t slot = blockIdx.x / A.n_split;
    const unsigned part = blockIdx.x % A.n_split;
    const int lane = threadIdx.x & 31;
    const size_t at0 = ((size_t)blockIdx.y * A.n_sel + slot) * A.n_rows * A.n_cols;  // first direction of the pair
    const size_t block = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    if (!mask_block_fill(A, S, blockIdx.y, slot)) {  // invalid radiating bubble: sentinel outputs
        const size_t nd = (size_t)A.n_rows * A.n_cols;
        for (size_t d = nd * part / A.n_split + threadIdx.x; d < nd * (part + 1) / A.n_split; d += kMaskListThreads) {
            A.tau[at0 + d] = CUDART_NAN;
            if (A.codes) A.codes[at0 + d] = INT32_MIN;
        }
        if (threadIdx.x == 0 && A.open) A.open[block] = 0;
        return;
    }
    // Work items: lane_cols columns by up to rows_per_item rows, walked in tiles of 32 directions (lane_cols
    // columns by 32 / lane_cols rows).  The bubble's items are shared out over its blocks, a block's over
    // its warps by a counter.
    const int lane_rows = 32 / A.lane_cols;
    const int lane_r = lane / A.lane_cols;
    const int n_strips = (A.n_cols + A.lane_cols - 1) / A.lane_cols;
    const unsigned n_items = (unsigned)n_strips * (unsigned)((A.n_rows + A.rows_per_item - 1) / A.rows_per_item);
    const unsigned i_begin = (unsigned)((size_t)n_items * part / A.n_split);
    const unsigned i_end = (unsigned)((size_t)n_items * (part + 1) / A.n_split);
    float4* pform = S.pform[threadIdx.x >> 5];
    int* ppos = S.ppos[threadIdx.x >> 5];
    double cp = 1.0, sp = 0.0;  // the lane's column
    // what is loaded for a direction (its row's s and c, or all of it), and the direction
    auto fetch = [&](int row, int c) {
        const D4* v = A.dirs + (size_t)row * A.n_cols + (GRID ? 0 : c);
        return GRID ? D4{1.0, v->x, 0.0, v->z} : *v;
    };
    auto turn = [&](const D4& v, double cph, double sph) {
        return GRID ? D4{1.0, dmul(v.x, cph), dmul(v.x, sph), v.z} : v;
    };
    for (;;) {
      unsigned item = 0;
      if (lane == 0) item = atomicAdd(&S.next, 1u);
      item = i_begin + __shfl_sync(0xffffffffu, item, 0);
      if (item >= i_end) break;
      const int c_first = (int)(item % n_strips) * A.lane_cols;
      const int col = c_first + lane % A.lane_cols;
      const int c_mid = min(c_first + (A.lane_cols - 1) / 2, A.n_cols - 1);
      const int c_dir = col < A.n_cols ? col : c_mid;
      if constexpr (GRID) {
          cp = A.cosphi[c_dir];
          sp = A.sinphi[c_dir];
      }
      int r_first = (int)(item / n_strips) * A.rows_per_item;
      const int r_end = min(A.n_rows, r_first + A.rows_per_item);
      // an item whose patch list overflows is halved (down to one tile of rows)
      for (int len = A.rows_per_item; r_first < r_end;) {
      const int r_last = min(r_end, r_first + len) - 1;
      D4 v_next = fetch(min(r_first + lane_r, r_last), c_dir);
      float t_cut = -1.0f;  // least upper bound on a first collision's delay; < 0: no patch list
      int n_patch = 0;
      if (!S.no_patch) {
          // the cap: its axis is the item's middle direction, its radius covers every direction (FP32; the
          // margins below cover its roundings, a few 1e-7 each)
          const D4 ud = turn(fetch((r_first + r_last) >> 1, c_mid), GRID ? A.cosphi[c_mid] : 1.0,
                             GRID ? A.sinphi[c_mid] : 0.0);
          const float ux = (float)ud.x, uy = (float)ud.y, uz = (float)ud.z;
          float cr = 1.0f;
          auto widen = [&](const D4& v) { cr = fminf(cr, fmaf((float)v.z, uz, fmaf((float)v.y, uy, (float)v.x * ux))); };
          widen(turn(v_next, cp, sp));
          for (int r = r_first + lane_rows + lane_r; r <= r_last; r += lane_rows) widen(turn(fetch(r, c_dir), cp, sp));
          // order-preserving integers for the warp minimum (cr + 2 is positive)
          cr = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(cr + 2.0f))) - 2.0f;
          cr = fmaxf(cr - 2e-6f, -1.0f);
          const float sr = sqrtf((1.0f - cr) * (1.0f + cr)) + 1e-6f;
          // bounds on d / s = (dx.n - dt) / s over the cap, widened by 1e-5 (|dx| + |dt|) / s (the form's w too)
          auto bounds = [&](const float4& p, float r, float& d_lo, float& d_hi) {
              const float du = fmaf(p.z, uz, fmaf(p.y, uy, p.x * ux));
              const float vx = fmaf(p.y, uz, -p.z * uy), vy = fmaf(p.z, ux, -p.x * uz), vz = fmaf(p.x, uy, -p.y * ux);
              const float sn = __fsqrt_rn(fmaf(vz, vz, fmaf(vy, vy, vx * vx))) * sr;
              const float mg = 1e-5f * (r + fabsf(p.w));
              d_hi = (du < r * cr ? fmaf(du, cr, sn) : r) + p.w + mg;
              d_lo = (du > -r * cr ? fmaf(du, cr, -sn) : -r) + p.w - mg;
          };
          // T: the least 1 / (2 D-) over the list (its first 32 entries' values are kept)
          float4 f0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          float hi0 = 0.0f;
          unsigned T = 0x7f800000u;  // bits of a positive float order as the float does
          for (int e0 = 0; e0 < S.n && S.key[e0] <= (double)__uint_as_float(T); e0 += 32) {
              const int e = e0 + lane;
              unsigned t = 0x7f800000u;
              if (e < S.n) {
                  const float4 f = S.form[e];
                  float lo, hi;
                  bounds(f, S.fval[e].x, lo, hi);
                  if (lo > 0.0f && lo < CUDART_INF_F) t = __float_as_uint(__fdividef(0.500005f, lo));
                  if (e0 == 0) {
                      f0 = f;
                      hi0 = hi;
                  }
              }
              T = min(T, __reduce_min_sync(0xffffffffu, t));
          }
          t_cut = __uint_as_float(T);
          const double last = (double)t_cut * (1.0 + 1e-5);
          for (int e0 = 0; e0 < S.n && S.key[e0] <= last; e0 += 32) {
              const int e = e0 + lane;
              bool keep = false;
              float4 f = f0;
              if (e < S.n) {
                  float lo, hi = hi0;
                  const float4 v = S.fval[e];
                  if (e0) {
                      f = S.form[e];
                      bounds(f, v.x, lo, hi);
                  }
                  // 1 / 2 - T max(D+, 0) > margin (over s), with the FP32 roundings on the side of keeping
                  const float reach = hi > 0.0f ? t_cut * hi : 0.0f;
                  keep = !(0.5f - reach > v.z + 2e-6f * (0.5f + reach));
              }
              const unsigned m = __ballot_sync(0xffffffffu, keep);
              const int at = n_patch + __popc(m & ((1u << lane) - 1u));
              if (keep && at < kPatchList) {
                  pform[at] = f;
                  ppos[at] = e;
              }
              n_patch += __popc(m);
          }
          if (n_patch > kPatchList && len > lane_rows && r_last > r_first) {
              len = max(lane_rows, len >> 1);
              continue;
          }
          if (n_patch > kPatchList) t_cut = -1.0f;  // one tile of rows: the whole list is used
          __syncwarp();
      }
      for (int rt = r_first; rt <= r_last; rt += lane_rows) {  // warp-uniform
        const int rw = rt + lane_r;
        const D4 x = turn(v_next, cp, sp);
        // the next tile's load is issued now, so that its latency overlaps the search
        if (rt + lane_rows <= r_last) v_next = fetch(min(rw + lane_rows, r_last), c_dir);
        double tau = kOpenTau;
        int q = -1;
        if (!S.no_patch) {
            const float xf = (float)x.x, yf = (float)x.y, zf = (float)x.z;
            float g1 = -CUDART_INF_F, g2 = -CUDART_INF_F;
            int best = 0;
            auto visit = [&](const float4& f, int e) {
                const float g = fmaf(f.z, zf, fmaf(f.y, yf, fmaf(f.x, xf, f.w)));
                g2 = fmaxf(g2, fminf(g, g1));
                best = g > g1 ? e : best;
                g1 = fmaxf(g1, g);
            };
            if (t_cut >= 0.0f) {
#pragma unroll 4
                for (int e = 0; e < n_patch; ++e) visit(pform[e], e);
                q = n_patch ? ppos[best] : -1;
            } else {
                // the whole list, until the keys exceed every lane's delay and its bound theta (2 w < 0.01 g below
                // and slope < 1e-5, so both are under 0.52 / g)
                for (int e0 = 0; e0 < S.n; e0 += 16) {
                    const unsigned t = g1 > 0.0f ? __float_as_uint(__fdividef(0.52f, g1)) : 0x7f800000u;
                    if (e0 && S.key[e0] > (double)__uint_as_float(__reduce_max_sync(0xffffffffu, t))) break;
                    for (int e = e0; e < min(e0 + 16, S.n); ++e) visit(S.form[e], e);
                }
                q = best;
            }
            // no collider: every form negative and the list complete
            if (g1 <= 0.0f && (t_cut < 0.0f || t_cut == CUDART_INF_F) && S.kmax == CUDART_INF && S.no == 0) {
                tau = 0.0;
                q = -1;
            }
            if (q >= 0) {
                const float w2 = S.fval[q].y;
                bool sure = g2 < g1 - w2;
                if (t_cut < 0.0f) {
                    sure = sure && w2 < 0.01f * g1;
                } else if (!sure) {
                    const int r = resolve_tie(S, pform, ppos, n_patch, best, x);
                    sure = r >= 0;
                    q = sure ? r : q;
                }
                const double dd = mdot(S.pos[q], x);
                // tau with the reference's operations (compute_delta_tab, GBF:457-466)
                const double tq = __ddiv_rn(S.nrm[q], dmul(2.0, dd));
                const float top = t_cut >= 0.0f ? fminf(t_cut, S.fval[q].w) : S.fval[q].w;
                // (tq > 0: a null or timelike collider passes every check with a delay that is not positive)
                if (sure && dd > 1e-10 && tq > 0.0 && __double2float_ru(tq) <= top &&
                    (S.no == 0 || passes_outliers(S, q, x)))
                    tau = tq;
            }
        }
        if (rw <= r_last && col < A.n_cols) {
            const size_t d = at0 + (size_t)rw * A.n_cols + col;
            A.tau[d] = tau;
            if (tau == kOpenTau)
                S.open = 1;  // every writer stores 1
            else if (A.codes)
                A.codes[d] = q < 0 ? -1 : mask_code(A, S.idx[q]);
        }
      }
      r_first = r_last + 1;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0 && A.open) A.open[block] = S.open;
}

// Steps 1-3 for the directions that k_masks_list left open (2.5 in 1e5 of the benchmark configurations').
__global__ void __launch_bounds__(kMaskListThreads) k_masks_rest(MaskArgs A) {
    extern __shared__ __align__(16) unsigned char smem_mask[];
    MaskBlock& S = *reinterpret_cast<MaskBlock*>(smem_mask);
    if (A.open && !A.open[(size_t)blockIdx.y * gridDim.x + blockIdx.x]) return;
    const size_t slot = blockIdx.x / A.n_split;
    const unsigned part = blockIdx.x % A.n_split;
    if (!mask_block_fill(A, S, blockIdx.y, slot)) return;
    const int lane = threadIdx.x & 31;
    const size_t at0 = ((size_t)blockIdx.y * A.n_sel + slot) * A.n_rows * A.n_cols;
    const int lane_rows = 32 / A.lane_cols;
    const int n_strips = (A.n_cols + A.lane_cols - 1) / A.lane_cols;
    const unsigned n_items = (unsigned)n_strips * (unsigned)((A.n_rows + A.rows_per_item - 1) / A.rows_per_item);
    const unsigned i_begin = (unsigned)((size_t)n_items * part / A.n_split);
    const unsigned i_end = (unsigned)((size_t)n_items * (part + 1) / A.n_split);
    // directions that left the list, for the exhaustive scan: a warp takes one at a time, and those of a
    // block are shared out over its warps (368 neighbouring ones, one warp's 32 in turn, took 4.8 ms)
    constexpr unsigned kQueue = 1024;
    __shared__ size_t queue[kQueue];
    __shared__ unsigned queued;
    if (threadIdx.x == 0) queued = 0;
    __syncthreads();
    auto put = [&](size_t at, long result, double tau) {
        A.tau[at0 + at] = result >= 0 ? tau : 0.0;
        if (A.codes) A.codes[at0 + at] = mask_code(A, result);
    };
    auto scan = [&](size_t at) {  // by a whole warp
        const D4 x = A.dirs[at];
        const long result = exhaustive_warp(S.B, S.n_tot, S.a, S.xa, x);
        if (lane) return;
        double tau = 0.0;
        if (result >= 0) {
            // compute_delta_tab (GBF:457-466)
            const D4 dba = dsub4(S.B[result], S.xa);
            const double dot = mdot(dba, x);
            tau = fabs(dot) < 1e-10 ? 0.0 : __ddiv_rn(mdot(dba, dba), dmul(2.0, dot));
        }
        put(at, result, tau);
        atomicAdd(A.counters, 1ull);
    };
    for (unsigned item = i_begin + (threadIdx.x >> 5); item < i_end; item += kMaskListThreads / 32) {
        const int col = (int)(item % n_strips) * A.lane_cols + lane % A.lane_cols;
        const int r_first = (int)(item / n_strips) * A.rows_per_item;
        const int r_end = min(A.n_rows, r_first + A.rows_per_item);
        for (int rt = r_first; rt < r_end; rt += lane_rows) {  // warp-uniform
            const int rw = rt + lane / A.lane_cols;
            const size_t at = (size_t)rw * A.n_cols + col;
            const bool need = rw < r_end && col < A.n_cols && A.tau[at0 + at] == kOpenTau;
            bool full = false;
            if (need) {
                double tau;
                const long result = decide_slow(S, A.dirs[at], tau, full);
                if (!full) put(at, result, tau);
            }
            unsigned pos = full ? atomicAdd(&queued, 1u) : 0u;
            if (full && pos < kQueue) queue[pos] = at;
            for (unsigned h = __ballot_sync(0xffffffffu, full && pos >= kQueue); h; h &= h - 1)
                scan(__shfl_sync(0xffffffffu, at, __ffs(h) - 1));
        }
    }
    __syncthreads();
    for (unsigned q = threadIdx.x >> 5; q < min(queued, kQueue); q += kMaskListThreads / 32) scan(queue[q]);
}

template <bool GRID>
static void launch_search(const MaskArgs& A, size_t kn, cudaStream_t stream) {
    const size_t gx = (size_t)A.n_split * A.n_sel;
    if (gx > 0x7fffffffULL || kn > 65535) throw Error{"too many (bubble, patch) pairs for one launch"};
    const dim3 grid((unsigned)gx, (unsigned)kn);
    // more shared memory than the 48 KB a kernel may use without asking
    allow_shared(k_masks_list<GRID>, sizeof(MaskBlock));
    allow_shared(k_masks_rest, sizeof(MaskBlock));
    k_masks_list<GRID><<<grid, kMaskListThreads, sizeof(MaskBlock), stream>>>(A);
    CUDA_OK(cudaGetLastError());
    k_masks_rest<<<grid, kMaskListThreads, sizeof(MaskBlock), stream>>>(A);
    CUDA_OK(cudaGetLastError());
}

// Items and blocks of the search.  An item is a patch of at most about 1/64 of the sphere (a larger one
// keeps more colliders in its list: 16 x 32 directions of a 64 x 64 grid needed 360 and overflowed it), at
// most 256 directions (the list costs about 400 instructions, a direction about 150): 8 columns by 4 to 32
// rows, or 32 columns of one row when the directions have no rows.  Blocks take eight items (one per warp)
// or more, up to about 16384 directions, once there are eight blocks per SM: each gathers the candidate list.
struct MaskShape {
    int rows_per_item, lane_cols;
    unsigned n_split;
};
static MaskShape mask_shape(size_t nd, size_t row_len, size_t n_pairs, int n_sm, int chunking) {
    const size_t fill = 8 * (size_t)n_sm;  // eight blocks per SM
    const size_t n_rows = nd / row_len;
    MaskShape m;
    m.lane_cols = n_rows >= 4 ? 8 : 32;
    m.rows_per_item = 32 / m.lane_cols;
    while (m.rows_per_item < 32 && (size_t)(m.lane_cols * m.rows_per_item) * 96 < nd) m.rows_per_item *= 2;
    if (n_rows < 4) m.rows_per_item = 1;
    const size_t strips = (row_len + m.lane_cols - 1) / m.lane_cols;
    // few bubbles: smaller items, so that every SM has a few
    size_t groups = (n_rows + m.rows_per_item - 1) / m.rows_per_item;
    while (m.rows_per_item > 32 / m.lane_cols && n_pairs * strips * groups < fill) {
        m.rows_per_item /= 2;
        groups = (n_rows + m.rows_per_item - 1) / m.rows_per_item;
    }
    const size_t total = strips * groups;  // of one bubble and frame
    if (total * m.lane_cols > 0x7fffffffULL) throw Error{"too many directions for the mask search"};
    const size_t items = std::min<size_t>(std::max<size_t>(8, n_pairs * total / fill),
                                          std::max<size_t>(8, 16384 / (m.lane_cols * m.rows_per_item)));
    // the launch shape may ask for 2 or 4 times the automatic number of blocks
    m.n_split = (unsigned)std::min(total, (total + items - 1) / items * (size_t)std::max(1, std::min(chunking, 4)));
    return m;
}

// ------------------------------------------------------------------ host
void launch_masks_with_lists(cudaStream_t stream, const D4* bub, size_t n_int, size_t n_tot, const uint32_t* sel,
                             size_t n_sel, const D4* dirs, size_t nd, NbList* lists, double* tau, int32_t* codes,
                             unsigned long long* counters, int n_sm) {
    if (n_tot < 2) {
        CUDA_OK(cudaMemsetAsync(tau, 0, n_sel * nd * sizeof(double), stream));
        if (codes) CUDA_OK(cudaMemsetAsync(codes, 0xff, n_sel * nd * sizeof(int32_t), stream));
        return;
    }
    launch_neighbors(bub, n_int, n_tot, sel, nullptr, n_sel, lists, stream);
    // the directions' row structure is not known here: one row of nd directions
    if (nd > 0x7fffffffULL) throw Error{"too many directions for the mask search"};
    const MaskShape shape = mask_shape(nd, nd, n_sel, n_sm, 1);
    const MaskArgs A{bub,  n_int,   n_tot,          sel,           nullptr,         n_sel, lists, dirs,    nullptr, nullptr,
                     1,    (int)nd, shape.n_split, shape.rows_per_item, shape.lane_cols, tau,   codes, nullptr, counters};
    launch_search<false>(A, 1, stream);
}

void launch_mask_pipeline(Device* dev, const D4* bub_unrot, const D4* bub_frames, size_t n_int, size_t n_tot,
                          const uint32_t* sel, const uint2* ranges, size_t n_sel, const D4* dirs,
                          const double* cosphi, const double* sinphi, size_t nd, size_t row_len, size_t kn, double* tau, int32_t* codes, unsigned long long* counters,
                          bool build_lists, uint64_t* launches, int chunking) {
    if (n_tot < 2) {
        // a lone bubble has no collider: every direction is None
        CUDA_OK(cudaMemsetAsync(tau, 0, kn * n_sel * nd * sizeof(double), dev->stream));
        if (codes) CUDA_OK(cudaMemsetAsync(codes, 0xff, kn * n_sel * nd * sizeof(int32_t), dev->stream));
        return;
    }
    dev->nblists.ensure(n_sel * sizeof(NbList));
    if (build_lists) {
        launch_neighbors(bub_unrot, n_int, n_tot, sel, ranges, n_sel, (NbList*)dev->nblists.p, dev->stream);
        if (launches) ++*launches;
    }
    const MaskShape shape = mask_shape(nd, row_len, n_sel * kn, dev->n_sm, chunking);
    dev->mask_open.ensure(n_sel * kn * shape.n_split * sizeof(unsigned));
    const MaskArgs A{bub_frames,
                     n_int,
                     n_tot,
                     sel,
                     ranges,
                     n_sel,
                     (const NbList*)dev->nblists.p,
                     dirs,
                     cosphi,
                     sinphi,
                     (int)(nd / row_len),
                     (int)row_len,
                     shape.n_split,
                     shape.rows_per_item,
                     shape.lane_cols,
                     tau,
                     codes,
                     (unsigned*)dev->mask_open.p,
                     counters};
    launch_search<true>(A, kn, dev->stream);
    if (launches) *launches += 2;
}

}  // namespace bgw
