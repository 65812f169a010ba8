"""Kernels at the sizes where their tiling can go wrong, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from gw_fopt_b200 import many_bubbles as mb
from gw_fopt_b200 import workloads as W


def flow(interior, exterior, n_cos, n_phi, coeffs, powers, damping=None, kernel="fp64_direct", cls=mb.GeneralizedBulkFlow):
    g = cls(mb.LatticeBubbles(mb.EmptyLattice(), interior, exterior))
    g.set_resolution(n_cos, n_phi)
    g.set_gradient_scaling_params([list(map(float, r)) for r in coeffs], [list(map(float, r)) for r in powers], damping)
    g.set_kernel(kernel)
    return g


def per_w(got, ref):
    g, r = got.reshape(-1, got.shape[-1]), ref.reshape(-1, ref.shape[-1])
    return float(np.max(np.linalg.norm(g - r, axis=0) / np.linalg.norm(r, axis=0)))


@pytest.mark.gpu
@pytest.mark.parametrize("sets", [2, 3, 5, 6, 7])
def test_mixed_sets_straddling_the_column_halves(gpu_available, sets):
    """With 3, 5, 6 or 7 sets a bubble's columns straddle the GEMM's two 64-column halves (bubble
    10 of 21 with 3 sets): both halves' sums use that bubble's own phases, in every run.  1e-6 per
    w is the mixed kernel's stated error."""
    b, e = W.exponential_nucleation(30, 5.0, seed=7, max_rejections=20000)
    w = np.geomspace(1.0, 200.0, 70)
    co, po = [[1.0]] * sets, [[5.0 - 0.3 * s] for s in range(sets)]
    ref = O.compute_c_integral(b, e, 40, 24, w, 1.5, 70, t_begin=0.0, coefficients=co, powers=po)
    g = flow(b, e, 40, 24, co, po, kernel="mixed")
    got = [g.compute_c_integral(w, t_begin=0.0, t_end=1.5, n_t=70) for _ in range(8)]
    assert per_w(got[0], ref) < 1e-6
    assert all(np.array_equal(got[0], o) for o in got[1:])


def first_colliders(interior, exterior, n_cos, n_phi, a0, a1):
    import ctypes as C
    from gw_fopt_b200 import _lib as L
    g = flow(interior, exterior, n_cos, n_phi, [[1.0]], [[3.0]])
    codes = np.empty((a1 - a0, n_cos, n_phi), dtype=np.int32)
    tau = np.empty((a1 - a0, n_cos, n_phi))
    L.check(L.lib().bgwx_generalized_bulk_flow_first_colliding(
        g._h, a0, a1, codes.ctypes.data_as(C.POINTER(C.c_int32)), tau.ctypes.data_as(C.POINTER(C.c_double))))
    return codes, tau


# Patches of directions and their lists: grids below and above one tile (8 x 4), with remainders, items of
# 4 to 32 rows, two rows only; one bubble and several; with images (late collisions towards the corners
# overflow the list), without (directions that meet nothing), a list that is complete and one that is not,
# and mirror-symmetric positions (exact ties at the mirror planes).
@pytest.mark.gpu
@pytest.mark.parametrize("n_cos,n_phi", [(2, 2), (2, 33), (3, 70), (5, 9), (33, 8), (40, 41), (97, 66), (200, 60)])
@pytest.mark.parametrize("kind", ["images", "alone", "many", "mirror"])
def test_first_colliders_bitwise(gpu_available, n_cos, n_phi, kind):
    if kind == "many":
        b, e = W.exponential_nucleation(300, 7.0, seed=3, max_rejections=20000)
    else:
        b, e = W.exponential_nucleation(20, 5.0, seed=9, max_rejections=20000)
    if kind in ("alone", "mirror"):
        e = np.zeros((0, 4))
    if kind == "mirror":
        x = b[:6, 1:4] - 0.5
        b = np.array([[0.0, sx * p[0], sy * p[1], sz * p[2]] for p in x[:4] for sx in (1, -1) for sy in (1, -1)
                      for sz in (1, -1)])
        b = np.concatenate([[[0.0, 0.0, 0.0, 0.0]], b[np.linalg.norm(b[:, 1:], axis=1) > 0.05]])
    codes, tau = first_colliders(b, e, n_cos, n_phi, 0, 3)
    rc, rt = O.first_colliding(b, e, n_cos, n_phi, 0, 3, with_delta_tab=True)
    assert np.array_equal(codes, rc)
    assert np.array_equal(tau, rt)


EPS = 2.0 ** -52


def spectrum_bound(absout, w, extent, powers):
    """Rounding of a sum of |term| = absout whose phase w (t - z - dt c) and power r^p are rounded at each
    step: both sides form the phase from a few operations of size |w| extent (8 half-ulps) and the scaling
    from a power (its exponent |p ln r| <= 8 |p|) and some tens of multiplications."""
    return EPS * (64.0 + 8.0 * np.max(np.abs(powers)) + 8.0 * np.abs(w)[None, None, :] * extent) * absout


# The direct kernel at the edges of its work split: two, three and odd numbers of rows (rows c and -c are
# taken together, the middle one alone), steps around 32 and 128, one frequency and remainders of four, one
# to four sets and terms, damping; the powers, dampings and frequencies that take its general formulas
# (|p| > 16, a width of a fraction of a step, |w| extent beyond 1e9).
@pytest.mark.gpu
@pytest.mark.parametrize("n_cos,n_phi,n_t,n_w,sets,terms,damping", [
    (2, 2, 2, 1, 1, 1, None), (3, 5, 31, 2, 1, 2, None), (5, 33, 32, 3, 2, 1, 0.7), (16, 20, 33, 4, 3, 1, None),
    (17, 70, 127, 5, 4, 1, None), (8, 9, 128, 9, 1, 3, 0.2), (9, 64, 129, 33, 2, 2, None), (4, 3, 300, 66, 5, 2, None),
    (9, 12, 40, 5, 1, 1, 0.002)])
@pytest.mark.parametrize("powers,w_max", [(3.5, 300.0), (20.0, 50.0), (3.0, 3e9)])
def test_direct_edges(gpu_available, n_cos, n_phi, n_t, n_w, sets, terms, damping, powers, w_max):
    b, e = W.exponential_nucleation(8, 4.0, seed=21, max_rejections=20000)
    w = np.geomspace(0.3, w_max, n_w) if n_w > 1 else np.array([w_max])
    co = [[1.0 - 0.2 * s + 0.1 * m for m in range(terms)] for s in range(sets)]
    po = [[powers - 0.3 * s - 0.25 * m for m in range(terms)] for s in range(sets)]
    ref, mag = O.compute_c_integral(b, e, n_cos, n_phi, w, 1.7, n_t, t_begin=0.0, coefficients=co, powers=po,
                                    damping=damping, want_abs=True)
    got = flow(b, e, n_cos, n_phi, co, po, damping).compute_c_integral(w, t_begin=0.0, t_end=1.7, n_t=n_t)
    assert np.all(np.abs(got - ref) <= spectrum_bound(mag, w, 3.0, po))


# The FP64 factored path: step segments of 128 with and without events, patches below, at and beyond a
# warp's registers, an even and an odd number of steps about the middle of the grid, more rows than row
# parts and fewer.  An uncollided sum is a row total less the patches that collided, so beside the bound
# above it carries 2 n_phi roundings of the largest terms: 1e-12 of the sum of magnitudes holds both.
@pytest.mark.gpu
@pytest.mark.parametrize("n_cos,n_phi,n_t,n_w,sets,terms,damping", [
    (2, 2, 2, 1, 1, 1, None), (3, 31, 3, 2, 1, 2, None), (7, 32, 64, 5, 2, 1, 0.7), (8, 33, 65, 17, 3, 1, None),
    (33, 64, 127, 8, 4, 1, None), (9, 65, 128, 9, 1, 4, 0.4), (16, 129, 129, 64, 2, 2, None),
    (130, 193, 257, 70, 1, 1, None), (17, 250, 300, 65, 4, 2, None)])
def test_factored_edges(gpu_available, n_cos, n_phi, n_t, n_w, sets, terms, damping):
    b, e = W.exponential_nucleation(10, 4.0, seed=22, max_rejections=20000)
    w = np.geomspace(0.3, 60.0, n_w) if n_w > 1 else np.array([20.0])
    co = [[1.0 - 0.2 * s + 0.1 * m for m in range(terms)] for s in range(sets)]
    po = [[5.0 - 0.3 * s - 0.25 * m for m in range(terms)] for s in range(sets)]
    ref, mag = O.compute_c_integral(b, e, n_cos, n_phi, w, 1.6, n_t, t_begin=0.0, coefficients=co, powers=po,
                                    damping=damping, want_abs=True)
    g = flow(b, e, n_cos, n_phi, co, po, damping, kernel="fp64_factored")
    got = g.compute_c_integral(w, t_begin=0.0, t_end=1.6, n_t=n_t)
    assert np.all(np.abs(got - ref) <= 1e-12 * mag)


# The mixed path's digits from both of its event kernels: the one whose masks are read again by the
# adjoint and the other.  1e-6 per w is the mixed kernel's stated error.
@pytest.mark.gpu
@pytest.mark.parametrize("n_cos,n_phi,n_t,sets,terms", [
    (9, 31, 40, 1, 1), (16, 64, 128, 1, 2), (33, 70, 129, 2, 1), (40, 200, 300, 2, 2), (64, 65, 255, 4, 1)])
@pytest.mark.parametrize("kept", [False, True])
def test_mixed_edges(gpu_available, n_cos, n_phi, n_t, sets, terms, kept):
    import torch
    from gw_fopt_b200.autograd import BulkFlowSpectrum
    b, _ = W.uniform_config(20, 1.0, 0.05, seed=4)
    e = W.periodic_images(b, 1.0)
    w = np.geomspace(1.0, 40.0, 12)
    kh = W.fibonacci_khat(2)
    co = np.array([[1.0 - 0.2 * s + 0.1 * m for m in range(terms)] for s in range(sets)])
    po = np.array([[4.0 - 0.3 * s - 0.25 * m for m in range(terms)] for s in range(sets)])
    ref = O.compute_c_integral_khat(b, e, kh, n_cos, n_phi, w, 0.0, 1.2, n_t, coefficients=co, powers=po)
    if kept:
        m = BulkFlowSpectrum(n_cos=n_cos, n_phi=n_phi, w=w, khat=kh, t_begin=0.0, t_end=1.2, n_t=n_t, box=1.0,
                             kernel="mixed")
        t = [torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in (co, po, b)]
        got = m(*t).detach().numpy()
        got = got[..., 0] + 1j * got[..., 1]
    else:
        got = flow(b, e, n_cos, n_phi, co, po, kernel="mixed").compute_c_integral_khat(
            w, kh, t_begin=0.0, t_end=1.2, n_t=n_t)
    assert per_w(got, ref) < 1e-6


# The adjoint's two products and row sums: rows of a bubble split over two 64-row tiles (three sets), one
# tile and a remainder of steps, frequencies around a stage of 16 and too many to keep in shared memory
# (more than 77), steps around the chunks of 64, one to eight patches a lane.  The bounds are the ones of
# the library-against-oracle comparison: both sides sum in 64 bits.
@pytest.mark.gpu
@pytest.mark.parametrize("n,n_cos,n_phi,n_t,n_w,sets,terms,damping", [
    (24, 5, 7, 24, 5, 3, 1, None), (23, 4, 33, 64, 16, 3, 1, 0.8), (9, 6, 9, 65, 17, 4, 1, None),
    (12, 3, 70, 130, 100, 1, 1, None), (3, 4, 140, 63, 80, 2, 2, None), (17, 2, 5, 2, 1, 2, 1, 0.5),
    (2, 3, 256, 129, 3, 1, 4, None)])
def test_adjoint_edges(gpu_available, n, n_cos, n_phi, n_t, n_w, sets, terms, damping):
    from oracle import adjoint as OA
    from gw_fopt_b200.autograd import BulkFlowSpectrum
    b, _ = W.uniform_config(n, 1.0, 0.05, seed=6)
    e = W.periodic_images(b, 1.0)
    w = np.geomspace(1.0, 60.0, n_w) if n_w > 1 else np.array([7.0])
    kh = W.fibonacci_khat(2)
    co = np.array([[1.0 - 0.2 * s + 0.1 * m for m in range(terms)] for s in range(sets)])
    po = np.array([[5.0 - 0.3 * s - 0.25 * m for m in range(terms)] for s in range(sets)])
    rng = np.random.default_rng(8)
    G = rng.normal(size=(2, 2, sets, n_w)) + 1j * rng.normal(size=(2, 2, sets, n_w))
    m = BulkFlowSpectrum(n_cos=n_cos, n_phi=n_phi, w=w, khat=kh, t_begin=0.0, t_end=1.5, n_t=n_t, box=1.0,
                         damping=damping, kernel="fp64_factored")
    got = m.vjp(co, po, b, G)
    oc, op, ob = OA.spectrum_vjp(b, e, kh, n_cos, n_phi, w, 0.0, 1.5, n_t, G, co, po, damping=damping)
    for g, r in zip(got, (oc, op, ob[:n] + ob[n:].reshape(n, 6, 4).sum(1))):
        assert np.allclose(g, r, rtol=1e-9, atol=1e-12 * np.abs(r).max())
