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
