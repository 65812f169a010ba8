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
