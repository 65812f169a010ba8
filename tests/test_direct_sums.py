"""The direct FP64 kernel's sums: what is added to what depends on the call's grids alone."""
import numpy as np
import pytest

from gw_fopt_b200 import many_bubbles as mb
from gw_fopt_b200 import workloads as W

pytestmark = pytest.mark.gpu


def flow(n, n_cos, n_phi, sets, cls=mb.GeneralizedBulkFlow):
    b, e = W.exponential_nucleation(n, 5.0, seed=11, max_rejections=20000)
    g = cls(mb.LatticeBubbles(mb.EmptyLattice(), b, e))
    g.set_resolution(n_cos, n_phi)
    g.set_gradient_scaling_params([[1.0]] * sets, [[4.0 - 0.4 * s] for s in range(sets)], None)
    return g


# One direction's spectrum has the same bits alone, among others and with any number of frames per launch,
# in jobs of few and of many (bubble, direction) pairs.
@pytest.mark.parametrize("n,n_cos,n_t,n_w,sets", [
    (64, 64, 256, 64, 3), (40, 9, 300, 70, 1), (90, 16, 129, 130, 2), (3, 5, 40, 9, 1)])
@pytest.mark.parametrize("tensor", [False, True])
def test_frames_have_the_same_bits_alone(gpu_available, n, n_cos, n_t, n_w, sets, tensor):
    g = flow(n, n_cos, 16, sets, mb.NewGeneralizedBulkFlow if tensor else mb.GeneralizedBulkFlow)
    w, kh = np.geomspace(0.5, 200.0, n_w), W.fibonacci_khat(6)
    call = g.compute_c_tensor_khat if tensor else g.compute_c_integral_khat
    together = call(w, kh, t_begin=0.0, t_end=1.5, n_t=n_t)
    for q in (0, 3, 5):
        assert np.array_equal(call(w, kh[q:q + 1], t_begin=0.0, t_end=1.5, n_t=n_t)[0], together[q])
    g.set_launch_shape(2, 0)
    assert np.array_equal(call(w, kh, t_begin=0.0, t_end=1.5, n_t=n_t), together)
