"""The direct FP64 kernel's phases: the table lookup, with the row of opposite cos theta taken from it to first order,
against the library's sine and cosine, which one more frequency beyond the table's range brings in for a whole call."""
import numpy as np
import pytest

from gw_fopt_b200 import many_bubbles as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

B = np.array([[0.0, 0.0, 0.0, 0.0], [0.1, 0.4, 0.3, 0.2], [0.05, -0.3, 0.2, 0.4]])


def sum_of_magnitudes(n_cos, n_phi, t):
    """(2, 1, 1): the magnitudes of the terms (bubble, row, step) of each polarisation, added up, for (tau / dt)^3."""
    _, tau = O.first_colliding(B, np.zeros((0, 4)), n_cos, n_phi, with_delta_tab=True)
    c, phi = np.linspace(-1.0, 1.0, n_cos), np.linspace(0.0, 2.0 * np.pi, n_phi)
    ends = lambda n: np.where((np.arange(n) == 0) | (np.arange(n) == n - 1), 0.5, 1.0)  # noqa: E731
    weights = np.stack([np.cos(2.0 * phi), np.sin(2.0 * phi)]) * ends(n_phi) * (2.0 * np.pi / n_phi)
    row = 0.5 * (1.0 - c * c) * ends(n_cos) * (2.0 / (n_cos - 1)) / (6.0 * np.pi)
    total = np.zeros(2)
    for a in range(B.shape[0]):
        for k, u in enumerate(ends(t.size) * (t[1] - t[0])):
            dt = t[k] - B[a, 0]
            if dt > 0.0:
                f = np.where((tau[a] > 0.0) & (dt >= tau[a]), (tau[a] / dt) ** 3, 1.0)
                total += (np.abs(f @ weights.T) * row[:, None]).sum(0) * dt ** 3 * u
    return total[:, None, None]


# Both calls form the same arguments, so they differ by the phases alone: two of each term (row and step), either
# within 1.5 half-ulps of 1 on either side, and by the roundings of a sum of at most n_cos rows.  In units of
# 2^-52 of the sum of the terms' magnitudes: 3 for the phases, 1 for their products, n_cos / 2 for the sums.
@pytest.mark.parametrize("n_cos", [6, 12, 20, 33, 193])
@pytest.mark.parametrize("largest", [1e3, 3.9e6, 3e7, 9.5e8])
def test_phases_against_the_library(gpu_available, n_cos, largest):
    g = mb.GeneralizedBulkFlow(mb.LatticeBubbles(mb.EmptyLattice(), B))
    g.set_resolution(n_cos, 4)
    g.set_gradient_scaling_params([[1.0]], [[3.0]], None)
    w = np.geomspace(0.3, 1.0, 200) * largest / 2.3  # times up to 1.7, positions within 0.6
    args = dict(t_begin=0.0, t_end=1.7, n_t=3)
    table = g.compute_c_integral(w, **args)
    library = g.compute_c_integral(np.append(w, 1e12), **args)[..., :-1]
    mag = sum_of_magnitudes(n_cos, 4, np.linspace(0.0, 1.7, 3))
    assert np.all(np.abs(table) <= 1.0001 * mag)
    assert np.all(np.abs(table - library) <= 2.0 ** -52 * (4.0 + 0.5 * n_cos) * mag)
