"""The direct FP64 kernel's work arrays: cut into ranges of pairs and of steps, and to the memory that is free."""
import numpy as np
import pytest

from gw_fopt_b200 import many_bubbles as mb
from gw_fopt_b200 import workloads as W

pytestmark = pytest.mark.gpu

SETS = 8  # 16 columns: B takes 128 bytes per (pair, row, step)


def flow(n, n_cos, n_phi, sets=SETS):
    b, e = W.uniform_config(n, 1.0, 0.05, seed=2)
    g = mb.GeneralizedBulkFlow(mb.LatticeBubbles(mb.EmptyLattice(), b, np.zeros((0, 4))))
    g.set_resolution(n_cos, n_phi)
    g.set_gradient_scaling_params([[1.0]] * sets, [[5.0 - 0.3 * s] for s in range(sets)], None)
    return g


W3 = np.array([1.0, 20.0, 90.0])


# 24 bubbles x 6 directions x 64 rows x 1024 steps: 1.2 GB of B, so two ranges of pairs at least.  Each
# direction alone needs 0.2 GB.
def test_ranges_of_pairs(gpu_available):
    kh = W.fibonacci_khat(6)
    g = flow(24, 64, 8)
    together = g.compute_c_integral_khat(W3, kh, t_begin=0.0, t_end=1.5, n_t=1024)
    for q in range(6):
        alone = g.compute_c_integral_khat(W3, kh[q:q + 1], t_begin=0.0, t_end=1.5, n_t=1024)
        assert np.array_equal(alone[0], together[q])


# 4096 rows: 1.15 GB of B for one pair's 2200 steps, so two ranges of steps; one set alone needs 0.14 GB.
def test_ranges_of_steps(gpu_available):
    got = flow(2, 4096, 8).compute_c_integral(W3, t_begin=0.0, t_end=1.5, n_t=2200)
    one = flow(2, 4096, 8, 1).compute_c_integral(W3, t_begin=0.0, t_end=1.5, n_t=2200)
    assert np.all(np.abs(got[:, 0] - one[:, 0]) <= 1e-12 * np.abs(one[:, 0]).max())


# The integrand's sum over the steps is the spectrum: ranges of pairs that cut a part's bubbles in two, and
# ranges of steps.
@pytest.mark.parametrize("n,n_cos,n_t", [(150, 64, 1024), (2, 4096, 2200)])
def test_integrand_ranges(gpu_available, n, n_cos, n_t):
    g = flow(n, n_cos, 8)
    step = g.compute_c_integrand(W3, t_begin=0.0, t_end=1.5, n_t=n_t)
    total = g.compute_c_integral(W3, t_begin=0.0, t_end=1.5, n_t=n_t)
    assert np.all(np.abs(step.sum(-1) - total) <= 1e-12 * np.abs(step).sum(-1).max())


# A job that would take 1 GiB of work arrays runs, with the same bits, on a card that has less left.
@pytest.mark.parametrize("left_mib", [700, 150])
def test_little_memory_left(gpu_available, left_mib):
    import torch
    kh = W.fibonacci_khat(6)

    def both():
        g = flow(24, 64, 8)
        i = flow(150, 64, 8)
        return (g.compute_c_integral_khat(W3, kh, t_begin=0.0, t_end=1.5, n_t=1024),
                i.compute_c_integrand(W3, t_begin=0.0, t_end=1.5, n_t=1024))
    ref = both()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (left_mib << 20), dtype=torch.uint8, device="cuda")
    try:
        got = both()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))
