"""Handles used by several host threads at once (the library call runs without the interpreter's lock)."""
import threading

import numpy as np
import pytest

from gw_fopt_b200 import many_bubbles as mb
from gw_fopt_b200 import workloads as W

pytestmark = pytest.mark.gpu


def flow(interior, n_cos, n_phi, kernel="fp64_direct"):
    g = mb.GeneralizedBulkFlow(mb.LatticeBubbles(mb.EmptyLattice(), interior))
    g.set_resolution(n_cos, n_phi)
    g.set_gradient_scaling_params([[1.0]], [[3.0]], None)
    g.set_kernel(kernel)
    return g


# Calls whose kernels need different amounts of shared memory: few and many colliders, few and many rows or
# patches.  Every thread gets its own results, and no launch is refused: the large call's, in one thread, beside
# five that make small calls all the while.
@pytest.mark.parametrize("kind", ["colliders", "rows", "factored", "mixed"])
def test_threads_of_different_sizes(gpu_available, kind):
    w = np.array([1.0, 7.0])
    b, _ = W.uniform_config(8, 1.0, 0.05, seed=4)

    def call(large):
        if kind == "colliders":
            n, rng = 8000 if large else 40, np.random.default_rng(3)
            g = flow(np.column_stack([np.zeros(n), rng.random((n, 3))]), 4, 4)
            return lambda: g.compute_first_colliding_bubble(0)
        g = flow(b, 2000 if large and kind == "rows" else 9, 600 if large and kind != "rows" else 8,
                 "fp64_direct" if kind == "rows" else "fp64_factored" if kind == "factored" else "mixed")
        return lambda: g.compute_c_integral(w, t_begin=0.0, t_end=1.2, n_t=20)
    done, errors = threading.Event(), []

    def work(large):
        try:
            c = call(large)
            ref = c()
            start.wait()
            for _ in range(2500 if large else 10 ** 9):
                if not np.array_equal(c(), ref):
                    raise AssertionError("another result")
                if done.is_set():
                    break
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            errors.append((large, e))
            start.abort()
        if large or errors:
            done.set()
    start = threading.Barrier(6)
    threads = [threading.Thread(target=work, args=(q == 0,)) for q in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
