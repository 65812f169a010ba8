"""First-collider search where a collider is at or near the light cone, bit for bit against the oracle.

Both entry points are compared: the handle's, whose directions are the angular grid's rows, and the
allocation-free one, which takes the directions as a table and validates no bubbles.
"""
import ctypes as C
import math

import numpy as np
import pytest

from gw_fopt_b200 import _lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 4))


def by_handle(interior, n_cos, n_phi):
    lib, h, n = L.lib(), C.c_void_p(), interior.shape[0]
    interior = np.ascontiguousarray(interior)
    L.check(lib.bgwx_generalized_bulk_flow_new_unchecked(C.byref(h), L.ptr(interior), n, None, 0))
    try:
        L.check(lib.bgw_generalized_bulk_flow_set_resolution(h, n_cos, n_phi, False))
        codes = np.empty((n, n_cos, n_phi), dtype=np.int32)
        tau = np.empty((n, n_cos, n_phi))
        L.check(lib.bgwx_generalized_bulk_flow_first_colliding(
            h, 0, n, codes.ctypes.data_as(C.POINTER(C.c_int32)), L.ptr(tau)))
    finally:
        lib.bgw_generalized_bulk_flow_free(h)
    return codes, tau


def by_table(interior, n_cos, n_phi):
    import torch
    n, nd = interior.shape[0], n_cos * n_phi
    dirs = []
    for i in range(n_cos):
        c = -1.0 + (2.0 / (n_cos - 1)) * i
        s = abs(math.sqrt(1.0 - c * c))
        for j in range(n_phi):
            p = (2.0 * math.pi / (n_phi - 1)) * j
            dirs.append((1.0, s * math.cos(p), s * math.sin(p), c))
    dev = torch.device("cuda", 0)
    b = torch.tensor(interior, dtype=torch.float64, device=dev)
    d = torch.tensor(dirs, dtype=torch.float64, device=dev)
    sel = torch.arange(n, dtype=torch.int32, device=dev)
    codes = torch.empty((n, nd), dtype=torch.int32, device=dev)
    tau = torch.empty((n, nd), dtype=torch.float64, device=dev)
    st = torch.cuda.current_stream(dev)
    L.check(L.lib().bgwx_first_colliding_noalloc(
        C.c_void_p(b.data_ptr()), n, n, C.c_void_p(sel.data_ptr()), n, C.c_void_p(d.data_ptr()), nd,
        C.c_void_p(codes.data_ptr()), C.c_void_p(tau.data_ptr()), C.c_void_p(st.cuda_stream)))
    torch.cuda.synchronize()
    shape = (n, n_cos, n_phi)
    return codes.cpu().numpy().reshape(shape), tau.cpu().numpy().reshape(shape)


def spacelike(n, seed):
    rng = np.random.default_rng(seed)
    return np.column_stack([0.1 * rng.random(n), 2.0 + 3.0 * rng.random((n, 3))])


# Pairs whose interval is zero (exactly: the differences are powers of two) or negative do not collide:
# the reference skips every delay that is not positive.  Alone, beside one other bubble, and among many.
@pytest.mark.parametrize("n_cos,n_phi", [(5, 8), (2, 2), (33, 20)])
@pytest.mark.parametrize("pair", [
    [[0.0, 0.25, 0.0, 0.0], [0.5, 0.75, 0.0, 0.0]], [[0.25, 0.5, 0.5, 0.5], [0.25, 0.5, 0.5, 0.5]],
    [[0.0, 0.25, 0.0, 0.0], [0.6, 0.3, 0.05, 0.0]]], ids=["null", "same", "timelike"])
@pytest.mark.parametrize("others", [0, 1, 40])
@pytest.mark.parametrize("search", [by_handle, by_table])
def test_pairs_that_never_collide(gpu_available, n_cos, n_phi, pair, others, search):
    b = np.concatenate([np.array(pair), spacelike(others, 3)])
    codes, tau = search(b, n_cos, n_phi)
    rc, rt = O.first_colliding(b, NONE, n_cos, n_phi, with_delta_tab=True)
    assert np.array_equal(codes, rc)
    assert np.array_equal(tau, rt)
    assert np.all((codes >= 0) == (tau > 0.0))


# Colliders that nucleate just ahead of the wall, D / A = (|dx| - dt) / (|dx| + |dt|) from 1e-6 (where a
# collider is set aside) to 1e-3, all within a relative 1e-5 of one delay: the bound up to which a check can
# fail reaches past the candidate's own delay there.
@pytest.mark.parametrize("n_cos,n_phi", [(33, 40), (64, 65)])
@pytest.mark.parametrize("lo,hi", [(1.5e-6, 3e-6), (3e-6, 3e-5), (3e-5, 1e-3)])
@pytest.mark.parametrize("search", [by_handle, by_table])
def test_near_lightlike_colliders(gpu_available, n_cos, n_phi, lo, hi, search):
    rng = np.random.default_rng(12)
    n = 60
    u = rng.normal(size=(n, 3))
    u[30:] = u[:30] + 1e-4 * rng.normal(size=(30, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    d = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    r = 0.5 * (1.0 + 1e-5 * rng.uniform(-1.0, 1.0, n))
    b = np.concatenate([[[0.0, 0.0, 0.0, 0.0]], np.column_stack([r * (1.0 - 2.0 * d), r[:, None] * u])])
    codes, tau = search(b, n_cos, n_phi)
    rc, rt = O.first_colliding(b, NONE, n_cos, n_phi, with_delta_tab=True)
    assert np.array_equal(codes, rc)
    assert np.array_equal(tau, rt)
