"""Measured cases of the bulk-flow framework: calls of its public entry points at the sizes users run.

Every case is one call (for the fit, one forward and backward) on a bubble configuration drawn from the
seed: exponential nucleation in a periodic unit box, or a handful of uniform bubbles without images, as in
the benchmark configurations of gw_fopt_b200/workloads.py.  ``exact`` evaluates the same quantities with
plain torch in 64 bits from the definition: brute-force first colliders, the scaling function of every
patch at every time step, one complex phase per (bubble, row, step, frequency).
"""
import math

import numpy as np
import torch

from gw_fopt_b200 import many_bubbles as mb
from gw_fopt_b200 import workloads
from gw_fopt_b200.autograd import BulkFlowSpectrum, log_power_residual
from gw_fopt_b200.ensemble import BulkFlowEnsemble

T_END = 1.5  # final time, in units of the box side

_BASE = {"what": "spectrum", "n": 5, "periodic": True, "n_cos": 32, "n_phi": 32, "n_t": 128, "n_w": 32, "w_max": 1000.0,
         "n_khat": 0, "kernel": "fp64_direct", "sets": 1, "terms": 1, "damping": 0.0, "cutoff": False}


def _case(**kw):
    c = dict(_BASE)
    c.update(kw)
    return c


def listed():
    return [
        # One spectrum of a handful of bubbles with the default kernel: the first call of a new user and the
        # size of the reference's own criterion benchmark (5 bubbles, 50 x 100 patches, 800 steps, 120 w).
        _case(name="single_5b", n=5, periodic=False, n_cos=50, n_phi=100, n_t=800, n_w=120, w_max=100.0),
        # Benchmark configuration 1: a direction scan of 8 bubbles, default kernel; latency and launches count.
        _case(name="khat_scan_8b", n=8, n_khat=16),
        # A production run with the default kernel: three scaling powers at once and the time cutoff.
        _case(name="default_64b", n=64, n_cos=64, n_phi=64, n_t=256, n_w=64, n_khat=4, sets=3, cutoff=True),
        # Benchmark configuration 2 with the factored FP64 kernel, four of its directions per call.
        _case(name="factored_512b", n=512, n_cos=128, n_phi=128, n_t=512, n_w=128, w_max=3000.0, n_khat=4,
              kernel="fp64_factored"),
        # Benchmark configuration 3 (mixed kernel, the headline workload), eight of its directions: the largest.
        _case(name="mixed_4096b", n=4096, n_cos=192, n_phi=192, n_t=1024, n_w=256, w_max=1e4, n_khat=8,
              kernel="mixed"),
        # Ragged sizes and every scaling option on the mixed kernel: two sets of two terms, damped.
        _case(name="mixed_ragged_101b", n=101, n_cos=65, n_phi=75, n_t=301, n_w=45, n_khat=6, sets=2, terms=2,
              damping=0.5, kernel="mixed"),
        # Benchmark configuration 4 (Monte Carlo ensemble, mixed kernel): 16 realizations of 50 to 800 bubbles.
        _case(name="ensemble_16r", what="ensemble", n=16, n_cos=96, n_phi=96, n_t=384, n_w=128, w_max=3000.0,
              n_khat=8, kernel="mixed"),
        # Benchmark configuration 5: one step of the scaling fit, forward and backward, mixed kernel.
        _case(name="fit_mixed_256b", what="fit", n=256, n_cos=64, n_phi=64, n_t=256, n_w=64, n_khat=32, terms=2,
              kernel="mixed"),
        # The same fit step on a smaller, odd-sized problem with the autograd function's default FP64 kernel.
        _case(name="fit_fp64_48b", what="fit", n=48, n_cos=47, n_phi=50, n_t=200, n_w=40, n_khat=8, terms=2,
              kernel="fp64_factored"),
        # The tensor form C_ij (TT projection downstream), a few directions.
        _case(name="tensor_16b", what="tensor", n=16, n_cos=33, n_phi=64, n_t=200, n_w=50, n_khat=4),
        # The time-resolved integrand of a handful of bubbles (inspection plots).
        _case(name="integrand_5b", what="integrand", n=5, periodic=False, n_cos=50, n_phi=100, n_t=400, n_w=60,
              w_max=100.0),
        # The first colliding bubble of every wall patch of one bubble: the smallest call.
        _case(name="collider_512b", what="collider", n=512, n_cos=128, n_phi=128, n_t=2, n_w=1),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what, kernel = rng.choice([("spectrum", "fp64_direct"), ("spectrum", "fp64_direct"), ("spectrum", "fp64_factored"),
                               ("spectrum", "mixed"), ("spectrum", "mixed"), ("ensemble", "mixed"), ("fit", "mixed"),
                               ("fit", "fp64_factored"), ("tensor", "fp64_direct"), ("integrand", "fp64_direct"),
                               ("collider", "fp64_direct")])
    c = _case(what=what, kernel=kernel, w_max=float(10 ** rng.uniform(2.0, 4.0)))
    fast = kernel != "fp64_direct"
    c["n"] = _log_int(rng, 4, 24) if what == "ensemble" else _log_int(rng, 5, 24) if what in ("tensor", "integrand") \
        else _log_int(rng, 16, 256) if what == "fit" else _log_int(rng, 32, 4096) if fast or what == "collider" \
        else _log_int(rng, 5, 64)
    c["periodic"] = c["n"] > 8 or what == "ensemble" or rng.random() < 0.5
    top = 192 if fast and what == "spectrum" else 96
    c["n_cos"] = rng.randint(24, top if what != "fit" else 64)
    c["n_phi"] = rng.randint(24, top if what != "fit" else 64)
    c["n_t"] = _log_int(rng, 64, 1024 if fast and what == "spectrum" else 400)
    c["n_w"] = _log_int(rng, 8, 256 if fast and what == "spectrum" else 64)
    c["n_khat"] = _log_int(rng, 4, 32) if what == "fit" else _log_int(rng, 1, 8) if what in ("ensemble", "tensor") \
        else rng.choice([0, _log_int(rng, 1, 16)]) if what == "spectrum" else 0
    if what in ("spectrum", "tensor") and c["n"] <= 512:
        c["sets"], c["terms"] = rng.choice([(1, 1), (1, 1), (3, 1), (2, 2), (1, 2)])
        c["damping"] = rng.choice([0.0, 0.0, round(rng.uniform(0.3, 2.0), 3)])
        c["cutoff"] = what == "spectrum" and rng.random() < 0.3
    if what == "fit":
        c["terms"] = 2
    if what == "collider":
        c["n_t"], c["n_w"] = 2, 1
    # no drawn case costs more than the largest listed one of its kernel
    most = {"fp64_direct": 3e8, "fp64_factored": 1.7e10, "mixed": 1.2e12}[kernel] if what in ("spectrum", "tensor") \
        else {"ensemble": 1.9e11, "fit": 8.6e9, "integrand": 1e8, "collider": 1e12}[what]
    while _patch_steps(c) * c["sets"] * c["terms"] > most:
        big = max(("n_khat", "n_t", "n"), key=lambda k: c[k] / {"n_khat": 1, "n_t": 64, "n": 8}[k])
        c[big] = max(1, int(c[big] * 0.7))
    return c


def _bubbles_of(case):
    return 425 * case["n"] if case["what"] == "ensemble" else case["n"]


def _patch_steps(case):
    return max(1, case["n_khat"]) * _bubbles_of(case) * case["n_cos"] * case["n_phi"] * case["n_t"]


def _bubbles(case, seed):
    """(interior, exterior) of the case's configuration."""
    n = case["n"]
    if n <= 8:
        interior, exterior = workloads.uniform_config(n, 1.0, 0.2, seed=seed)
    else:
        beta = max(5.0, 20.0 * (n / 4096.0) ** 0.45)
        interior, exterior = workloads.exponential_nucleation(n, beta, seed=seed, max_rejections=20000)
    return interior, exterior if case["periodic"] else np.zeros((0, 4))


def _scaling(case):
    """(coefficients, powers), each (sets, terms); every set's coefficients add up to 1."""
    s, m = case["sets"], case["terms"]
    powers = np.array([[5.0 - 0.5 * q - 1.0 * t for t in range(m)] for q in range(s)])
    share = np.array([0.75, 0.25])[:m] if m > 1 else np.ones(1)
    return np.tile(share, (s, 1)), powers


def _grids(case):
    w = np.geomspace(1.0, case["w_max"], case["n_w"])
    return w, workloads.fibonacci_khat(case["n_khat"]) if case["n_khat"] else None


def _fit_inputs(case, seed):
    rng = np.random.default_rng(seed)
    w, khat = _grids(case)
    target = 10.0 ** rng.uniform(-6.0, -4.0, (khat.shape[0], 1, w.size)) / (1.0 + w ** 2)
    alpha, delta = 0.8 + 0.1 * rng.random(), 0.2 + 0.1 * rng.random()
    return np.array([[alpha, delta]]), np.array([[4.6, 4.5]]) + 0.2 * rng.random((1, 2)), target


def prepare(case, seed):
    dev = torch.device("cuda")
    w, khat = _grids(case)
    state = {"case": case, "w": w, "khat": khat}
    if case["what"] == "ensemble":
        rng = np.random.default_rng(seed)
        state["flow"] = BulkFlowEnsemble(
            [workloads.exponential_nucleation(int(rng.integers(50, 801)), float(rng.uniform(5.0, 15.0)),
                                              seed=int(rng.integers(0, 2 ** 31 - 1)), max_rejections=20000)
             for _ in range(case["n"])], validate=False)
    elif case["what"] == "fit":
        interior, _ = _bubbles(case, seed)
        state["flow"] = BulkFlowSpectrum(n_cos=case["n_cos"], n_phi=case["n_phi"], w=w, khat=khat, t_end=T_END,
                                         n_t=case["n_t"], box=1.0, kernel=case["kernel"])
        co, po, target = _fit_inputs(case, seed)
        state["leaves"] = [torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)
                           for v in (co, po, interior)]
        state["target"] = torch.tensor(target, dtype=torch.float64, device=dev)
        return state
    else:
        interior, exterior = _bubbles(case, seed)
        lattice = mb.CartesianLattice.with_origin_and_sizes([0.0, 0.0, 0.0], [1.0, 1.0, 1.0]) if case["periodic"] \
            else mb.EmptyLattice()
        bubbles = mb.LatticeBubbles(lattice, interior)
        if case["periodic"]:
            bubbles.with_boundary_condition("periodic")
        state["flow"] = (mb.NewGeneralizedBulkFlow if case["what"] == "tensor" else mb.GeneralizedBulkFlow)(bubbles)
    flow = state["flow"]
    flow.set_resolution(case["n_cos"], case["n_phi"])
    flow.set_gradient_scaling_params(*[v.tolist() for v in _scaling(case)], case["damping"] or None)
    if case["kernel"] != "fp64_direct":
        flow.set_kernel(case["kernel"])
    state["cutoff"] = mb.ExponentialTimeCutoff(T_END, 0.8, 0.25) if case["cutoff"] else None
    return state


def run(state):
    case, flow, w, khat, n_t = state["case"], state["flow"], state["w"], state["khat"], state["case"]["n_t"]
    if case["what"] == "collider":
        return flow.compute_first_colliding_bubble(case["n"] // 2)
    if case["what"] == "integrand":
        return flow.compute_c_integrand(w, t_end=T_END, n_t=n_t)
    if case["what"] == "tensor":
        return flow.compute_c_tensor_khat(w, khat, t_end=T_END, n_t=n_t)
    if case["what"] == "fit":
        c = flow(*state["leaves"])
        loss = log_power_residual(c, state["target"])
        grads = torch.autograd.grad(loss, state["leaves"])
        return {"spectrum": c.detach(), "loss": loss.detach(), "coefficients": grads[0], "powers": grads[1],
                "bubbles": grads[2]}
    if khat is None:
        return flow.compute_c_integral(w, t_end=T_END, n_t=n_t, time_cutoff=state["cutoff"])
    return flow.compute_c_integral_khat(w, khat, t_end=T_END, n_t=n_t, time_cutoff=state["cutoff"])


def work(case):
    """Per (direction, bubble, row): the patches' delays and scaling weights once each, then one real product of
    (cos, sin) x columns per (step, frequency).  Bytes: the bubbles in, the result out."""
    rows = max(1, case["n_khat"]) * _bubbles_of(case) * case["n_cos"]
    columns = (6 if case["what"] == "tensor" else 2) * case["sets"]
    n_in = 32.0 * 7 * _bubbles_of(case)
    if case["what"] == "collider":
        patches = case["n_cos"] * case["n_phi"]
        return {"bytes": n_in + 4.0 * patches, "flops": 30.0 * patches}
    flops = rows * (case["n_phi"] * (30.0 + 4.0 * columns * case["terms"]) +
                    case["n_t"] * columns * (4.0 * case["n_w"] + 4.0 * case["terms"]))
    out = 16.0 * max(1, case["n_khat"]) * columns * case["n_w"] * (case["n"] if case["what"] == "ensemble" else 1)
    if case["what"] == "integrand":
        out *= case["n_t"]
    return {"bytes": n_in + out, "flops": flops * (3.0 if case["what"] == "fit" else 1.0)}


# --------------------------------------------------------------------------------------------------------------
def _rotation(k):
    """Rodrigues rotation taking the unit vector k to z about k x z."""
    ax, ay = k[1], -k[0]
    s2 = ax * ax + ay * ay
    if s2 < 1e-30:
        return np.diag([1.0, 1.0, 1.0] if k[2] >= 0.0 else [1.0, -1.0, -1.0])
    s = math.sqrt(s2)
    ux, uy, c = ax / s, ay / s, k[2]
    v = 1.0 - c
    return np.array([[c + v * (ux * ux), v * (ux * uy), s * uy], [v * (uy * ux), c + v * (uy * uy), -(s * ux)],
                     [-(s * uy), s * ux, c]])


def _linspace(a, b, n):
    step = (b - a) / (n - 1)
    return np.array([a + step * i for i in range(n)])


def _mdot(a, b):
    return ((-a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]) + a[3] * b[3]


class _Exact:
    """The definition, in 64 bits, for one configuration and any number of directions."""

    def __init__(self, case, dev):
        self.case, self.dev = case, dev
        tensor = case["what"] == "tensor"
        cos_t = _linspace(-1.0, 1.0, case["n_cos"])
        phi = _linspace(0.0, 2.0 * math.pi, case["n_phi"])
        sin_t = np.sqrt(np.maximum(1.0 - cos_t * cos_t, 0.0))
        cp, sp = (np.array([f(p) for p in phi]) for f in (math.cos, math.sin))
        self.dirs = [self._t(v) for v in (np.ones((cos_t.size, phi.size)), sin_t[:, None] * cp, sin_t[:, None] * sp,
                                          np.broadcast_to(cos_t[:, None], (cos_t.size, phi.size)).copy())]
        ends = np.ones(phi.size)
        ends[[0, -1]] = 0.5
        if tensor:  # xx, xy, xz, yy, yz, zz
            g = [(cp * cp, sin_t ** 2), (cp * sp, sin_t ** 2), (cp, sin_t * cos_t), (sp * sp, sin_t ** 2),
                 (sp, sin_t * cos_t), (np.ones_like(cp), cos_t ** 2)]
        else:  # +, x
            g = [(np.array([f(2.0 * p) for p in phi]), 0.5 * (1.0 - cos_t * cos_t)) for f in (math.cos, math.sin)]
        row_ends = np.ones(cos_t.size)
        row_ends[[0, -1]] = 0.5
        self.phi_w = self._t(np.stack([a * ends for a, _ in g], 1) * (2.0 * math.pi / phi.size))  # (n_phi, G)
        self.row_w = self._t(np.stack([b * row_ends for _, b in g], 1) * (2.0 / (cos_t.size - 1)))  # (n_cos, G)
        self.cos_t = self._t(cos_t)
        self.t = self._t(_linspace(0.0, T_END, case["n_t"]))
        u = np.ones(case["n_t"])
        u[[0, -1]] = 0.5
        if case["cutoff"]:
            t_cut = 0.8 * T_END
            t_0 = 0.25 * (T_END - t_cut)
            t = _linspace(0.0, T_END, case["n_t"])
            u = u * np.where(t < t_cut, 1.0, np.exp(-((t - t_cut) ** 2) / t_0 ** 2))
        self.t_w = self._t(u) * (self.t[1] - self.t[0]) / (6.0 * math.pi)
        self.w = self._t(_grids(case)[0])

    def _t(self, v):
        return torch.as_tensor(np.array(v, dtype=np.float64), device=self.dev)

    def colliders(self, bub, a):
        """Index of the first collider of every patch of bubbles `a`, -1 where there is none: the least delay."""
        n_tot, patches = bub.shape[0], self.case["n_cos"] * self.case["n_phi"]
        d = torch.stack([v.reshape(-1) for v in self.dirs], 1) * torch.tensor([-1.0, 1.0, 1.0, 1.0], device=self.dev,
                                                                              dtype=torch.float64)
        out = torch.empty((len(a), patches), dtype=torch.int64, device=self.dev)
        for q, b in enumerate(a):
            delta = bub - bub[b]
            s = _mdot(delta.T, delta.T)
            least = torch.full((patches,), math.inf, dtype=torch.float64, device=self.dev)
            who = torch.full((patches,), -1, dtype=torch.int64, device=self.dev)
            for c0 in range(0, n_tot, 4096):
                dot = d @ delta[c0:c0 + 4096].T
                tau = torch.where(dot > 1e-10, s[c0:c0 + 4096] / (2.0 * dot), math.inf)
                tau = torch.where(tau > 0.0, tau, math.inf)
                if c0 <= b < c0 + 4096:
                    tau[:, b - c0] = math.inf
                m, i = tau.min(1)
                who = torch.where(m < least, i + c0, who)
                least = torch.minimum(m, least)
            out[q] = who
        return out.reshape(len(a), self.case["n_cos"], self.case["n_phi"])

    def delays(self, bub, a, who):
        """The collision delay of every patch (0: none), with the derivative with respect to the bubbles."""
        xa, xb = bub[a], bub[who.clamp(min=0)]
        delta = [xb[..., q] - xa[:, None, None, q] for q in range(4)]
        dot = _mdot(delta, self.dirs)
        return torch.where(who >= 0, _mdot(delta, delta) / (2.0 * torch.where(who >= 0, dot, 1.0)), 0.0)

    def sum_over(self, bub, a, tau, co, po, per_step=False):
        """(G, S, W) of bubbles `a` ((G, S, W, T) with per_step), in chunks of steps."""
        case, n_a = self.case, len(a)
        ta, za = bub[a][:, 0], bub[a][:, 3]
        S, M = co.shape
        G = self.phi_w.shape[1]
        total = 0.0
        steps = max(1, int(1.5e7 / (n_a * case["n_cos"] * max(case["n_phi"], case["n_w"]))))
        parts = []
        for k0 in range(0, case["n_t"], steps):
            t = self.t[k0:k0 + steps]
            dt = t[None, :] - ta[:, None]                                          # (A, T)
            on = dt > 0.0
            safe = torch.where(on, dt, 1.0)[:, :, None, None]
            hit = (tau[:, None] > 0.0) & (dt[:, :, None, None] >= tau[:, None]) & on[:, :, None, None]
            ratio = torch.where(hit, tau[:, None] / safe, 1.0)                     # (A, T, n_cos, n_phi)
            damp = torch.exp(-safe * (1.0 - ratio) / case["damping"]) if case["damping"] else 1.0
            cube = torch.where(on, dt ** 3, 0.0)[:, :, None, None]
            ph = -self.w * dt[:, :, None, None] * self.cos_t[:, None]              # (A, T, n_cos, W)
            e_re, e_im = torch.cos(ph), torch.sin(ph)
            zp = self.w * (t[None, :, None] - za[:, None, None])                   # (A, T, W)
            turn = torch.complex(torch.cos(zp), torch.sin(zp)) * self.t_w[None, k0:k0 + steps, None]
            rows = []
            for s in range(S):
                f = sum(co[s, m] * ratio ** po[s, m] for m in range(M)) * damp
                f = torch.where(hit, f, 1.0)
                B = (f.reshape(-1, case["n_phi"]) @ self.phi_w).reshape(n_a, -1, case["n_cos"], G) * self.row_w * cube
                Bt = B.transpose(2, 3)                                             # (A, T, G, n_cos)
                A = torch.complex(Bt @ e_re, Bt @ e_im) * turn[:, :, None]         # (A, T, G, W)
                rows.append(A.sum(0).permute(1, 2, 0) if per_step else A.sum((0, 1)))
            got = torch.stack(rows, 1)                                             # (G, S, W[, T])
            if per_step:
                parts.append(got)
            else:
                total = total + got
        return torch.cat(parts, -1) if per_step else total


def _groups(case, n):
    """Bubbles evaluated at once (few for the fit, whose derivative keeps every intermediate)."""
    most = 1e5 if case["what"] == "fit" else 4e6
    size = max(1, min(n, int(most / (case["n_cos"] * max(case["n_phi"], case["n_w"])))))
    return [list(range(q, min(n, q + size))) for q in range(0, n, size)]


def exact(case, seed):
    if case["what"] in ("collider", "ensemble"):
        return None
    n_tot = case["n"] * (7 if case["periodic"] or case["what"] == "fit" else 1)
    frames = max(1, case["n_khat"])
    cost = _patch_steps(case) * (case["sets"] * case["terms"] + 2.0) * (4.0 if case["what"] == "fit" else 1.0) + \
        2.0 * frames * case["n"] * case["n_cos"] * case["n_t"] * case["n_w"] * (4.0 if case["what"] == "fit" else 1.0) + \
        3.0 * frames * case["n"] * case["n_cos"] * case["n_phi"] * n_tot
    if cost > 6e11:
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    ex = _Exact(case, dev)
    interior, exterior = _bubbles(case, seed)
    w, khat = _grids(case)
    rots = [None] if khat is None else [ex._t(_rotation(k)) for k in khat]
    fit = case["what"] == "fit"
    co, po = _fit_inputs(case, seed)[:2] if fit else _scaling(case)
    leaves = [ex._t(v) for v in (co, po, interior)]
    images = ex._t(workloads.periodic_images(interior) - np.repeat(interior, 6, axis=0)) if fit else None

    def frame(inner, rot):
        rows = torch.cat([inner, inner.repeat_interleave(6, 0) + images if fit else ex._t(exterior)])
        if rot is None:
            return rows
        x = rows[:, 1:4]
        turned = [(rot[i, 0] * x[:, 0] + rot[i, 1] * x[:, 1]) + rot[i, 2] * x[:, 2] for i in range(3)]
        return torch.stack([rows[:, 0]] + turned, 1)

    found, out = [], []
    with torch.no_grad():
        for rot in rots:
            bub, acc, masks = frame(leaves[2], rot), 0.0, []
            for a in _groups(case, case["n"]):
                who = ex.colliders(bub, a)
                masks.append(who)
                acc = acc + ex.sum_over(bub, a, ex.delays(bub, a, who), leaves[0], leaves[1],
                                        case["what"] == "integrand")
            found.append(masks if fit else None)
            out.append(acc)
    spectrum = torch.stack(out) if khat is not None else out[0]
    if not fit:
        return spectrum.cpu().numpy()
    c = torch.view_as_real(spectrum).clone().requires_grad_(True)
    power = (c ** 2).sum(-1).sum(1)
    loss = ((torch.log(power) - torch.log(ex._t(_fit_inputs(case, seed)[2]))) ** 2).mean()
    (g,) = torch.autograd.grad(loss, c)
    grads = [torch.zeros_like(v) for v in leaves]
    for k, rot in enumerate(rots):
        for q, a in enumerate(_groups(case, case["n"])):
            live = [v.clone().requires_grad_(True) for v in leaves]
            bub = frame(live[2], rot)
            got = torch.view_as_real(ex.sum_over(bub, a, ex.delays(bub, a, found[k][q]), live[0], live[1]))
            for v, d in zip(grads, torch.autograd.grad((got * g[k]).sum(), live)):
                v += d
    return {"spectrum": c.detach().cpu(), "loss": loss.detach().cpu(), "coefficients": grads[0].cpu(),
            "powers": grads[1].cpu(), "bubbles": grads[2].cpu()}
