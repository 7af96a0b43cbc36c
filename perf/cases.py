"""The work a user of the package has it do, as cases that can be timed and compared.

Every case goes through a public entry point: the tensor functions of
``openonda_b200.kernels``, the reference's own functions in
``openonda_b200.vpm.ParticlesPhysicsB200`` (numpy in, numpy out), the time step of
``ParticleSystem`` and the differentiable forms in ``openonda_b200.autodiff``.  Fields are the
seeded workloads of ``openonda_b200.configs`` at any particle count: the random cloud (cores
that differ) and rings on a torus lattice (one core for all).

* ``listed()``  -- the cases that stand for the range, each with the use it stands for;
* ``draw(rng)`` -- one more case of the same ranges;
* ``prepare(case, seed)`` / ``run(state)`` -- the inputs, and one pass;
* ``work(case)`` -- what a pass cannot do without: bytes in and out, and the flops of the pair
  terms with each unordered pair of a self sum evaluated once;
* ``exact(case, seed)`` -- the outputs of ``run`` in FP64 from plain torch.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from openonda_b200 import autodiff, configs, kernels
from openonda_b200.vpm import ParticlesPhysicsB200 as physics
from openonda_b200.vpm.vpmModule import ParticleSystem

F64 = torch.float64
EPS = 1e-8  # probe sums skip pairs with r^2 <= EPS, as the reference does
DT = 1e-3  # time step of the system and trajectory cases
STEPS = 2  # RK4 steps of the trajectory cases
MAX_PAIRS_EXACT = 2.0e10  # pairs that plain torch sums in seconds


def listed():
    return [
        # one velocity sum of a small system: launches and latency are all there is
        {"name": "velocity_fp64_1000", "kind": "velocity", "n": 1000, "precision": "fp64",
         "field": "cloud"},
        # a small simulation: the graph-replayed step of advance(), two velocity sums and the
        # stretching, core spreading (the default scheme)
        {"name": "system_cs_rk2_fp64_2000", "kind": "system", "n": 2000, "precision": "fp64",
         "field": "ring", "model": "DNS", "scheme": "CoreSpreading", "method": "RK2"},
        # the thick ring of the first workload: DNS with PSE, RK4, five pair sums a step
        {"name": "system_pse_rk4_fp64_8192", "kind": "system", "n": 8192, "precision": "fp64",
         "field": "ring", "model": "DNS", "scheme": "PSE", "method": "RK4"},
        # the reference's own calls on host arrays: velocity, stretching and PSE of one step
        {"name": "dropin_numpy_fp64_30011", "kind": "dropin", "n": 30011, "precision": "fp64",
         "field": "cloud"},
        # right-hand side of an ordinary FP64 simulation, cores that differ, an odd size
        {"name": "fused_fp64_100003", "kind": "fused", "n": 100003, "precision": "fp64",
         "field": "cloud"},
        # the large right-hand side: velocity and stretching of 2^20 particles in FP32c
        {"name": "fused_fp32c_1048576", "kind": "fused", "n": 1 << 20, "precision": "fp32c",
         "field": "cloud"},
        # the four sums of a dynamic-LES step, one core for all
        {"name": "les_fp32c_131072", "kind": "les", "n": 131072, "precision": "fp32c",
         "field": "ring"},
        # velocity on a sampling grid, FP64 (the default)
        {"name": "probe_velocity_fp64_100000x10007", "kind": "probe_velocity", "m": 100000,
         "n": 10007, "precision": "fp64", "field": "cloud"},
        # vorticity on a 64^3 grid for a picture, FP32c
        {"name": "probe_vorticity_fp32c_262144x32768", "kind": "probe_vorticity", "m": 262144,
         "n": 32768, "precision": "fp32c", "field": "ring"},
        # kinetic energy, enstrophy and helicity, as log_diagnostics evaluates them (FP64); a
        # plane ring has no helicity, so what its sum gives is rounding: the cloud has some
        {"name": "diagnostics_fp64_32768", "kind": "diagnostics", "n": 32768,
         "precision": "fp64", "field": "cloud"},
        # forward and backward of the right-hand side with PSE in FP32c
        {"name": "adjoint_pse_fp32c_32768", "kind": "adjoint", "n": 32768,
         "precision": "fp32c", "field": "ring", "pse": True},
        # a differentiated RK4 trajectory with the kinetic-energy loss, FP64 (the default)
        {"name": "trajectory_fp64_4096", "kind": "trajectory", "n": 4096, "precision": "fp64",
         "field": "ring"},
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["velocity", "pse", "fused", "les", "system", "dropin", "probe_velocity",
                       "probe_vorticity", "diagnostics", "adjoint", "trajectory"])
    precision = rng.choice(["fp64", "fp64", "fp32c"])
    case = {"kind": kind, "precision": precision, "field": rng.choice(["cloud", "ring"])}
    if kind in ("velocity", "pse", "fused"):
        case["n"] = _size(rng, 200, 300000)
    elif kind == "les":
        case["n"] = _size(rng, 500, 200000)
    elif kind == "system":
        case["n"] = _size(rng, 300, 20000)
        case["field"] = "ring"
        case["model"] = rng.choice(["DNS", "DNS", "pseudo2D", "LES"])
        case["scheme"] = rng.choice(["PSE", "CoreSpreading"])
        case["method"] = rng.choice(["Euler", "RK2", "RK4"])
    elif kind == "dropin":
        case["precision"] = "fp64"
        case["n"] = _size(rng, 300, 60000)
    elif kind in ("probe_velocity", "probe_vorticity"):
        case["m"] = _size(rng, 500, 300000)
        case["n"] = _size(rng, 300, 60000)
    elif kind == "diagnostics":
        case["precision"], case["field"] = "fp64", "cloud"
        case["n"] = _size(rng, 300, 100000)
    elif kind == "adjoint":
        case["n"] = _size(rng, 300, 60000)
        case["pse"] = rng.random() < 0.5
    else:
        case["n"] = _size(rng, 300, 16384)
        case["precision"] = "fp64"
    return case


# ---- inputs ------------------------------------------------------------------------------------
def _field(case, seed):
    """(positions, strengths, radii, viscosities) as float64 numpy arrays."""
    n = case["n"]
    if case["field"] == "cloud":
        f = configs.random_cloud(n, seed=seed)
    else:
        planes = max(16, int(round(math.sqrt(n))))
        make = configs.les_ring if case["kind"] == "les" else configs.perturbed_ring
        f = make(planes, -(-n // planes), seed=seed)
    return f.positions[:n], f.strengths[:n], f.radii[:n], f.viscosities[:n]


def _grid(m, seed):
    """m points of a regular grid over the box that holds the field, shifted by the seed."""
    k = max(2, int(math.ceil(m ** (1.0 / 3.0))))
    lo, hi = -1.5, 1.5
    shift = np.random.default_rng(seed).uniform(0.0, (hi - lo) / k, size=3)
    i = np.arange(m)
    cell = np.stack([i // (k * k), (i // k) % k, i % k], axis=1).astype(np.float64)
    return lo + shift + cell * ((hi - lo) / k)


def _cuda(arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def prepare(case, seed):
    kind = case["kind"]
    arrays = _field(case, seed)
    state = {"case": case, "uniform": case["field"] == "ring"}
    if kind == "dropin":
        state["host"] = arrays
        return state
    if kind == "system":
        x, a, s, nu = arrays
        # time step 1: the run's first backup, at step 0, is behind it
        ps = ParticleSystem(time_step_size=DT, time_integration_method=case["method"],
                            flow_model=case["model"], viscous_scheme=case["scheme"],
                            time_step=1, backup_frequency=10 ** 9,
                            precision=case["precision"])
        ps.add_particle_field(x, np.zeros_like(x), a, s, nu)
        state["system"] = ps
        return state
    state["x"], state["a"], state["s"], state["nu"] = _cuda(arrays)
    if kind in ("probe_velocity", "probe_vorticity"):
        state["t"] = _cuda([_grid(case["m"], seed)])[0]
    elif kind == "adjoint":
        rng = np.random.default_rng(seed + 1)
        state["gu"], state["gr"] = _cuda([rng.normal(size=(case["n"], 3)) for _ in range(2)])
        for key in ("x", "a", "s") + (("nu",) if case["pse"] else ()):
            state[key].requires_grad_()
    elif kind == "trajectory":
        for key in ("x", "a", "s"):
            state[key].requires_grad_()
    return state


# ---- one pass ----------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind, p, uc = case["kind"], case["precision"], state["uniform"]
    if kind == "dropin":
        x, a, s, nu = state["host"]
        return (physics.get_selfinduced_velocity(x, a, s), physics.get_strength_gradients(x, a, s),
                physics.get_strength_gradients_PSE(x, a, s, nu))
    if kind == "system":
        ps = state["system"]
        ps.advance(1)
        return ps.positions, ps.strengths, ps.radii
    x, a, s, nu = state["x"], state["a"], state["s"], state["nu"]
    if kind == "velocity":
        return kernels.selfinduced_velocity(x, a, s, precision=p, uniform_core=uc)
    if kind == "pse":
        return kernels.strength_gradients_pse(x, a, s, nu, precision=p, uniform_core=uc)
    if kind == "fused":
        return kernels.velocity_and_strength_gradients(x, a, s, precision=p, uniform_core=uc)
    if kind == "les":
        return kernels.les_step_sums(x, a, s, precision=p, uniform_core=uc)
    if kind == "probe_velocity":
        return kernels.induced_velocity_at(state["t"], x, a, s, precision=p)
    if kind == "probe_vorticity":
        return kernels.vorticity_field_at(state["t"], x, a, s, precision=p)
    if kind == "diagnostics":
        return (kernels.total_kinetic_energy(x, a, s, precision=p),
                kernels.total_enstrophy(x, a, s, precision=p),
                kernels.total_helicity(x, a, s, precision=p))
    if kind == "adjoint":
        inputs = (x, a, s, nu) if case["pse"] else (x, a, s)
        u, rate = autodiff.rhs(x, a, s, nu if case["pse"] else None, precision=p,
                               uniform_core=uc)
        grads = torch.autograd.grad((u, rate), inputs, (state["gu"], state["gr"]))
        return (u.detach(), rate.detach()) + grads
    xt, at = autodiff.trajectory(x, a, s, dt=DT, steps=STEPS, precision=p)
    loss = autodiff.kinetic_energy(xt, at, s, precision=p)
    return (loss.detach(), xt.detach(), at.detach()) + torch.autograd.grad(loss, (x, a, s))


# ---- what a pass cannot do without --------------------------------------------------------------
# flops of a pair term (FMA = 2, the reciprocal square root = 1): of an unordered pair for both
# particles in the self sums, of a target-source pair in the probe sums
PAIR_FLOPS = {"velocity": 49, "stretch": 67, "fused": 85, "pse": 36, "les": 115, "ke": 36,
              "ens": 22, "hel": 34, "vjp": 205, "vjp_pse": 240, "ke_grad": 74,
              "probe_velocity": 33, "probe_vorticity": 24}


def work(case):
    kind, n = case["kind"], case["n"]
    f = PAIR_FLOPS
    if kind in ("probe_velocity", "probe_vorticity"):
        return {"bytes": 56 * n + 48 * case["m"], "flops": f[kind] * case["m"] * n}
    pairs = n * (n - 1) / 2
    if kind == "dropin":
        return {"bytes": 64 * n + 72 * n, "flops": (f["velocity"] + f["stretch"] + f["pse"]) * pairs}
    if kind == "system":
        stages = {"Euler": 0, "RK2": 1, "RK4": 3}[case["method"]]
        first = {"DNS": "fused", "LES": "les", "pseudo2D": "velocity"}[case["model"]]
        flops = f[first] + stages * f["velocity"] + (f["pse"] if case["scheme"] == "PSE" else 0)
        return {"bytes": 2 * 152 * n, "flops": flops * pairs}
    if kind == "diagnostics":
        return {"bytes": 56 * n + 24, "flops": (f["ke"] + f["ens"] + f["hel"]) * pairs}
    if kind == "adjoint":
        pse = case["pse"]
        flops = f["fused"] + (f["pse"] + f["vjp_pse"] if pse else f["vjp"])
        return {"bytes": (64 + 48 + 48 + 64) * n, "flops": flops * pairs}
    if kind == "trajectory":
        # forward, the segment's recompute in the backward, and one VJP per evaluation
        evals = 4 * STEPS
        flops = evals * (2 * f["fused"] + f["vjp"]) + f["ke"] + f["ke_grad"]
        return {"bytes": (56 + 48 + 56) * n, "flops": flops * pairs}
    out = {"velocity": 24, "pse": 24, "fused": 48, "les": 72}[kind]
    return {"bytes": (64 if kind == "pse" else 56) * n + out * n, "flops": f[kind] * pairs}


# ---- the same in FP64 with plain torch -----------------------------------------------------------
def _rows(m, n):
    step = max(1, (1 << 24) // max(n, 1))
    return [(b, min(b + step, m)) for b in range(0, m, step)]


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _pair(x, a, s, b, e):
    """r (3 components), a_i, a_j, pair core^2, r^2 + core^2 of target rows [b, e)."""
    r = [x[b:e, k, None] - x[None, :, k] for k in range(3)]
    ai = [a[b:e, k, None] for k in range(3)]
    aj = [a[None, :, k] for k in range(3)]
    core = 0.5 * (s[b:e, None] + s[None, :])
    s2 = core * core
    return r, ai, aj, core, s2, _dot(r, r) + s2


def _block(x, a, s, nu, b, e, want):
    """The sums in `want` (velocity, stretch, pse, vorticity, enstrophy rows, ke rows)."""
    r, ai, aj, core, s2, q = _pair(x, a, s, b, e)
    c = 1.0 / (4.0 * math.pi)
    out = {}
    y = q.rsqrt()
    if "velocity" in want or "stretch" in want:
        g = (q + 1.5 * s2) * y ** 5
        w = _cross(r, aj)
        if "velocity" in want:
            out["velocity"] = torch.stack([-c * (g * w[k]).sum(1) for k in range(3)], 1)
        if "stretch" in want:
            h = 3.0 * (q + 2.5 * s2) * y ** 7 * _dot(ai, w)
            ax = _cross(ai, aj)
            out["stretch"] = torch.stack([c * (g * ax[k] + h * r[k]).sum(1) for k in range(3)], 1)
    if "pse" in want:
        k7 = core ** 7 * y ** 9
        out["pse"] = torch.stack([105.0 * c * nu[b:e] * (k7 * (aj[k] - ai[k])).sum(1)
                                  for k in range(3)], 1)
    if "vorticity" in want:
        out["vorticity"] = _probe_block(x[b:e], x, a, s, "probe_vorticity")
    if "enstrophy" in want:
        k3 = (q + 2.2 * s2) * y ** 3
        out["enstrophy"] = (k3 * _dot(ai, aj)).sum()
    if "ke" in want:
        y3 = y ** 3
        k = _dot(ai, aj) * (y + s2 * y3) + y3 * _dot(r, ai) * _dot(r, aj)
        i = torch.arange(b, e, device=x.device)
        k = k.index_put((i - b, i), torch.zeros((), dtype=F64, device=x.device))
        out["ke"] = k.sum()
    return out


def _probe_block(t, x, a, s, kind):
    r = [t[:, k, None] - x[None, :, k] for k in range(3)]
    aj = [a[None, :, k] for k in range(3)]
    r2 = _dot(r, r)
    s2 = (s * s)[None, :]
    y = (r2 + s2).rsqrt()
    c = 1.0 / (4.0 * math.pi)
    if kind == "probe_velocity":
        w, k = _cross(r, aj), -c * (r2 + 2.5 * s2) * y ** 5
    else:
        w, k = aj, 7.5 * c * s2 * s2 * y ** 7
    k = torch.where(r2 > EPS, k, torch.zeros_like(k))
    return torch.stack([(k * w[d]).sum(1) for d in range(3)], 1)


def _sums(x, a, s, nu, want):
    got = {}
    for b, e in _rows(x.shape[0], x.shape[0]):
        for k, v in _block(x, a, s, nu, b, e, want).items():
            got.setdefault(k, []).append(v)
    return {k: torch.cat(v) if v[0].dim() else sum(v) for k, v in got.items()}


def _system_step(case, x, a, s, nu):
    """One step of ParticleSystem from time step 1 (BDF2 with a zero history)."""
    stretch = case["model"] == "DNS"
    now = _sums(x, a, s, nu, {"velocity", "stretch"} if stretch else {"velocity"})
    last = torch.zeros_like(a)
    for rate in ("stretch", "pse"):
        if rate == "pse" and case["scheme"] == "PSE":
            now["pse"] = _sums(x, a, s, nu, {"pse"})["pse"]
        if rate in now:
            a = (4.0 * a - last) / 3.0 + (2.0 / 3.0) * DT * now[rate]
            last = a
    if case["scheme"] == "CoreSpreading":
        s = torch.sqrt(s * s + 5.34 * nu * DT)
    k1 = now["velocity"]

    def velocity(at):
        return _sums(at, a, s, nu, {"velocity"})["velocity"]

    if case["method"] == "Euler":
        return x + DT * k1, a, s
    k2 = velocity(x + 0.5 * DT * k1)
    if case["method"] == "RK2":
        return x + DT * k2, a, s
    k3 = velocity(x + 0.5 * DT * k2)
    k4 = velocity(x + DT * k3)
    return x + DT / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4), a, s


def _trajectory(x, a, s):
    def rhs(x_, a_):
        def block(xb, ab, sb, b, e):
            got = _block(xb, ab, sb, None, b, e, {"velocity", "stretch"})
            return got["velocity"], got["stretch"]

        parts = [torch.utils.checkpoint.checkpoint(block, x_, a_, s, b, e, use_reentrant=False)
                 for b, e in _rows(x_.shape[0], x_.shape[0])]
        return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])

    for _ in range(STEPS):
        k1, l1 = rhs(x, a)
        k2, l2 = rhs(x + DT / 2 * k1, a + DT / 2 * l1)
        k3, l3 = rhs(x + DT / 2 * k2, a + DT / 2 * l2)
        k4, l4 = rhs(x + DT * k3, a + DT * l3)
        x = x + DT / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        a = a + DT / 6 * (l1 + 2 * l2 + 2 * l3 + l4)
    return x, a


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    pairs = float(case.get("m", n)) * n
    heavy = {"adjoint": 8.0, "trajectory": 40.0, "les": 2.0, "diagnostics": 1.5}.get(kind, 1.0)
    if pairs * heavy > MAX_PAIRS_EXACT or case.get("model") == "LES":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, a, s, nu = [torch.from_numpy(np.array(v, dtype=np.float64)).to(dev)
                   for v in _field(case, seed)]
    if kind == "dropin":
        got = _sums(x, a, s, nu, {"velocity", "stretch", "pse"})
        return tuple(got[k].cpu().numpy() for k in ("velocity", "stretch", "pse"))
    if kind == "system":
        return _system_step(case, x, a, s, nu)
    if kind in ("velocity", "pse"):
        return _sums(x, a, s, nu, {kind})[kind]
    if kind == "fused":
        got = _sums(x, a, s, nu, {"velocity", "stretch"})
        return got["velocity"], got["stretch"]
    four_pi = 4.0 * math.pi
    if kind == "les":
        got = _sums(x, a, s, nu, {"velocity", "stretch", "vorticity", "enstrophy"})
        return (got["velocity"], got["stretch"], got["vorticity"],
                got["enstrophy"] / (2.0 * four_pi) / four_pi)
    if kind in ("probe_velocity", "probe_vorticity"):
        t = torch.from_numpy(_grid(case["m"], seed)).to(dev)
        return torch.cat([_probe_block(t[b:e], x, a, s, kind) for b, e in _rows(case["m"], n)])
    if kind == "diagnostics":
        got = _sums(x, a, s, nu, {"velocity", "enstrophy", "ke"})
        return (got["ke"] / (4.0 * four_pi), got["enstrophy"] / (2.0 * four_pi) / four_pi,
                (a * got["velocity"]).sum() / four_pi)
    if kind == "adjoint":
        rng = np.random.default_rng(seed + 1)
        gu, gr = [torch.from_numpy(rng.normal(size=(n, 3))).to(dev) for _ in range(2)]
        leaves = [v.requires_grad_() for v in ((x, a, s, nu) if case["pse"] else (x, a, s))]
        u, rate, grads = [], [], [torch.zeros_like(v) for v in leaves]
        step = max(1, (1 << 22) // n)
        for b in range(0, n, step):
            e = min(b + step, n)
            got = _block(x, a, s, nu, b, e,
                         {"velocity", "stretch", "pse"} if case["pse"] else {"velocity", "stretch"})
            r = got["stretch"] + got["pse"] if case["pse"] else got["stretch"]
            for k, v in enumerate(torch.autograd.grad((got["velocity"], r), leaves,
                                                      (gu[b:e], gr[b:e]))):
                grads[k] += v
            u.append(got["velocity"].detach())
            rate.append(r.detach())
        return (torch.cat(u), torch.cat(rate)) + tuple(grads)
    leaves = [v.requires_grad_() for v in (x, a, s)]
    xt, at = _trajectory(*leaves)
    loss = sum(torch.utils.checkpoint.checkpoint(
        lambda xb, ab, sb, b, e: _block(xb, ab, sb, None, b, e, {"ke"})["ke"],
        xt, at, s, b, e, use_reentrant=False) for b, e in _rows(n, n)) / (4.0 * four_pi)
    return (loss.detach(), xt.detach(), at.detach()) + torch.autograd.grad(loss, leaves)
