"""The work that a program has this framework do, as cases that can be timed and checked.

Each case is one call (or one short run) through the public entry points: right-hand sides in both
precisions, adaptive integrations of one system and of a batch, leapfrog, the energy diagnostics,
the element-wise Runge-Kutta kernels and the training of the step-size proposer.  Initial states are
Plummer spheres, cold uniform spheres and uniform balls in units of G = M = 1, as in the benchmark.
"""
import math
import os

import numpy as np
import torch

import ode_prototyping_gb300 as gb
from ode_prototyping_gb300 import learned

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(gb.__file__)), "weights")
FLOPS = 20  # per ordered pair, the usual count for softened gravity


def listed():
    return [
        # a small cluster's right-hand side, called once per stage by a program with its own loop: latency
        {"name": "rhs_f64_257", "kind": "rhs", "precision": "f64", "ic": "plummer", "n": 257, "eps": 0.02},
        # the FP64 right-hand side at the benchmark's headline size: the accuracy reference of every run
        {"name": "rhs_f64_16384", "kind": "rhs", "precision": "f64", "ic": "plummer", "n": 16384, "eps": 0.005},
        # the mixed-precision right-hand side at an ordinary size ...
        {"name": "rhs_mixed_4096", "kind": "rhs", "precision": "mixed", "ic": "plummer", "n": 4096, "eps": 0.005},
        # ... and on a large, ragged cold collapse
        {"name": "rhs_mixed_100003", "kind": "rhs", "precision": "mixed", "ic": "cold", "n": 100003, "eps": 0.002},
        # the plain FP64 method on a uniform ball of 1024 bodies (DOPRI5, tol 1e-10), with samples at output times
        {"name": "integrate_f64_1024", "kind": "integrate", "precision": "f64", "ic": "ball", "n": 1024, "eps": 0.01,
         "tableau": "DOPRI5", "tol": 1e-10, "tf": 0.05, "controller": "reference", "outputs": 8},
        # the headline integration: Plummer 16384, RKF78, mixed precision, tol 1e-11, learned proposer, a short span
        {"name": "integrate_mixed_16384", "kind": "integrate", "precision": "mixed", "ic": "plummer", "n": 16384,
         "eps": 0.005, "tableau": "RKF78", "tol": 1e-11, "tf": 0.03, "controller": "learned", "outputs": 0},
        # an ensemble of Plummer spheres of 64 to 4096 bodies advanced together, mixed precision
        {"name": "batch_mixed_128", "kind": "batch", "precision": "mixed", "systems": 128, "n_min": 64, "n_max": 4096,
         "tol": 1e-9, "tf": 0.05},
        # a smaller ensemble in FP64
        {"name": "batch_f64_24", "kind": "batch", "precision": "f64", "systems": 24, "n_min": 64, "n_max": 1024,
         "tol": 1e-9, "tf": 0.02},
        # fixed-step leapfrog in FP64 with a mass for each body, odd size
        {"name": "leapfrog_f64_3001", "kind": "leapfrog", "precision": "f64", "ic": "plummer", "n": 3001, "eps": 0.01,
         "masses": True, "steps": 16},
        # energy and momenta of the headline system, taken before and after every run
        {"name": "energy_16384", "kind": "energy", "ic": "plummer", "n": 16384, "eps": 0.005},
        # the element-wise kernels of one RKF78 attempt for a program that brings its own right-hand side
        {"name": "rk_rkf78_600018", "kind": "rk", "tableau": "RKF78", "n_var": 600018},
        # training the step-size proposer on one system's controller logs
        {"name": "train_2000", "kind": "train", "samples": 2000, "epochs": 100},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs_f64", "rhs_f64", "rhs_mixed", "rhs_mixed", "integrate_f64", "integrate_mixed",
                       "batch_mixed", "batch_f64", "leapfrog", "energy", "rk", "train"])
    ic = rng.choice(["plummer", "cold", "ball"])
    eps = round(0.002 * 10.0 ** rng.uniform(0.0, 1.0), 5)
    if kind == "rhs_f64":
        return {"kind": "rhs", "precision": "f64", "ic": ic, "n": _log_uniform(rng, 100, 16000), "eps": eps,
                "masses": rng.random() < 0.3}
    if kind == "rhs_mixed":
        return {"kind": "rhs", "precision": "mixed", "ic": ic, "n": _log_uniform(rng, 1000, 100000), "eps": eps,
                "masses": rng.random() < 0.3}
    if kind == "integrate_f64":
        return {"kind": "integrate", "precision": "f64", "ic": "ball", "n": _log_uniform(rng, 100, 2000), "eps": 0.01,
                "tableau": rng.choice(["DOPRI5", "RKF78"]), "tol": 1e-9, "tf": 0.05, "controller": "reference",
                "outputs": 0}
    if kind == "integrate_mixed":
        return {"kind": "integrate", "precision": "mixed", "ic": "ball", "n": _log_uniform(rng, 1000, 16000),
                "eps": 0.01, "tableau": rng.choice(["DOPRI5", "RKF78"]), "tol": 1e-9, "tf": 0.03,
                "controller": rng.choice(["reference", "pi"]), "outputs": 0}
    if kind == "batch_mixed":
        return {"kind": "batch", "precision": "mixed", "systems": rng.randint(16, 128), "n_min": 64,
                "n_max": _log_uniform(rng, 300, 4000), "tol": 1e-9, "tf": 0.04}
    if kind == "batch_f64":
        return {"kind": "batch", "precision": "f64", "systems": rng.randint(4, 24), "n_min": 64,
                "n_max": _log_uniform(rng, 100, 1000), "tol": 1e-9, "tf": 0.02}
    if kind == "leapfrog":
        return {"kind": "leapfrog", "precision": rng.choice(["f64", "mixed"]), "ic": ic,
                "n": _log_uniform(rng, 200, 3000), "eps": max(eps, 0.005), "masses": rng.random() < 0.5,
                "steps": rng.randint(4, 16)}
    if kind == "energy":
        return {"kind": "energy", "ic": ic, "n": _log_uniform(rng, 300, 16000), "eps": eps}
    if kind == "rk":
        return {"kind": "rk", "tableau": rng.choice(["RKF78", "DOPRI5"]), "n_var": 6 * _log_uniform(rng, 1000, 100000)}
    return {"kind": "train", "samples": rng.randint(300, 2000), "epochs": rng.randint(40, 100)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _directions(r, n):
    c = r.uniform(-1.0, 1.0, n)
    ph = r.uniform(0.0, 2.0 * np.pi, n)
    s = np.sqrt(1.0 - c * c)
    return np.stack([s * np.cos(ph), s * np.sin(ph), c], axis=1)


def _state(ic, n, seed):
    """Positions and velocities, 6 n numbers, centre of mass at rest at the origin."""
    r = np.random.default_rng(seed)
    if ic == "plummer":
        radius = 1.0 / np.sqrt(r.uniform(1e-3, 0.999, n) ** (-2.0 / 3.0) - 1.0)
        speed = r.beta(1.5, 4.5, n) ** 0.5 * np.sqrt(2.0) * (1.0 + radius * radius) ** -0.25
    else:
        radius = r.uniform(0.0, 1.0, n) ** (1.0 / 3.0)
        speed = np.abs(r.normal(0.0, 0.01 if ic == "cold" else 0.1, n))
    x, v = radius[:, None] * _directions(r, n), speed[:, None] * _directions(r, n)
    return np.concatenate([(x - x.mean(0)).ravel(), (v - v.mean(0)).ravel()])


def _masses(n, seed):
    m = np.random.default_rng(seed + 77).uniform(0.5, 1.5, n)
    return m / m.sum()


def _batch_sizes(case):
    k = case["systems"]
    return np.round(np.geomspace(case["n_min"], case["n_max"], k)).astype(np.int64)


def _batch_states(case, seed):
    return [_state("plummer", int(n), 1000 * seed + k) for k, n in enumerate(_batch_sizes(case))]


def _batch_eps(case):
    return 0.04 / np.cbrt(_batch_sizes(case))


def _energy_state(case, seed):
    """The system seen from a frame in which it moves, as on an orbit."""
    n = case["n"]
    x = _state(case["ic"], n, seed)
    x[: 3 * n].reshape(-1, 3)[:] += (0.5, -0.25, 0.125)
    x[3 * n:].reshape(-1, 3)[:] += (0.1, 0.2, -0.3)
    return x


def _rk_vectors(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nv = case["n_var"]
    s = gb.tableau(case["tableau"]).n_stages
    x0 = torch.randn(nv, dtype=torch.float64, device="cuda", generator=g)
    ks = torch.randn(s * nv, dtype=torch.float64, device="cuda", generator=g)
    return x0, ks


def _train_data(case, seed):
    """Features and targets with the scales of a controller log."""
    r = np.random.default_rng(seed)
    x = r.normal(-4.0, 1.0, (case["samples"], 16)).astype(np.float32)
    y = np.tanh(x[:, :4].sum(1) * 0.3 + 5.0) * 0.2 + 0.05 * r.normal(size=case["samples"])
    return x, y.astype(np.float32)


def _dev(a):
    return torch.as_tensor(a, device="cuda")


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("rhs", "leapfrog", "integrate"):
        n = case["n"]
        s["x"] = _dev(_state(case["ic"], n, seed))
        s["m"] = _dev(_masses(n, seed)) if case.get("masses") else None
        s["ode"] = gb.NBodyODE(n, case["eps"], 1.0 / n, s["m"])
    if kind == "rhs":
        s["out"] = torch.empty_like(s["x"])
        if case["precision"] == "mixed":
            s["work"] = torch.empty(gb.lib().gb_nbody_mixed_workspace_bytes(case["n"]), dtype=torch.uint8,
                                    device="cuda")
    elif kind == "leapfrog":
        s["exe"] = gb.Gb300Executor(precision=case["precision"])
    elif kind == "integrate":
        mlp = None
        if case["controller"] == "learned":
            with open(os.path.join(WEIGHTS, "proposer_plummer16384_rkf78_tol1e-11.bin"), "rb") as f:
                mlp = gb.GbMlp.from_buffer_copy(f.read())
        exe = gb.Gb300Executor(precision=case["precision"], controller=case["controller"], mlp=mlp)
        s["it"] = gb.Integrator(case["tableau"], s["ode"], exe)
        if case["outputs"]:
            s["it"].set_dense_output(_output_times(case))
    elif kind == "batch":
        s["x"] = _dev(np.concatenate(_batch_states(case, seed)))
        s["batch"] = gb.Batch("DOPRI5", _batch_sizes(case), _batch_eps(case), precision=case["precision"])
    elif kind == "energy":
        s["x"] = _dev(_energy_state(case, seed))
    elif kind == "rk":
        s["tab"] = gb.tableau(case["tableau"])
        s["x0"], s["ks"] = _rk_vectors(case, seed)
        s["stages"] = [torch.empty_like(s["x0"]) for _ in range(s["tab"].n_stages - 1)]
        s["xnew"], s["err"], s["target"] = (torch.empty_like(s["x0"]) for _ in range(3))
        s["atol"] = torch.full_like(s["x0"], 1e-8)
        s["rtol"] = torch.full_like(s["x0"], 1e-8)
    elif kind == "train":
        s["xy"] = _train_data(case, seed)
    return s


def _output_times(case):
    return np.linspace(0.0, case["tf"], case["outputs"] + 2)[1:-1]


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rhs":
        n, o = case["n"], s["ode"]
        if case["precision"] == "f64":
            return gb.nbody_rhs_f64(s["x"], n, o.softening, o.mass, o.masses, out=s["out"])
        return gb.nbody_rhs_mixed(s["x"], n, o.softening, o.mass, o.masses, out=s["out"], work=s["work"])
    if kind == "leapfrog":
        x, _ = gb.ParallelLeapfrogIntegrator.integrate(s["x"], 0.0, _leapfrog_tf(case), LEAPFROG_DT, s["ode"], None,
                                                       s["exe"])
        return x
    if kind == "integrate":
        it = s["it"]
        it.start(s["x"], 0.0, case["tf"], case["tol"], case["tol"])
        gb.check(it.advance(), "advance")
        x, t = it.state()
        return {"x": x, "t": t, "samples": it.dense_output() if case["outputs"] else None}
    if kind == "batch":
        b = s["batch"]
        b.start(s["x"], 0.0, case["tf"], case["tol"], case["tol"])
        gb.check(b.advance(), "advance")
        x, t = b.state()
        return {"x": x, "t": t}
    if kind == "energy":
        n = case["n"]
        return gb.energy(s["x"], n, case["eps"], 1.0 / n)
    if kind == "rk":
        t, nv, x0, ks = s["tab"], case["n_var"], s["x0"], s["ks"]
        for k, y in enumerate(s["stages"]):
            gb.rk_stage(t, k + 1, RK_DT, x0, ks, y, nv)
        gb.rk_update(t, RK_DT, x0, ks, s["xnew"], s["err"], nv)
        gb.rk_error_target(s["atol"], s["rtol"], s["xnew"], x0, s["target"], nv)
        return {"stages": s["stages"], "x": s["xnew"], "err": s["err"], "target": s["target"],
                "norm": gb.rk_norm(s["err"], s["target"], nv)}
    x, y = s["xy"]
    m, loss = learned.train(x, y, epochs=case["epochs"])
    return {"weights": np.frombuffer(bytes(m), dtype=np.float32), "loss": loss}


LEAPFROG_DT = 1.0 / 1024
RK_DT = 1e-3


def _leapfrog_tf(case):
    return case["steps"] * LEAPFROG_DT  # exact: the step is a power of two


# ---------------------------------------------------------------------------
# the work of one pass: inputs read once, outputs written once, 20 operations an ordered pair
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "rhs":
        n = case["n"]
        return {"bytes": 96 * n + (8 * n if case.get("masses") else 0), "flops": FLOPS * n * (n - 1)}
    if kind == "leapfrog":
        n = case["n"]
        return {"bytes": 96 * n + (8 * n if case.get("masses") else 0),
                "flops": FLOPS * n * (n - 1) * (case["steps"] + 1)}
    if kind == "integrate":
        # right-hand sides of the accepted steps of a typical run (steps of 0.002 at tol 1e-9 to 1e-11 with
        # DOPRI5, twice that with RKF78)
        n = case["n"]
        rhs = math.ceil(case["tf"] / 0.002) * 6 if case["tableau"] == "DOPRI5" else math.ceil(case["tf"] / 0.004) * 13
        return {"bytes": 96 * n + 48 * n * case["outputs"], "flops": FLOPS * n * (n - 1) * rhs}
    if kind == "batch":
        sizes = _batch_sizes(case).astype(float)
        rhs = math.ceil(case["tf"] / 0.004) * 6
        return {"bytes": 96 * float(sizes.sum()), "flops": FLOPS * float((sizes * (sizes - 1)).sum()) * rhs}
    if kind == "energy":
        n = case["n"]
        return {"bytes": 48 * n + 64, "flops": FLOPS // 2 * n * (n - 1)}
    if kind == "rk":
        t, nv = gb.tableau(case["tableau"]), case["n_var"]
        s = t.n_stages
        nnz = sum(t.a[k][j] != 0.0 for k in range(s - 1) for j in range(k + 1))
        upd = sum(t.b[j] != 0.0 for j in range(s)) + sum(t.b[j] != t.bt[j] for j in range(s))
        # x0, the stage derivatives and both tolerances in; the stage states, x, its error and target out
        return {"bytes": 8 * nv * (1 + s + 2 + (s - 1) + 3) + 8, "flops": nv * (2 * (nnz + upd) + 2 * s + 8)}
    weights = 16 * 64 + 64 * 64 + 64
    return {"bytes": 68 * case["samples"] + 8 * weights, "flops": 6 * weights * case["samples"] * case["epochs"]}


# ---------------------------------------------------------------------------
# the same in 64 bits, with torch
# ---------------------------------------------------------------------------
def _acc(x, eps, m):
    """Accelerations of bodies at x (n, 3), masses m (a number or n of them), rows at a time."""
    n = x.shape[0]
    out = torch.empty_like(x)
    rows = max(1, min(n, (1 << 26) // n))
    w = m if torch.is_tensor(m) else torch.full((n,), m, dtype=x.dtype, device=x.device)
    for i in range(0, n, rows):
        d = x[None, :, :] - x[i:i + rows, None, :]
        f = d.square().sum(2).add_(eps * eps)
        f = w / (f * f.sqrt())
        out[i:i + rows] = torch.bmm(f[:, None, :], d)[:, 0]
    return out


_DP_C = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
         (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
         (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
         (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))


def _orbit(x, eps, m, times, h_max):
    """The state at each of `times`: fixed steps of the fifth-order Dormand-Prince formula, short enough that
    their error is below the tolerance of the run that they stand for."""
    n = x.numel() // 6
    f = lambda y: torch.cat([y[3 * n:], _acc(y[: 3 * n].view(n, 3), eps, m).reshape(-1)])  # noqa: E731
    t, got = 0.0, []
    for to in times:
        k = max(1, math.ceil((to - t) / h_max - 1e-9))
        h = (to - t) / k
        for _ in range(k):
            ks = [f(x)]
            for row in _DP_C:
                y = x + h * sum(c * kj for c, kj in zip(row, ks) if c)
                if len(ks) < 6:
                    ks.append(f(y))
            x = y
        t = to
        got.append(x)
    return got


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhs":
        n = case["n"]
        x = _dev(_state(case["ic"], n, seed))
        m = _dev(_masses(n, seed)) if case.get("masses") else 1.0 / n
        return torch.cat([x[3 * n:], _acc(x[: 3 * n].view(n, 3), case["eps"], m).reshape(-1)])
    if kind == "leapfrog":
        n, h = case["n"], LEAPFROG_DT
        x = _dev(_state(case["ic"], n, seed))
        m = _dev(_masses(n, seed)) if case.get("masses") else 1.0 / n
        p, v = x[: 3 * n].view(n, 3).clone(), x[3 * n:].view(n, 3).clone()
        a = _acc(p, case["eps"], m)
        for _ in range(case["steps"]):
            p += h * (v + 0.5 * h * a)
            b = _acc(p, case["eps"], m)
            v += 0.5 * h * (a + b)
            a = b
        return torch.cat([p.reshape(-1), v.reshape(-1)])
    if kind == "integrate":
        n = case["n"]
        x = _dev(_state(case["ic"], n, seed))
        times = [float(t) for t in _output_times(case)] if case["outputs"] else []
        got = _orbit(x, case["eps"], 1.0 / n, times + [case["tf"]], 0.001)
        return {"x": got[-1], "t": np.float64(case["tf"]),
                "samples": torch.stack(got[:-1]).cpu().numpy() if case["outputs"] else None}
    if kind == "batch":
        got = [_orbit(_dev(x), float(e), 1.0 / int(n), [case["tf"]], 0.002)[0]
               for x, e, n in zip(_batch_states(case, seed), _batch_eps(case), _batch_sizes(case))]
        return {"x": torch.cat(got), "t": np.full(case["systems"], case["tf"])}
    if kind == "energy":
        n = case["n"]
        s = _dev(_energy_state(case, seed))
        x, v = s[: 3 * n].view(n, 3), s[3 * n:].view(n, 3)
        ke = 0.5 / n * v.square().sum().item()
        pe = 0.0
        for i in range(0, n, 1024):
            r2 = (x[None, :, :] - x[i:i + 1024, None, :]).square().sum(2) + case["eps"] ** 2
            pe -= 0.5 / n / n * r2.rsqrt().sum().item()
        pe += 0.5 / n / case["eps"]  # no body acts on itself
        return {"ke": np.float64(ke), "pe": np.float64(pe), "e": np.float64(ke + pe), "p": v.mean(0).cpu().numpy(),
                "l": torch.linalg.cross(x, v).mean(0).cpu().numpy()}
    if kind == "rk":
        t, nv = gb.tableau(case["tableau"]), case["n_var"]
        x0, ks = _rk_vectors(case, seed)
        k = ks.view(t.n_stages, nv)
        stages = [x0 + RK_DT * sum(t.a[i][j] * k[j] for j in range(i + 1)) for i in range(t.n_stages - 1)]
        x = x0 + RK_DT * sum(t.b[j] * k[j] for j in range(t.n_stages))
        err = RK_DT * sum((t.b[j] - t.bt[j]) * k[j] for j in range(t.n_stages))
        target = 1e-8 + 1e-8 * torch.maximum(x.abs(), x0.abs())
        return {"stages": stages, "x": x, "err": err, "target": target,
                "norm": ((err / target).square().sum() / nv).sqrt().reshape(1)}
    return None  # a hundred Adam steps in 32 bits: the trained weights have no 64-bit value
