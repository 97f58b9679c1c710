"""Performance cases of the ensemble solver and of the surrogate network.

A case is one call that a user's program makes: an ensemble handed to the
solver with host arrays, integrated over one or more acoustic periods and read
back, or one pass of the surrogate network on device tensors.  ``listed()``
gives the named cases, ``draw(rng)`` others of the same ranges, ``prepare`` what
the program holds before the call, ``run`` the call itself with its whole
results, ``work`` the bytes and operations it cannot do without and ``exact``
what it returns in plain 64-bit numpy or torch where that is quick enough.

Every period has a budget of attempted steps (``budget``), as long sweeps are
run: a system at its minimum step ends there instead of holding the others up.
"""
import math

import numpy as np
import torch

from bubbleensemble_implicitextension_b200 import solver as S
from bubbleensemble_implicitextension_b200 import surrogate as SG
from bubbleensemble_implicitextension_b200 import workloads as W

V = S.ListOfVariables
O = S.ListOfSolverOptions


def listed():
    return [
        # one small cluster of bubbles, one period: the shortest call (latency of one system's serial chain)
        {"name": "cluster_1x8", "kind": "line", "n_pa": 1, "n_f": 1, "units": 8, "geometry": False, "recurrence": 0,
         "pa_lo": 0.9, "pa_hi": 0.9, "f_lo": 90.0, "f_hi": 90.0, "periods": 1, "reset": -1, "budget": 10000},
        # amplitude x frequency map of one 32-bubble line, the bubbles' geometry shared and the radii as factors,
        # with the single-reduction recurrence
        {"name": "map_256x32_geometry", "kind": "line", "n_pa": 16, "n_f": 16, "units": 32, "geometry": True,
         "recurrence": 1, "pa_lo": 0.5, "pa_hi": 2.0, "f_lo": 20.0, "f_hi": 200.0, "periods": 1, "reset": -1,
         "budget": 10000},
        # the same map with the coupling matrix in the reference's format and every option at its default
        {"name": "map_256x32_matrix", "kind": "line", "n_pa": 16, "n_f": 16, "units": 32, "geometry": False,
         "recurrence": 0, "pa_lo": 0.5, "pa_hi": 2.0, "f_lo": 20.0, "f_hi": 200.0, "periods": 1, "reset": -1,
         "budget": 10000},
        # training data for the surrogate: random drives, one radius draw and one matrix per system, the first
        # period discarded
        {"name": "runs_1024x32", "kind": "runs", "systems": 1024, "units": 32, "periods": 2, "reset": 1,
         "budget": 3000},
        # uneven clouds of 4 to 64 bubbles in one launch plan, dual-frequency drive, two tolerances
        {"name": "mixed_384", "kind": "mixed", "each": 64, "budget": 1500},
        # one 128-bubble geometry shared by systems that differ in their initial radii
        {"name": "shared_512x128", "kind": "cloud", "systems": 512, "units": 128, "own_radii": False,
         "shared": True, "recurrence": 0, "budget": 4000},
        # one geometry, each system with its own radii; an odd number of bubbles
        {"name": "radii_256x51", "kind": "cloud", "systems": 256, "units": 51, "own_radii": True, "shared": True,
         "recurrence": 0, "budget": 4000},
        # own matrix per system above 64 bubbles, an odd number of them
        {"name": "own_148x101", "kind": "cloud", "systems": 148, "units": 101, "own_radii": True, "shared": False,
         "recurrence": 0, "budget": 2000},
        # rings coupled to their neighbours only: banded storage
        {"name": "ring_512x128", "kind": "ring", "systems": 512, "units": 128, "band": 1, "budget": 4000},
        # fixed-step integration with dense output of the trajectories
        {"name": "rk4_dense_64x16", "kind": "rk4", "systems": 64, "units": 16, "steps": 1000, "slots": 64},
        # the network over a sweep's grid of 128 x 128 points
        {"name": "network_forward_16384", "kind": "forward", "batch": 16384, "width": 256, "depth": 4},
        # one training step of the network on a minibatch: loss, gradients, Adam
        {"name": "network_train_512", "kind": "train", "batch": 512, "width": 256, "depth": 4},
    ]


_SIZES = (4, 8, 16, 32, 48, 64)   # bubbles of the uneven clouds


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "runs", "mixed", "cloud", "cloud", "ring", "rk4", "forward", "train"])
    if kind == "line":
        lo, flo = rng.uniform(0.4, 1.0), rng.uniform(20.0, 100.0)
        return {"kind": kind, "n_pa": rng.randint(1, 16), "n_f": rng.randint(1, 16), "units": rng.randint(4, 32),
                "geometry": rng.random() < 0.5, "recurrence": rng.randint(0, 1), "pa_lo": lo,
                "pa_hi": lo + rng.uniform(0.1, 1.0), "f_lo": flo, "f_hi": 2.0 * flo, "periods": 1, "reset": -1,
                "budget": 8000}
    if kind == "runs":
        return {"kind": kind, "systems": _log_int(rng, 32, 1024), "units": rng.randint(6, 32), "periods": 2,
                "reset": 1, "budget": 2500}
    if kind == "mixed":
        return {"kind": kind, "each": _log_int(rng, 2, 64), "budget": 1200}
    if kind == "cloud":
        shared = rng.random() < 0.6
        return {"kind": kind, "systems": _log_int(rng, 8, 384 if shared else 148), "units": rng.randint(33, 128),
                "own_radii": rng.random() < 0.5 if shared else True, "shared": shared,
                "recurrence": rng.randint(0, 1), "budget": 1500}
    if kind == "ring":
        return {"kind": kind, "systems": _log_int(rng, 8, 512), "units": rng.randint(8, 128),
                "band": rng.randint(1, 3), "budget": 3000}
    if kind == "rk4":
        return {"kind": kind, "systems": _log_int(rng, 4, 256), "units": rng.randint(4, 32),
                "steps": rng.randint(400, 1000), "slots": rng.randint(4, 64)}
    if kind == "forward":
        return {"kind": kind, "batch": _log_int(rng, 64, 65536), "width": rng.choice([64, 96, 128, 256]),
                "depth": rng.randint(2, 4)}
    return {"kind": "train", "batch": _log_int(rng, 64, 1024), "width": rng.choice([64, 96, 128, 256]),
            "depth": rng.randint(2, 4)}


# ---- ensembles ---------------------------------------------------------------------------------

def _cloud(case, seed):
    n, ns = case["units"], case["systems"]
    if case["own_radii"]:
        ens = W.c3_radii_ensemble(n_systems=ns, n_units=n, seed=1000 * seed, n_periods=1)
        return ens if case["shared"] else W.explicit_matrices(ens)
    return W.c3_ensemble(n_systems=ns, n_units=n, seed=seed, n_periods=1)


def _ensemble(case, seed):
    kind = case["kind"]
    if kind == "line":
        ens = W.c1_ensemble(n_pa=case["n_pa"], n_f=case["n_f"], n_units=case["units"], seed=seed,
                            n_periods=case["periods"], reset_at=case["reset"],
                            pa_range=(case["pa_lo"], case["pa_hi"]), f_range=(case["f_lo"], case["f_hi"]),
                            factored=case["geometry"])
    elif kind == "runs":
        rng = np.random.default_rng(seed)
        ns = case["systems"]
        pa = rng.uniform(0.5, 2.0, ns)
        fr = 10.0 ** rng.uniform(np.log10(20.0), np.log10(200.0), ns)
        R = rng.uniform(2.0, 8.0, (ns, case["units"]))
        ens = SG.line_ensemble(pa, fr, R, n_periods=case["periods"], reset_at=case["reset"])
    elif kind == "mixed":
        # the first `each` systems of every size: other inputs, the same shapes
        every = W.c2_ensemble(n_systems=12 * case["each"] + 96, seed=seed, n_periods=1, reset_at=-1)
        chosen = np.concatenate([np.nonzero(every.units == n)[0][:case["each"]] for n in _SIZES])
        ens = every.subset(np.sort(chosen))
    elif kind == "cloud":
        ens = _cloud(case, seed)
    elif kind == "ring":
        ens = W.ring_ensemble(n_systems=case["systems"], n_units=case["units"], band_width=case["band"], seed=seed)
    else:
        rng = np.random.default_rng(seed)
        ns = case["systems"]
        ens = SG.line_ensemble(rng.uniform(0.2, 0.6, ns), rng.uniform(80.0, 200.0, ns),
                               rng.uniform(2.0, 8.0, (ns, case["units"])), n_periods=1, reset_at=-1)
        ens.dt0 = 1.0 / case["steps"]
    ens.max_steps_per_period = case.get("budget", 1_000_000)
    return ens


def _network(case, seed):
    rng = np.random.default_rng(seed)
    b = case["batch"]
    radii = rng.uniform(2.0, 8.0, (b, 32))
    x = SG.features(rng.uniform(0.5, 2.0, b), 10.0 ** rng.uniform(np.log10(20.0), np.log10(200.0), b), radii)
    # outputs of a smooth map with the ranges of (log10 collapse strength, max R/R_E)
    t = np.stack([0.4 * x[:, 0] * (2.3 - x[:, 1]) + 0.2 * np.sin(3.0 * x[:, 0]), 1.0 + x[:, 0] * (2.5 - x[:, 1])], 1)
    norm = [np.asarray(a, np.float32) for a in (x.mean(0), x.std(0) + 1e-6, t.mean(0), t.std(0) + 1e-6)]
    return x.astype(np.float32), t.astype(np.float32), norm


def prepare(case, seed):
    if case["kind"] in ("forward", "train"):
        x, t, norm = _network(case, seed)
        net = SG.MLP(width=case["width"], depth=case["depth"], max_batch=4096, seed=seed)
        net.set_normalization(*norm)
        return {"kind": case["kind"], "net": net, "x": torch.as_tensor(x, device="cuda"),
                "t": torch.as_tensor(t, device="cuda")}
    ens = _ensemble(case, seed)
    rk4 = case["kind"] == "rk4"
    ps = ens.make_solver(algorithm=S.Algorithms.RK4 if rk4 else S.Algorithms.RKCK45,
                         n_dense_output=case.get("slots", 0))
    if case.get("recurrence"):
        ps.SolverOption(O.BiCGRecurrence, 1)
    if rk4:
        ps.SolverOption(O.DenseOutputMinimumTimeStep, 1.0 / case["slots"])
    ps.SynchroniseFromHostToDevice(V.All)
    ps.InsertSynchronisationPoint()
    ps.SynchroniseSolver()
    return {"kind": case["kind"], "solver": ps, "periods": ens.n_periods, "reset": ens.reset_at, "state": ens.state,
            "uacc": ens.initial_uacc(), "iuacc": ens.initial_iuacc(), "dense": rk4, "index": np.zeros(ens.n_systems)}


def run(st):
    if st["kind"] == "forward":
        return st["net"].forward(st["x"])
    if st["kind"] == "train":
        net = st["net"]
        loss = net.backward(st["x"], st["t"])
        net.adam_step(1e-3)
        return {"loss": loss, "gradients": net.gradients()}
    ps = st["solver"]
    ps.set_array(V.ActualState, st["state"])
    ps.set_array(V.UnitAccessories, st["uacc"])
    ps.set_array(V.IntegerUnitAccessories, st["iuacc"])
    for var in (V.ActualState, V.UnitAccessories, V.IntegerUnitAccessories):
        ps.SynchroniseFromHostToDevice(var)
    if st["dense"]:
        ps.set_array(V.DenseIndex, st["index"])
        ps.SynchroniseFromHostToDevice(V.DenseOutput)
    ps.solve_periods(st["periods"], st["reset"])
    out = [V.ActualState, V.ActualTime, V.UnitAccessories, V.IntegerUnitAccessories]
    for var in out + ([V.DenseOutput] if st["dense"] else []):
        ps.SynchroniseFromDeviceToHost(var)
    ps.InsertSynchronisationPoint()
    ps.SynchroniseSolver()
    if st["dense"]:
        out += [V.DenseIndex, V.DenseTime, V.DenseState]
    return {var.name: ps.get_array(var) for var in out}


# ---- work --------------------------------------------------------------------------------------

# attempted steps and BiCG iterations per right-hand side of a typical system of each kind
_STEPS = {"line": 3000, "runs": 3000, "mixed": 1500, "cloud": 1500, "ring": 1500}
_ITERATIONS = {"line": 7.0, "runs": 7.0, "mixed": 8.0, "cloud": 9.0, "ring": 6.0, "rk4": 4.0}


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        w, d, b = case["width"], case["depth"], case["batch"]
        weights = SG.N_IN * w + (d - 1) * w * w + w * SG.N_OUT
        params = weights + d * w + SG.N_OUT
        if kind == "forward":
            return {"bytes": 4.0 * b * (SG.N_IN + SG.N_OUT) + 2.0 * weights + 4.0 * (params - weights),
                    "flops": 2.0 * b * weights}
        # a step reads the weights, writes the gradients and updates the weights and both moments
        return {"bytes": 4.0 * b * (SG.N_IN + SG.N_OUT) + 4.0 * (params * 8), "flops": 6.0 * b * weights}
    if kind == "mixed":
        ns, n1, n2 = 6 * case["each"], sum(_SIZES) / 6.0, sum(n * n for n in _SIZES) / 6.0
        couplings = n2
    else:
        ns = case["systems"] if "systems" in case else case["n_pa"] * case["n_f"]
        n1, n2 = case["units"], case["units"] ** 2
        couplings = n2 if kind == "ring" or kind in ("runs", "rk4") or case.get("shared") is False else n2 / ns
        if kind == "ring":
            n2 = case["units"] * (2 * case["band"] + 1)
    k = _ITERATIONS[kind]
    rhs = 55 * n1 + 5 * n2 + 5 * n1 + k * (6 * n2 + 17 * n1)
    if kind == "rk4":
        steps, stages, periods = case["steps"], 4, 1
    else:
        steps, stages, periods = min(_STEPS[kind], case["budget"]), 6, case.get("periods", 1)
    slots = case.get("slots", 0)
    # state, unit parameters, accessories and the coupling in; state, accessories and dense output out
    per_unit = 8 * (2 + 21 + 64 + 2 + 64) + 8 + 16 * slots
    return {"bytes": ns * (n1 * per_unit + 8.0 * couplings + 80.0),
            "flops": float(ns) * periods * steps * (stages * rhs + 110 * n1)}


# ---- exact results -----------------------------------------------------------------------------

def _layers(p, width, depth):
    sizes = [(SG.N_IN if l == 0 else width, SG.N_OUT if l == depth else width) for l in range(depth + 1)]
    out, k = [], 0
    for i, o in sizes:
        out.append((p[k:k + i * o].reshape(o, i), p[k + i * o:k + i * o + o]))
        k += i * o + o
    return out


def _exact_network(case, seed):
    x, t, norm = _network(case, seed)
    net = SG.MLP(width=case["width"], depth=case["depth"], max_batch=16, seed=seed)
    p = torch.as_tensor(net.parameters()).double().requires_grad_(True)
    net.close()
    im, sd, om, os_ = (torch.as_tensor(a).double() for a in norm)
    a = (torch.as_tensor(x).double() - im) / sd
    layers = _layers(p, case["width"], case["depth"])
    for l, (w, b) in enumerate(layers):
        a = a @ w.T + b
        if l + 1 < len(layers):
            a = torch.nn.functional.gelu(a, approximate="tanh")
    if case["kind"] == "forward":
        return (a * os_ + om).detach()
    loss = ((a - (torch.as_tensor(t).double() - om) / os_) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "gradients": p.grad.numpy()}


def _rhs(T, X, u, C):
    """Derivatives of [systems, 2, units] states: the coupled accelerations from a direct solve."""
    r, v = X[:, 0], X[:, 1]
    p = r ** -u[10]
    g = u[9] * v + 1.0
    s1, c1 = np.sin(2.0 * np.pi * T), np.cos(2.0 * np.pi * T)
    ang = 2.0 * np.pi * u[11] * T + u[12]
    single = (u[11] == 0.0) & (u[12] == 0.0)
    s2, c2 = np.where(single, 0.0, np.sin(ang)), np.where(single, 1.0, np.cos(ang))
    num = (u[0] + u[1] * v) * p - u[2] * g - u[3] / r - u[4] * v / r - (1.5 - 0.5 * u[9] * v) * v * v
    num = num - (u[5] * s1 + u[6] * s2) * g - r * (u[7] * c1 + u[8] * c2)
    den = r - u[9] * r * v + u[4] * u[9]
    A = C * (r * r)[:, None, :] / den[:, :, None]
    A[:, np.arange(r.shape[1]), np.arange(r.shape[1])] += 1.0
    b = num / den + np.einsum("sij,sj->si", C, -2.0 * r * v * v) / den
    return np.stack([v, np.linalg.solve(A, b[..., None])[..., 0]], 1)


_NODES = (0.0, 1 / 5, 3 / 10, 3 / 5, 1.0, 7 / 8)
_STAGES = ((), (1 / 5,), (3 / 40, 9 / 40), (3 / 10, -9 / 10, 6 / 5), (-11 / 54, 5 / 2, -70 / 27, 35 / 27),
           (1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096))
_FIFTH = (37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771)
_FOURTH = (2825 / 27648, 0.0, 18575 / 48384, 13525 / 55296, 277 / 14336, 1 / 4)


def _step(case, T, h, X, u, C):
    """One trial step of every system: the new states and, with RKCK45, the error estimates."""
    hh, t = h[:, None, None], T[:, None]
    if case["kind"] == "rk4":
        k1 = _rhs(t, X, u, C)
        k2 = _rhs(t + 0.5 * h[:, None], X + 0.5 * hh * k1, u, C)
        k3 = _rhs(t + 0.5 * h[:, None], X + 0.5 * hh * k2, u, C)
        k4 = _rhs(t + h[:, None], X + hh * k3, u, C)
        return X + hh * (k1 + 2.0 * k2 + 2.0 * k3 + k4) / 6.0, None
    k = []
    for node, row in zip(_NODES, _STAGES):
        k.append(_rhs(t + node * h[:, None], X + hh * sum((a * f for a, f in zip(row, k)), 0.0 * X), u, C))
    Y = X + hh * sum(c * f for c, f in zip(_FIFTH, k))
    return Y, hh * np.abs(sum((c - d) * f for c, d, f in zip(_FIFTH, _FOURTH, k))) + 1e-18


def _exact_trajectories(case, seed):
    """One period of every system, each with its own time and step size; an event cuts its system's step."""
    ens = _ensemble(case, seed)
    ns, n, slots = ens.n_systems, case["units"], case.get("slots", 0)
    u = ens.upar.reshape(W.NUP, ns, n)
    X = ens.state.reshape(2, ns, n).transpose(1, 0, 2).copy()
    C = ens.coupling.reshape(-1, n, n)[ens.matrix_of_system].transpose(0, 2, 1)
    uacc, count = np.zeros((2 * W.NCOLL, ns, n)), np.full((ns, n), -1)
    dt0, ev, T, taken = ens.dt0, X[:, 1].copy(), np.zeros(ns), 0
    newdt, done = np.full(ns, dt0), np.zeros(ns, bool)
    d_idx, d_time, due = np.ones(ns, np.int64), np.zeros((slots, ns)), np.full(ns, 1.0 / max(slots, 1))
    d_state = np.zeros((slots, 2, ns, n))
    d_state[:1] = X.transpose(1, 0, 2)
    sys_i, unit_i = np.meshgrid(np.arange(ns), np.arange(n), indexing="ij")
    while not done.all() and taken < ens.max_steps_per_period:
        taken += 1
        last = newdt > 1.0 - T
        h = np.where(last, 1.0 - T, newdt)
        Y, err = _step(case, T, h, X, u, C)
        if err is None:
            newdt, ok = np.full(ns, dt0), ~done
        else:
            tol = np.maximum(ens.rtol.T[:, :, None] * np.maximum(np.abs(Y), np.abs(X)), ens.atol.T[:, :, None])
            passed, room = (err < tol).all((1, 2)), (tol / err).min((1, 2))
            grow = 0.8 * room ** np.where(passed, 0.2, 0.25)
            newdt = np.clip(h * np.clip(grow, ens.shrink, ens.grow), ens.dtmin, ens.dtmax)
            ok = passed & ~done
        n_ev = Y[:, 1]
        cross = (ev > ens.event_tol) & (n_ev < -ens.event_tol)
        with np.errstate(divide="ignore", invalid="ignore"):
            where = np.minimum(np.where(cross, -ev / (n_ev - ev) * h[:, None], np.inf).min(1), h)
        cut = ok & cross.any(1) & (where >= ens.dtmin)
        newdt = np.where(cut, where, newdt)
        ok &= ~cut
        T = np.where(ok, T + h, T)
        X = np.where(ok[:, None, None], Y, X)
        slot = np.clip(count, -1, W.NCOLL - 1) + W.NCOLL
        low = ok[:, None] & (count < W.NCOLL) & (X[:, 0] < uacc[slot, sys_i, unit_i])
        uacc[slot[low], sys_i[low], unit_i[low]] = X[:, 0][low]
        hit = ok[:, None] & (ev > ens.event_tol) & (np.abs(n_ev) < ens.event_tol)
        count = count + hit
        rec = hit & (count < W.NCOLL)
        for first in (0, W.NCOLL):
            uacc[count[rec] + first, sys_i[rec], unit_i[rec]] = X[:, 0][rec]
        ev = np.where(ok[:, None], X[:, 1], ev)
        end = ok & last
        for s in np.nonzero(ok & (d_idx < slots) & ((due < T) | end))[0]:
            d_state[d_idx[s], :, s] = X[s]
            d_time[d_idx[s], s] = T[s]
            d_idx[s] += 1
            due[s] = min(T[s] + 1.0 / slots, 1.0)
        done |= end
    out = {"ActualState": X.transpose(1, 0, 2).reshape(-1), "ActualTime": T, "UnitAccessories": uacc.reshape(-1),
           "IntegerUnitAccessories": count.reshape(-1).astype(np.int32)}
    if slots:
        out.update(DenseIndex=d_idx.astype(np.int32), DenseTime=d_time.reshape(-1), DenseState=d_state.reshape(-1))
    return out


def exact(case, seed):
    """The network's results, the fixed-step trajectories and those of a few small systems in 64 bits; the larger
    ensembles (thousands of adaptive steps, each with six coupled solves of every system) take minutes in numpy."""
    if case["kind"] in ("forward", "train"):
        return _exact_network(case, seed)
    if case["kind"] == "rk4" and case["systems"] * case["units"] <= 1024:
        return _exact_trajectories(case, seed)
    if case["kind"] == "line" and not case["geometry"] and case["n_pa"] * case["n_f"] * case["units"] <= 64:
        return _exact_trajectories(case, seed)
    return None
