"""The work that a user of this framework has it do, as measurable cases.

Three kinds of program stand behind the cases:

* a run of one MPCD + active-colloid system (`system`), in either precision form, which steps
  the system and takes the state out at the end of an output interval; or, as the reference's
  main() does, reads the diagnostics after every step;
* a batched ensemble of independent replicas of uneven size (`ensemble`);
* the learned closure: training steps (`train`), inference over a batch (`forward`) and the
  colloid-only dynamics that it drives (`surrogate`).

A pass of a stepping case advances the state of the program, so each pass continues the run of
the pass before it, as a user's program would.
"""
import math

import numpy as np
import torch

import brownian_gb300 as bg
from brownian_gb300 import closure

STATE = ("pos_fl", "vel_fl", "pos_colloid", "vel_colloid", "ang_vel_colloid", "ra", "f")
DIAG = ("ke_fluid", "ke_colloid", "ang_ke_colloid", "potential_colloid", "energy_colloid", "temperature_fluid")
IN, HID, OUT, NY = 81, 256, 12, 6
LAYERS = ((IN, HID), (HID, HID), (HID, HID), (HID, OUT))
SUR_RADIUS, SUR_DENSITY, SUR_DRAG = 2.0, 10, 0.05


def _system(name, box, density, colloids, radius, precision, steps, **kw):
    case = {"name": name, "kind": "system", "lx": box[0], "ly": box[1], "lz": box[2], "density": density,
            "colloids": colloids, "radius": radius, "precision": precision, "steps": steps, "n_sub": 10,
            "theta": 90.0, "v0": 0.01, "dr": 0.001, "diag": False}
    case.update(kw)
    return case


def listed():
    return [
        # the small system: a run that fits a workstation, where latency and launches count
        _system("fp64_20cube", (20, 20, 20), 10.0, 20, 2.0, "fp64", 50),
        # the reference's own workload (30^3, density 10, ten colloids, 130 degrees, no rotational
        # diffusion), driven as its main() does, with the diagnostics read after every step
        _system("fp64_30cube_diag", (30, 30, 30), 10.0, 10, 2.0, "fp64", 20, theta=130.0, dr=0.0, diag=True),
        # an uneven, crowded box with another density: a suspension at a fifth volume fraction
        _system("fp64_ragged_dense", (53, 37, 41), 7.3, 480, 2.0, "fp64", 20),
        # the headline system in both precision forms
        _system("fp64_64cube", (64, 64, 64), 10.0, 500, 2.0, "fp64", 50),
        _system("fp32c_64cube", (64, 64, 64), 10.0, 500, 2.0, "fp32c", 50),
        # a small box in the form that ensembles and sweeps use one system at a time
        _system("fp32c_24cube", (24, 24, 24), 10.0, 30, 2.0, "fp32c", 50, v0=0.05),
        # the large system: 21 million particles, 2,000 large colloids, 20 substeps
        _system("fp32c_128cube", (128, 128, 128), 10.0, 2000, 3.0, "fp32c", 20, n_sub=20, theta=130.0, v0=0.02,
                dr=0.0005),
        # a sweep over activity, crowding and box size, all replicas stepped together
        {"name": "ensemble_32", "kind": "ensemble", "replicas": 32, "density": 10, "steps": 20},
        # training: consecutive mini-batches of an epoch; then inference over a held-out batch
        {"name": "train_8192", "kind": "train", "batch": 8192, "batches": 8},
        {"name": "forward_16384", "kind": "forward", "rows": 16384},
        # colloid-only dynamics over the range that it is deployed in
        {"name": "surrogate_500", "kind": "surrogate", "colloids": 500, "fraction": 0.1, "steps": 200},
        {"name": "surrogate_2000", "kind": "surrogate", "colloids": 2000, "fraction": 0.2, "steps": 200},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("system",) * 7 + ("ensemble",) + ("train", "forward", "surrogate", "surrogate"))
    if kind == "system":
        side = _log(rng, 12, 80)
        box = [max(10, int(side * rng.uniform(0.8, 1.25))) for _ in range(3)]
        radius = rng.choice((1.5, 2.0, 2.0, 2.5, 3.0))
        volume = box[0] * box[1] * box[2]
        fraction = _log(rng, 0.01, 0.2)
        colloids = max(1, min(2000, int(fraction * volume / (4.0 / 3.0 * math.pi * radius ** 3))))
        c = _system("", box, round(rng.uniform(5.0, 15.0), 2), colloids, radius, rng.choice(("fp64", "fp32c")),
                    rng.choice((10, 17, 20)), n_sub=rng.choice((5, 10, 10, 20)),
                    theta=rng.choice((90.0, 130.0)), v0=round(rng.uniform(0.0, 0.1), 3),
                    dr=rng.choice((0.0, 0.0005, 0.001)), diag=rng.random() < 0.25)
        del c["name"]
        return c
    if kind == "ensemble":
        return {"kind": kind, "replicas": int(_log(rng, 3, 32)), "density": rng.choice((7, 10)), "steps": rng.choice((10, 20))}
    if kind == "train":
        return {"kind": kind, "batch": int(_log(rng, 200, 16384)), "batches": rng.randint(2, 8)}
    if kind == "forward":
        return {"kind": kind, "rows": int(_log(rng, 1, 65536))}
    return {"kind": kind, "colloids": int(_log(rng, 20, 2000)), "fraction": round(_log(rng, 0.02, 0.2), 3),
            "steps": rng.choice((50, 117, 200))}


# ---------------------------------------------------------------------------- one system

def _params(box, n_fluid, colloids, radius, density, precision, **kw):
    mass = bg.displaced_mass(radius, density)
    return dict(L=box, n_fluid=n_fluid, n_colloid=colloids, mass_colloid=mass, sig_colloid=2 * radius,
                sigma=2 * radius, I_colloid=0.4 * mass * radius ** 2,
                precision=bg.FP64 if precision == "fp64" else bg.FP32C, init_gap=0.2 if radius < 2 else 0.5, **kw)


def _system_params(case, seed):
    box = (case["lx"], case["ly"], case["lz"])
    return _params(box, int(box[0] * box[1] * box[2] * case["density"]), case["colloids"], case["radius"],
                   case["density"], case["precision"], n_sub=case["n_sub"], theta_deg=case["theta"], v0=case["v0"],
                   Dr=case["dr"], seed=1 + seed)


def _pinned(rows):
    # page-locked, so that reading the state out is a direct copy
    return torch.zeros((rows, 3), dtype=torch.float64).pin_memory().numpy()


def _out(n_fluid, colloids):
    return {k: _pinned(n_fluid if k in ("pos_fl", "vel_fl") else colloids) for k in STATE}


def _prepare_system(case, seed):
    sim = bg.Simulation(**_system_params(case, seed))
    sim.initialize(bg.INIT_PHYSICAL)
    sim.setup()
    return {"kind": "system", "sim": sim, "steps": case["steps"], "diag": case["diag"], "out": _out(sim.N, sim.Nc)}


def _run_system(s):
    sim = s["sim"]
    if not s["diag"]:
        sim.step(s["steps"])
        return sim.get_state(s["out"])
    rows = []
    for _ in range(s["steps"]):
        sim.step(1)
        d = sim.diag()
        rows.append([d[k] for k in DIAG] + d["momentum"])
    return dict(sim.get_state(s["out"]), diag=np.array(rows))


def _work_system(n, cells, steps, n_sub, precision, diags=0):
    # a step reads and writes every particle's position and velocity once and every cell's sums
    # (count, momentum, energy) once; at the end the state goes out as 64-bit triplets
    particle = 96 if precision == "fp64" else 56
    cell = 2 * 40
    flops = 18 + 9 + 6 * n_sub  # per particle: rotation about the cell mean, cell sums, streaming with wrapping
    return {"bytes": steps * (n * particle + cells * cell) + diags * cells * 40 + 48 * n, "flops": steps * n * flops}


# ---------------------------------------------------------------------------- an ensemble

def _ensemble_params(case, seed):
    # every size is there as often as any other, and the sweep's counts and activities are the
    # case's own, so that the work and the shapes do not depend on the seed
    rng = np.random.default_rng(7919 + case["replicas"])
    sides = (16, 24, 32, 40, 48)
    out = []
    for i in range(case["replicas"]):
        side = sides[i % len(sides)]
        n = side ** 3 * case["density"]
        cap = int(0.1 * side ** 3 / (4.0 / 3.0 * math.pi * 8.0))
        p = _params(side, n, int(min(rng.integers(5, 201), cap)), 2.0, case["density"], "fp32c", n_sub=10,
                    theta_deg=90.0, v0=float(rng.uniform(0, 0.1)), Dr=0.001, seed=1 + 1000 * seed + i)
        out.append(bg.make_params(**p))
    return out


def _prepare_ensemble(case, seed):
    ps = _ensemble_params(case, seed)
    ens = bg.Ensemble(ps)
    for s in ens:
        s.initialize(bg.INIT_PHYSICAL)
        s.setup()
    whole = _out(sum(p.n_fluid for p in ps), sum(p.n_colloid for p in ps))
    views, n0, c0 = [], 0, 0
    for p in ps:
        views.append({k: a[n0:n0 + p.n_fluid] if k in ("pos_fl", "vel_fl") else a[c0:c0 + p.n_colloid]
                      for k, a in whole.items()})
        n0, c0 = n0 + p.n_fluid, c0 + p.n_colloid
    return {"kind": "ensemble", "ens": ens, "steps": case["steps"], "whole": whole, "views": views}


def _run_ensemble(s):
    s["ens"].step(s["steps"])
    for sim, view in zip(s["ens"], s["views"]):
        sim.get_state(view)
    return s["whole"]


# ---------------------------------------------------------------------------- the closure

def _closure_data(rows, seed):
    """Features and exchanges like those of a run: a colloid's velocity, spin and orientation,
    its neighbours nearest first with the absent ones zero, and an exchange that follows the
    velocity with noise of its own size."""
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)

    mass = bg.displaced_mass(SUR_RADIUS, SUR_DENSITY)
    v, w, ra = 0.0547 * normal(rows, 3), 0.0432 * normal(rows, 3), torch.nn.functional.normalize(normal(rows, 3), dim=1)
    near = torch.cat([2.5 * normal(rows, 12, 3), 0.077 * normal(rows, 12, 3)], dim=2)
    present = torch.arange(12, device="cuda")[None, :] < torch.randint(0, 9, (rows, 1), generator=g, device="cuda")
    x = torch.cat([v, w, ra, (near * present[:, :, None]).reshape(rows, 72)], dim=1).contiguous()
    y = torch.cat([-SUR_DRAG * mass * v, -SUR_DRAG * 0.4 * mass * 4.0 * w], dim=1)
    y = (y + torch.tensor([5.8] * 3 + [7.3] * 3, device="cuda") * normal(rows, NY)).contiguous()
    return x, y


def _closure_weights(seed):
    """A flat parameter vector (W1, b1, ..., W4, b4) of scaled normal weights."""
    rng = np.random.default_rng(31 + seed)
    parts = []
    for k, n in LAYERS:
        parts += [rng.normal(0, 1.0 / math.sqrt(k), k * n), rng.normal(0, 0.05, n)]
    return np.concatenate(parts).astype(np.float32)


def _closure_norm():
    x_std = np.array([0.0547] * 3 + [0.0432] * 3 + [0.577] * 3 + ([2.5] * 3 + [0.077] * 3) * 12, np.float32)
    return np.zeros(IN, np.float32), x_std, np.zeros(NY, np.float32), np.array([5.8] * 3 + [7.3] * 3, np.float32)


def _network(rows, weights):
    net = closure.Network(max_batch=rows, seed=0)
    net.set_normalisation(*_closure_norm())
    net.set_params(weights)
    return net


def _prepare_train(case, seed):
    b, n = case["batch"], case["batches"]
    x, y = _closure_data(b * n, seed)
    torch.cuda.synchronize()
    weights = _closure_weights(seed)
    return {"kind": "train", "net": _network(b, weights), "weights": weights, "x": x, "y": y, "batch": b, "batches": n}


def _run_train(s):
    # a stretch of an epoch, the loss read after every batch as closure.train does; then the
    # gradient on the first batch and the weights, which a checkpoint keeps
    net, b = s["net"], s["batch"]
    losses = [net.train_step(s["x"][i * b:].data_ptr(), s["y"][i * b:].data_ptr(), b, 3e-4) for i in range(s["batches"])]
    loss, grad = net.grad(s["x"].data_ptr(), s["y"].data_ptr(), b)
    return {"losses": np.array(losses + [loss]), "grad": grad, "params": net.params()}


def _prepare_forward(case, seed):
    x, _ = _closure_data(case["rows"], seed)
    out = torch.empty((case["rows"], OUT), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return {"kind": "forward", "net": _network(case["rows"], _closure_weights(seed)), "x": x, "out": out,
            "rows": case["rows"]}


def _run_forward(s):
    s["net"].forward(s["x"].data_ptr(), s["out"].data_ptr(), s["rows"], torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _layers64(weights):
    out, o = [], 0
    w = torch.from_numpy(weights).cuda().double()
    for k, n in LAYERS:
        out += [w[o:o + k * n].reshape(k, n).clone(), w[o + k * n:o + k * n + n].clone()]
        o += k * n + n
    return [t.requires_grad_(True) for t in out]


def _net64(params, x):
    xm, xs, _, _ = (torch.from_numpy(a).cuda().double() for a in _closure_norm())
    a = ((x.double() - xm) / xs).clamp(-6, 6)
    for l in range(4):
        a = a @ params[2 * l] + params[2 * l + 1]
        if l < 3:
            a = torch.nn.functional.silu(a)
    return a


def _loss64(params, x, y):
    _, _, ym, ys = (torch.from_numpy(a).cuda().double() for a in _closure_norm())
    o = _net64(params, x)
    s = o[:, NY:].clamp(-6, 6)
    d = (y.double() - ym) / ys - o[:, :NY]
    return (0.5 * (d * d * torch.exp(-s) + s)).sum() / x.shape[0]


def _exact_train(case, seed):
    b = case["batch"]
    x, y = _closure_data(b * case["batches"], seed)
    params = _layers64(_closure_weights(seed))
    adam = torch.optim.Adam(params, lr=3e-4, betas=(0.9, 0.999), eps=1e-8)
    losses = []
    for i in range(case["batches"]):
        adam.zero_grad()
        loss = _loss64(params, x[i * b:(i + 1) * b], y[i * b:(i + 1) * b])
        loss.backward()
        adam.step()
        losses.append(loss.item())
    adam.zero_grad()
    loss = _loss64(params, x[:b], y[:b])
    loss.backward()
    return {"losses": np.array(losses + [loss.item()]),
            "grad": torch.cat([p.grad.reshape(-1) for p in params]).cpu().numpy(),
            "params": torch.cat([p.detach().reshape(-1) for p in params]).cpu().numpy()}


def _exact_forward(case, seed):
    x, _ = _closure_data(case["rows"], seed)
    _, _, ym, ys = (torch.from_numpy(a).cuda().double() for a in _closure_norm())
    with torch.no_grad():
        o = _net64(_layers64(_closure_weights(seed)), x)
    return torch.cat([o[:, :NY] * ys + ym, o[:, NY:].clamp(-6, 6) + 2 * torch.log(ys)], dim=1)


def _drag_weights(seed):
    """Weights of a network with the closure's behaviour: SiLU(z) - SiLU(-z) = z, so twelve hidden
    units carry the velocity and spin through the layers to a mean exchange that slows the
    colloid; the other units hold small normal weights, as a trained network's neighbour terms."""
    rng = np.random.default_rng(97 + seed)
    mats = [(rng.normal(0, 0.02 / math.sqrt(k), (k, n)), np.zeros(n)) for k, n in LAYERS]
    for l, (w, _) in enumerate(mats):
        if l < 3:
            w[:, :12] = 0.0
        for i in range(6):
            if l == 0:
                w[i, 2 * i], w[i, 2 * i + 1] = 1.0, -1.0
            elif l < 3:
                w[2 * i, 2 * i], w[2 * i + 1, 2 * i] = 1.0, -1.0
                w[2 * i, 2 * i + 1], w[2 * i + 1, 2 * i + 1] = -1.0, 1.0
            else:
                w[2 * i, i], w[2 * i + 1, i] = -0.158, 0.158
    return np.concatenate([np.concatenate([w.ravel(), b]) for w, b in mats]).astype(np.float32)


def _placed(L, n, gap, rng):
    """n sphere centres at least `gap` apart in a periodic box, by random sequential addition."""
    pos, k = np.empty((n, 3)), 0
    while k < n:
        for x in rng.uniform(0, L, (4 * n, 3)):
            d = pos[:k] - x
            d -= L * np.round(d / L)
            if k == 0 or np.min(np.einsum("ij,ij->i", d, d)) >= gap * gap:
                pos[k] = x
                k += 1
                if k == n:
                    break
    return pos


def _prepare_surrogate(case, seed):
    n = case["colloids"]
    L = max(12, int(round((n * 4.0 / 3.0 * math.pi * SUR_RADIUS ** 3 / case["fraction"]) ** (1.0 / 3.0))))
    rng = np.random.default_rng(53 + seed)
    p = _params(L, 1, n, SUR_RADIUS, SUR_DENSITY, "fp32c", n_sub=10, v0=0.05, theta_deg=90.0, Dr=0.001, seed=1 + seed)
    net = _network(max(n, 16), _drag_weights(seed))
    sur = closure.Surrogate(bg.make_params(**p), net)
    pos = _placed(float(L), n, 2 * SUR_RADIUS + 0.3, rng)
    ra = rng.normal(0, 1, (n, 3))
    sur.set_state(pos, rng.normal(0, 0.0547, (n, 3)), rng.normal(0, 0.0432, (n, 3)),
                  ra / np.linalg.norm(ra, axis=1, keepdims=True))
    return {"kind": "surrogate", "sur": sur, "net": net, "steps": case["steps"]}


def _run_surrogate(s):
    s["sur"].step(s["steps"])
    return s["sur"].get_state()


# ---------------------------------------------------------------------------- the cases' interface

_PREPARE = {"system": _prepare_system, "ensemble": _prepare_ensemble, "train": _prepare_train,
            "forward": _prepare_forward, "surrogate": _prepare_surrogate}
_RUN = {"system": _run_system, "ensemble": _run_ensemble, "train": _run_train, "forward": _run_forward,
        "surrogate": _run_surrogate}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    """64-bit values of the closure's training and inference.  The stepping cases have none: their
    draws are the framework's own."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "forward":
        return _exact_forward(case, seed)
    return None


def work(case):
    kind = case["kind"]
    n_params = sum(k * n + n for k, n in LAYERS)
    macs = sum(k * n for k, n in LAYERS)
    if kind == "system":
        cells = case["lx"] * case["ly"] * case["lz"]
        return _work_system(int(cells * case["density"]), cells, case["steps"], case["n_sub"], case["precision"],
                            case["steps"] if case["diag"] else 0)
    if kind == "ensemble":
        sides = [(16, 24, 32, 40, 48)[i % 5] for i in range(case["replicas"])]
        cells = sum(s ** 3 for s in sides)
        return _work_system(cells * case["density"], cells, case["steps"], 10, "fp32c")
    if kind == "train":
        b, n = case["batch"], case["batches"]
        # per batch: the rows in; weights and both moments read and written; forward and the two
        # backward products (none for the inputs' gradient); and the closing gradient
        flops = 2 * b * (3 * macs - IN * HID)
        return {"bytes": (n + 1) * b * (IN + NY) * 4 + n * 24 * n_params + 8 * n_params, "flops": (n + 1) * flops}
    if kind == "forward":
        return {"bytes": case["rows"] * (IN + OUT) * 4 + 4 * n_params, "flops": 2 * case["rows"] * macs}
    n, steps = case["colloids"], case["steps"]
    return {"bytes": steps * (n * 2 * 12 * 4 + 2 * n_params), "flops": steps * n * (2 * macs + 10 * 200)}
