"""The free-flight pass on the states its short forms are made of: positions on and beside the edges
of binades, cells and the box, moves of half an ulp and of none, offsets that round up to 1, moves of
half a cell and more, and more substeps than the FP64 jump takes.  One particle to an SRD cell keeps
its velocity through the collision, so the positions are those of the additions one by one, in numpy
and in the per-substep schedule, bit for bit; and the FP32 form's cell sums from pairs of particles
whose mean and thermostat factor are known."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L, COLUMNS = 64, 32
F = np.float32


def _sim(form, n_sub, dt, N, **kw):
    import brownian_gb300 as bg
    # (one small colloid between the columns, which none of the particles meets)
    return bg.Simulation(L, N, 1, n_sub=n_sub, ndt=n_sub * dt, mass_colloid=1e3, sig_colloid=0.8, sigma=0.8,
                         I_colloid=1e2, theta_deg=90.0, seed=3, max_per_cell=64,
                         precision=bg.FP64 if form == "fp64" else bg.FP32C, **kw)


def _run(form, axis, x, v, n_sub, dt, steps, flight):
    """Positions along `axis` of particles with x and v there, each in a column of its own, after every step."""
    N = len(x)
    sim = _sim(form, n_sub, dt, N, vmax=8192.0)
    pos, vel = np.empty((N, 3)), np.zeros((N, 3))
    col = np.arange(N)
    pos[:, axis], vel[:, axis] = x, v
    pos[:, (axis + 1) % 3] = 2.0 * (col % COLUMNS) + 1.0
    pos[:, (axis + 2) % 3] = 2.0 * (col // COLUMNS) + 1.0
    sim.set_state(pos, vel, np.full((1, 3), 4.0), np.zeros((1, 3)), np.zeros((1, 3)), np.array([[1.0, 0.0, 0.0]]))
    sim.set_flight(flight)
    sim.setup()
    out = []
    for _ in range(steps):
        sim.step(1)
        out.append(sim.get_state()["pos_fl"][:, axis])
    sim.close()
    return out


def _mod(x):
    q = (x - L * 0.5) / L
    t = np.trunc(q)
    t = np.where(np.abs(q - t) >= 0.5, t + np.sign(q), t)  # lround
    return x - L * t


def _moves64(kind, scale):
    rng = np.random.default_rng(len(kind))
    n = COLUMNS ** 2
    if kind == "edges":
        edge = 2.0 ** rng.integers(-32, 7, n)
        beside = [edge, np.nextafter(edge, 0), np.nextafter(edge, 2 * L), np.maximum(edge - scale, 1e-3), np.full(n, L)]
        x = np.minimum(np.choose(rng.integers(0, 5, n), beside), L)
        w = rng.choice([scale, -scale, scale / 16, -scale / 16, 1e-16, -1e-16, 0.0, 5e-324], n)
        return x, w
    x = rng.uniform(0.001, L, n)
    m = rng.integers(-9, 10, n) + rng.choice([0.0, 2.0 ** 20, 2.0 ** 35], n)
    return x, m * np.spacing(x) * rng.choice([0.5, 0.25], n)


@pytest.mark.parametrize("kind", ["edges", "ties"])
@pytest.mark.parametrize("n_sub,dt,scale,axis", [(10, 2.0 ** -6, 0.02, 0), (10, 2.0 ** -6, 0.02, 1), (10, 2.0 ** -6, 0.02, 2),
                                                 (1024, 2.0 ** -13, 2e-4, 0), (1025, 2.0 ** -13, 2e-4, 1)])
def test_fp64_positions_are_the_additions(kind, n_sub, dt, scale, axis):
    x, w = _moves64(kind, scale)
    steps = 5 if n_sub == 10 else 1
    got = _run("fp64", axis, x, w / dt, n_sub, dt, steps, True)
    per_substep = _run("fp64", axis, x, w / dt, n_sub, dt, steps, False)
    ref = x
    for k in range(steps):
        for _ in range(n_sub):
            ref = _mod(ref + w)
        assert np.array_equal(got[k], ref), k
        assert np.array_equal(per_substep[k], ref), k


def _moves32(dt):
    rng = np.random.default_rng(4)
    n = COLUMNS ** 2
    ulp = 2.0 ** -24
    o = rng.choice([0.0, 1 - ulp, 2.0 ** -149, 2.0 ** -30, ulp, 0.5, 0.25, 1 - 2 * ulp], n).astype(F)
    o = np.where(rng.random(n) < 0.3, rng.uniform(0, 1, n).astype(F), o)
    cell = np.where(o < 2.0 ** -40, 0, rng.choice([0, 1, 31, 62, 63], n))  # (c + o is exact in FP64)
    step = rng.choice([0.0, ulp, -ulp, 0.5 * ulp, -0.5 * ulp, -2.0 ** -30, 2.0 ** -30, 100 * ulp, -100 * ulp, 0.01, -0.01,
                       0.4999, -0.4999], n)
    return cell, o, (step / dt).astype(F)


@pytest.mark.parametrize("n_sub,dt,axis", [(10, 2.0 ** -6, 0), (10, 2.0 ** -6, 1), (37, 2.0 ** -6, 2), (10, 2.0 ** -2, 0),
                                           (10, 2.0 ** -2, 2), (1025, 2.0 ** -13, 1)])
def test_fp32_positions_are_the_additions(n_sub, dt, axis):
    # (0.25 time units a substep: a thermal particle's moves reach half a cell)
    cell, o, v = _moves32(dt)
    steps = 3 if n_sub < 100 else 1
    x = cell + o.astype(np.float64)
    got = _run("fp32c", axis, x, v, n_sub, dt, steps, True)
    per_substep = _run("fp32c", axis, x, v, n_sub, dt, steps, False)
    w = v.astype(np.longdouble) * np.longdouble(dt)  # exact
    for k in range(steps):
        for _ in range(n_sub):
            o = (o.astype(np.longdouble) + w).astype(F)
            f = np.floor(o)
            o = (o - f).astype(F)
            cell = cell + f.astype(int)
            up = o >= 1
            o, cell = np.where(up, F(0), o), (cell + up) % L
        ref = cell + o.astype(np.float64)
        assert np.array_equal(got[k], ref), k
        assert np.array_equal(per_substep[k], ref), k


@pytest.mark.parametrize("offset", [0.0, 8.0])
def test_fp32_cell_sums_of_pairs(offset):
    # Two particles of a cell with velocities c + a and c - a leave the collision with mean c and
    # sum |v - c|^2 = 3 kT / m.  The sums' unit is 2^-44 here: 2^-17 of the smallest pairs' sum of squares;
    # the FP32 map's rounding is a few 2^-24 of |v| times the factor, at most 2e-5 of a thermal speed.
    rng = np.random.default_rng(9)
    n = COLUMNS ** 2 // 2
    lo = -2 if offset else -14
    a = rng.choice([-1.0, 1.0], (n, 3)) * 2.0 ** rng.uniform(lo, 3.5, (n, 1)) * rng.uniform(0.6, 1.0, (n, 3))
    a = a.astype(F).astype(np.float64)
    c = offset * rng.choice([-1.0, 1.0], (n, 3))
    col = np.arange(n)
    pos = np.repeat(np.stack([2.0 * (col % COLUMNS) + 1.3, 2.0 * (col // COLUMNS) + 1.3, np.full(n, 33.3)], 1), 2, 0)
    vel = np.empty((2 * n, 3))
    vel[0::2], vel[1::2] = c + a, c - a
    vel = vel.astype(F).astype(np.float64)
    sim = _sim("fp32c", 10, 2.0 ** -10, 2 * n)
    sim.set_state(pos, vel, np.full((1, 3), 4.0), np.zeros((1, 3)), np.zeros((1, 3)), np.array([[1.0, 0.0, 0.0]]))
    sim.setup()
    sim.step(1)
    v = sim.get_state()["vel_fl"].reshape(n, 2, 3)
    mean = v.mean(1)
    want = vel.reshape(n, 2, 3).mean(1)
    assert np.abs(mean - want).max() <= 5e-5
    d = v - mean[:, None]
    assert np.abs((d * d).sum((1, 2)) / 3.0 - 1.0).max() <= 2e-4
    sim.close()
