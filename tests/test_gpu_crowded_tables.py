"""Cells that list more colloids than a cell table holds (16) in a step's flight table, whose reach
is longer: the free-flight step then builds the cell tables for their capacity check.  A run that
goes from it to a schedule that reads them goes on with the bits of one that never left that
schedule, and a table that overflows is refused in the same step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("pos_fl", "vel_fl", "pos_colloid", "vel_colloid", "ang_vel_colloid", "ra")


def _outside(X):
    """Uniform positions in the 32^3 box outside the spheres."""
    pos = np.random.default_rng(1).uniform(0.01, 31.99, (200_000, 3))
    free = np.ones(len(pos), bool)
    for x in X:
        d = pos - x
        d -= 32 * np.round(d / 32)
        free &= (d * d).sum(1) > 9.2
    return pos[free][:90_000]


def _crowd(form, as_params=False):
    """32^3 cells, 41 spheres of radius 3 (free to overlap) in a cube of side 10.33: up to 14 colloids in
    a cell table, 23 in a flight cell, and no particle in the run() shells of more than 6."""
    import brownian_gb300 as bg
    rng = np.random.default_rng(206)
    n, side = rng.integers(20, 60), rng.uniform(8, 14)
    X = 16 - side / 2 + rng.uniform(0, side, (n, 3))
    rng = np.random.default_rng(1)
    M = bg.displaced_mass(3.0, 10)
    pos = _outside(X)
    ra = rng.normal(0, 1, (n, 3))
    state = dict(pos_fl=pos, vel_fl=rng.normal(0, 1, pos.shape), pos_colloid=X,
                 vel_colloid=rng.normal(0, M ** -0.5, (n, 3)), ang_vel_colloid=np.zeros((n, 3)),
                 ra=ra / np.linalg.norm(ra, axis=1, keepdims=True))
    kw = dict(n_sub=10, mass_colloid=M, sig_colloid=0.01, sigma=6.0, I_colloid=0.4 * M * 9.0, v0=0.0, theta_deg=90.0,
              Dr=0.001, seed=3, precision=bg.FP64 if form == "fp64" else bg.FP32C)
    p = bg.make_params(32, len(pos), int(n), **kw)
    return (p, state) if as_params else (_start(bg.Simulation(32, len(pos), int(n), **kw), state), state)


def _start(sim, state):
    sim.set_state(*[state[k] for k in STATE])
    sim.setup()
    return sim


def _same(a, b):
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k


def _by_routine(sim, form):
    sim.rotation_mpcd()
    sim.run()
    for l in range(1, 11):
        sim.substep_routines() if form == "fp64" else sim.substep(l)


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
def test_a_schedule_that_reads_the_tables_goes_on_from_a_crowded_step(form):
    a, _ = _crowd(form)
    b, _ = _crowd(form)
    b.set_flight(False)
    for flight, k in ((True, 1), (False, 2), (True, 3), (False, 1)):
        a.set_flight(flight)
        a.step(k)
        b.step(k)
        _same(a, b)
    a.set_flight(True)
    for _ in range(2):
        a.step(1)
        b.step(1)
        _by_routine(a, form)
        _by_routine(b, form)
        _same(a, b)
    a.close()
    b.close()


def test_an_ensemble_goes_on_from_a_crowded_step():
    import brownian_gb300 as bg
    p, state = _crowd("fp32c", as_params=True)
    a, b = bg.Ensemble([p, p]), bg.Ensemble([p, p])
    b.set_flight(False)
    for e in (a, b):
        for s in e:
            _start(s, state)
    for flight, k in ((True, 2), (False, 1), (True, 1), (False, 2)):
        a.set_flight(flight)
        a.step(k)
        b.step(k)
        for x, y in zip(a, b):
            _same(x, y)
    a.close()
    b.close()


def test_another_state_at_the_step_after_a_crowded_one():
    # the mark of the crowded step does not outlive the state that it was made for
    a, state = _crowd("fp64")
    a.step(6)
    spread = dict(state)
    grid = np.stack(np.meshgrid(*[np.arange(4) * 8.0 + 4.3] * 3), -1).reshape(-1, 3)
    spread["pos_colloid"] = grid[:len(state["pos_colloid"])]
    spread["pos_fl"] = _outside(spread["pos_colloid"])
    b, _ = _crowd("fp64")
    b.set_flight(False)
    for s in (a, b):
        s.step_count = 5
        _start(s, spread)
        s.step(1)
    a.set_flight(False)
    for s in (a, b):
        s.step(2)
    _same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
@pytest.mark.parametrize("n_sub", [2, 3, 10])
def test_a_table_that_overflows_is_refused_in_the_same_step(form, n_sub):
    # 16 spheres around one point and one that comes within reach of a cell of the last substep's table
    # (whose reach is the run() shell's), never of the others'
    import brownian_gb300 as bg
    rng = np.random.default_rng(7)
    M = 200.0
    X = np.concatenate([10.5 + rng.uniform(-0.02, 0.02, (16, 3)), [[14.75, 10.5, 10.5]]])
    V = np.zeros((17, 3))
    V[16, 0] = -0.15
    pos = rng.uniform(0, 1, (2000, 3)) * [4.0, 23.9, 23.9] + [18.5, 0.05, 0.05]
    state = dict(pos_fl=pos, vel_fl=0.5 * rng.normal(0, 1, pos.shape), pos_colloid=X, vel_colloid=V,
                 ang_vel_colloid=np.zeros((17, 3)), ra=np.tile([1.0, 0.0, 0.0], (17, 1)))
    refused = []
    for flight in (True, False):
        sim = bg.Simulation(24, 2000, 17, n_sub=n_sub, mass_colloid=M, sig_colloid=0.001, sigma=2.0, I_colloid=80.0,
                            theta_deg=90.0, seed=3, precision=bg.FP64 if form == "fp64" else bg.FP32C)
        sim.set_flight(flight)
        _start(sim, state)
        for k in range(12):
            try:
                sim.step(1)
            except bg.MPCDError as e:
                assert e.code == bg.ERR_CAPACITY and "table" in str(e)
                refused.append(k)
                break
        sim.close()
    assert len(refused) == 2 and refused[0] == refused[1] > 0, refused


def _cluster(form, nc=300, side=12.0, L=48):
    """Small spheres on a jittered lattice in a corner of the box: seventeen expected within a flight cell's
    reach, one to five in a cell table."""
    import brownian_gb300 as bg
    rng = np.random.default_rng(2)
    m = int(np.ceil(nc ** (1 / 3)))
    a = side / m
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(m ** 3)[:nc]]
    X = 3 + (g + 0.5) * a + rng.uniform(-0.1, 0.1, (nc, 3)) * (a - 1.0)
    M = 50.0
    pos = rng.uniform(0.01, L - 0.01, (L ** 3 * 6, 3))
    near = (pos < side + 6).all(1)
    free = np.ones(len(pos), bool)
    free[near] = np.array([((X - p) ** 2).sum(1).min() > 0.26 for p in pos[near]])
    pos = pos[free]
    ra = rng.normal(0, 1, (nc, 3))
    state = dict(pos_fl=pos, vel_fl=rng.normal(0, 1, pos.shape), pos_colloid=X,
                 vel_colloid=rng.normal(0, M ** -0.5, (nc, 3)), ang_vel_colloid=np.zeros((nc, 3)),
                 ra=ra / np.linalg.norm(ra, axis=1, keepdims=True))
    sim = bg.Simulation(L, len(pos), nc, n_sub=10, mass_colloid=M, sig_colloid=0.9, sigma=1.0, I_colloid=5.0, v0=0.02,
                        theta_deg=90.0, Dr=0.001, seed=3, precision=bg.FP64 if form == "fp64" else bg.FP32C)
    return _start(sim, state)


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
def test_a_cluster_of_small_spheres_is_no_scan_of_all_spheres(form):
    # (the particles of its cells, which list more spheres than a flight cell holds, once scanned all 300 in
    # every substep: ten times the per-substep schedule's time)
    import time
    a, b = _cluster(form), _cluster(form)
    b.set_flight(False)
    took = []
    for s in (a, b):
        s.step(6)
        t = time.perf_counter()
        s.step(20)
        took.append(time.perf_counter() - t)
    _same(a, b)
    da, db = a.diag(), b.diag()
    assert da["events"] == db["events"] > 0 and da["shell_records"] == db["shell_records"] > 0
    assert took[0] < 2.0 * took[1], took
    a.close()
    b.close()
