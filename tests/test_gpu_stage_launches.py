"""The schedules that launch a kernel per stage of a substep (every particle in every pass; the
free-flight schedule on a device without room for the cooperative kernel), whose launch shapes a
step on that kernel does not use: the same bits at any shape.  And the ways in which steps are
grouped: several to a graph, an ensemble in several cooperative launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(form, L=16, nc=8, seed=11, **kw):
    import brownian_gb300 as bg
    M = bg.displaced_mass(2.0, 10)
    p = dict(n_sub=10, v0=0.05, theta_deg=90.0, Dr=0.001, sort_every=3)
    p.update(kw)
    return dict(L=L, n_fluid=L ** 3 * 10, n_colloid=nc, mass_colloid=M, sig_colloid=4.0, sigma=4.0, I_colloid=0.4 * M * 4.0,
                seed=seed, precision=bg.FP64 if form == "fp64" else bg.FP32C, **p)


def _sim(form, **kw):
    import brownian_gb300 as bg
    sim = bg.Simulation(**_params(form, **kw))
    sim.initialize(bg.INIT_PHYSICAL)
    sim.setup()
    return sim


def _ens(systems):
    import brownian_gb300 as bg
    e = bg.Ensemble([bg.make_params(**p) for p in systems])
    for s in e:
        s.initialize(bg.INIT_PHYSICAL)
        s.setup()
    return e


def _same(a, b):
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("schedule", ["every_particle", "free_flight"])
@pytest.mark.parametrize("form", ["fp64", "fp32c"])
def test_launch_shapes_of_the_stages_leave_the_same_bits(form, schedule):
    import brownian_gb300 as bg
    a, b = _sim(form), _sim(form)
    if schedule == "every_particle":
        b.set_flight(False)
    else:
        b.set_fault(bg.FAULT_ROOM, 1)
    for events, fin, aux, free in (((40, 64), (20, 64), (1, 256), (100, 3)), ((300, 32), (3, 128), (1, 64), (700, 0)),
                                   ((1, 128), (200, 32), (1, 128), (1, 9))):
        b.set_launch(bg.LAUNCH_EVENTS, *events)
        b.set_launch(bg.LAUNCH_FIN, *fin)
        b.set_launch(bg.LAUNCH_AUX, *aux)
        b.set_launch(bg.LAUNCH_FREE, *free)
        a.step(2)
        b.step(2)
        _same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("schedule", ["every_particle", "free_flight"])
def test_launch_shapes_of_an_ensembles_stages_leave_the_same_bits(schedule):
    import brownian_gb300 as bg
    systems = [_params("fp32c", L=L, nc=nc, seed=i) for i, (L, nc) in enumerate([(16, 8), (12, 2), (20, 16)])]
    a, b = _ens(systems), _ens(systems)
    if schedule == "every_particle":
        b.set_flight(False)
    else:
        b.set_fault(bg.FAULT_ROOM, 1)
    for events, run, fin, aux, free in ((1, 1, 32, 64, 1), (7, 9, 64, 256, 8), (64, 64, 128, 128, 3)):
        b.set_launch(bg.ENS_EVENTS, events)
        b.set_launch(bg.ENS_RUN, run)
        b.set_launch(bg.ENS_FIN, 1, fin)
        b.set_launch(bg.ENS_AUX, 1, aux)
        b.set_launch(bg.ENS_FREE, free)
        a.step(2)
        b.step(2)
        for x, y in zip(a, b):
            _same(x, y)
    a.close()
    b.close()


def test_an_ensemble_says_whether_its_substeps_are_one_kernel():
    import brownian_gb300 as bg
    e = _ens([_params("fp32c", L=12, nc=2)])
    assert e.one_kernel
    e.set_flight(False)
    assert not e.one_kernel
    e.set_flight(True)
    e.set_fault(bg.FAULT_ROOM, 1)
    assert not e.one_kernel
    e.close()


@pytest.mark.parametrize("sort_every", [-1, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("form", ["fp64", "fp32c"])
def test_steps_of_one_call_are_those_of_many(form, sort_every):
    # (three steps that do not sort are one graph; the counting sort comes between them or in their place)
    a, b = _sim(form, L=12, nc=3, sort_every=sort_every), _sim(form, L=12, nc=3, sort_every=sort_every)
    for n in (11, 3, 4, 1, 7):
        a.step(n)
        for _ in range(n):
            b.step(1)
        _same(a, b)
        assert a.step_count == b.step_count
    assert a.diag() == b.diag()
    a.close()
    b.close()


def test_an_ensemble_with_more_active_particles_than_the_blocks_hold():
    # eight systems with 660 spheres each: about 61,000 expected active particles a system where a launch of
    # 152 blocks has room for 408,000
    systems = [_params("fp32c", L=48, nc=660, seed=i, n_sub=4, init_gap=0.1, sort_every=-1) for i in range(8)]
    a, b, one = _ens(systems), _ens(systems), _ens(systems[:1])
    b.set_flight(False)
    counts = []
    for e in (one, a):
        before = e.launch_count
        e.step(1)
        counts.append(e.launch_count - before)
    assert counts[1] == counts[0] + 1  # a second cooperative launch
    a.step(2)
    b.step(3)
    for x, y in zip(a, b):
        _same(x, y)
    for e in (a, b, one):
        e.close()
