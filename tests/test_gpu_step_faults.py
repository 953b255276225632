"""Failure detection of the cooperative substeps, provoked from the host: a launch that is refused
fails the step and every step after it until it is taken, runs nothing and leaves no captured
graph; the steps that follow give the bits of a run that never failed; and a device without room
for the kernel takes a launch per stage.  A wait that runs out (its limit set to a few polls) fails
the step, and with the state set again the steps give those bits too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(form, seed=11):
    import brownian_gb300 as bg
    M = bg.displaced_mass(2.0, 10)
    return bg.make_params(16, 16 ** 3 * 10, 8, n_sub=5, mass_colloid=M, sig_colloid=4.0, sigma=4.0,
                          I_colloid=0.4 * M * 4.0, v0=0.05, theta_deg=90.0, Dr=0.001, seed=seed,
                          precision=bg.FP64 if form == "fp64" else bg.FP32C, sort_every=4)


class One:
    """A single system with an ensemble's calls."""

    def __init__(self, form):
        import ctypes

        import brownian_gb300 as bg
        h = ctypes.c_void_p()
        p = _params(form)
        assert bg.lib().mpcd_create(ctypes.byref(p), ctypes.byref(h)) == 0
        self.sim = bg.Simulation._view(h.value, p)
        self.sim._owned = True
        self.step, self.set_flight, self.set_fault, self.close = (
            self.sim.step, self.sim.set_flight, self.sim.set_fault, self.sim.close)

    def __iter__(self):
        return iter([self.sim])


def _start(form):
    import brownian_gb300 as bg
    e = bg.Ensemble([_params("fp32c", s) for s in (11, 12)]) if form == "ensemble" else One(form)
    for s in e:
        s.initialize(bg.INIT_PHYSICAL)
        s.setup()
    return e


def _state(e):
    return [s.get_state() for s in e]


def _same(a, b):
    for x, y in zip(a, b):
        for k in x:
            assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("form", ["fp64", "fp32c", "ensemble"])
def test_a_refused_launch_fails_every_step_until_it_is_taken(form):
    import brownian_gb300 as bg
    a, b = _start(form), _start(form)
    a.step(2)
    b.step(2)
    before = _state(a)
    a.set_fault(bg.FAULT_LAUNCH, 1)
    for n in (1, 1, 3, 5):
        with pytest.raises(bg.MPCDError) as err:
            a.step(n)
        assert err.value.code == bg.ERR_CUDA and "refused" in str(err.value)
    _same(_state(a), before)
    assert [s.step_count for s in a] == [2] * len(before)
    a.set_fault(bg.FAULT_LAUNCH, 0)
    a.step(7)
    b.step(7)
    _same(_state(a), _state(b))
    a.close()
    b.close()


@pytest.mark.parametrize("form", ["fp64", "fp32c", "ensemble"])
def test_another_schedule_goes_on_after_a_refused_launch(form):
    # (the set-up's cell table is still there: it is not built again)
    import brownian_gb300 as bg
    a, b = _start(form), _start(form)
    a.set_fault(bg.FAULT_LAUNCH, 1)
    with pytest.raises(bg.MPCDError):
        a.step(2)
    for e in (a, b):
        e.set_flight(False)
        e.step(3)
    _same(_state(a), _state(b))
    a.close()
    b.close()


@pytest.mark.parametrize("form", ["fp64", "fp32c", "ensemble"])
def test_a_device_without_room_takes_a_launch_per_stage(form):
    import brownian_gb300 as bg
    a, b = _start(form), _start(form)
    a.set_fault(bg.FAULT_LAUNCH, 1)  # (the cooperative kernel is not launched)
    for room, k in ((1, 6), (0, 3), (1, 2)):
        a.set_fault(bg.FAULT_ROOM, room)
        a.set_fault(bg.FAULT_LAUNCH, room)
        a.step(k)
        b.step(k)
        _same(_state(a), _state(b))
    a.close()
    b.close()


@pytest.mark.parametrize("form", ["fp64", "fp32c", "ensemble"])
@pytest.mark.parametrize("what", ["WAIT", "ORIENT"])
def test_a_wait_that_runs_out_is_reported(form, what):
    import brownian_gb300 as bg
    keys = ("pos_fl", "vel_fl", "pos_colloid", "vel_colloid", "ang_vel_colloid", "ra")
    a, b = _start(form), _start(form)
    first = _state(a)
    fault = getattr(bg, "FAULT_" + what)
    for polls, steps in ((0, 1), (0, 4)) + (((1, 2),) if what == "WAIT" else ()):
        a.set_fault(fault, polls)
        with pytest.raises(bg.MPCDError) as err:
            a.step(steps)
        assert err.value.code == bg.ERR_CUDA and "did not end within its limit" in str(err.value)
        if form != "ensemble":
            with pytest.raises(bg.MPCDError) as err:
                a.sim.diag()
            assert err.value.code == bg.ERR_CUDA
        a.set_fault(fault, -1)
        for s, x in zip(a, first):
            s.step_count = 0
            s.set_state(*[x[k] for k in keys])
            s.setup()
    a.step(5)
    b.step(5)
    _same(_state(a), _state(b))
    a.close()
    b.close()


def test_a_refused_launch_fails_a_traced_and_a_profiled_step():
    import brownian_gb300 as bg
    e = _start("fp64")
    sim = e.sim
    sim.set_fault(bg.FAULT_LAUNCH, 1)
    with pytest.raises(bg.MPCDError):
        sim.trace_step()
    assert sim.step_count == 0
    sim.profile(True)
    with pytest.raises(bg.MPCDError):
        sim.step(1)
    sim.profile(False)
    e.close()
