"""A sphere that moves several cells in a substep: the step is refused, and the steps enqueued behind it
in the same call do not take that move for the reach of their tables (every particle would be near)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ("fp64", "fp32c"))
def test_steps_behind_a_refused_one_keep_their_reach(form):
    import brownian_gb300 as bg
    M = bg.displaced_mass(2.0, 10)
    kw = dict(n_sub=10, mass_colloid=M, sig_colloid=4.0, sigma=4.0, I_colloid=0.4 * M * 4.0, v0=0.0, theta_deg=90.0,
              Dr=0.0, seed=9, precision=bg.FP64 if form == "fp64" else bg.FP32C)
    a, b = (bg.Simulation(48, 48 ** 3 * 10, 4, **kw) for _ in range(2))
    for s in (a, b):
        s.initialize(bg.INIT_PHYSICAL)
    st = a.get_state()
    v = st["vel_colloid"].copy()
    v[0] = (500.0, 0.0, 0.0)
    keys = ("pos_fl", "vel_fl", "pos_colloid", "vel_colloid", "ang_vel_colloid", "ra")
    a.set_state(*[v if k == "vel_colloid" else st[k] for k in keys])
    a.setup()
    with pytest.raises(bg.MPCDError) as e:
        a.step(3)
    assert e.value.code in (3, 4)
    assert 0 < a.flight_near() < 48 ** 3 * 10 // 2
    # from the state before it, the bits of a simulation that took other steps there
    b.setup()
    b.step(3)
    for s in (a, b):
        s.set_state(*[st[k] for k in keys])
        s.setup()
        s.step(3)
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()
