"""Spheres that reach beyond the boxes around their cell, whose collisions the reference takes from the
342 boxes only: most of the particles inside them meet nothing.  The cooperative substeps against the
per-substep schedule, and no exact test for particles that the box rule leaves out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(form, radius, nc, L=48):
    import brownian_gb300 as bg
    M = bg.displaced_mass(radius, 10)
    sim = bg.Simulation(L, L ** 3 * 10, nc, n_sub=10, mass_colloid=M, sig_colloid=2 * radius, sigma=2 * radius,
                        I_colloid=0.4 * M * radius ** 2, v0=0.02, theta_deg=90.0, Dr=0.001, seed=3, init_gap=0.05,
                        precision=bg.FP64 if form == "fp64" else bg.FP32C)
    sim.initialize(bg.INIT_PHYSICAL)
    sim.setup()
    return sim


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
@pytest.mark.parametrize("radius,nc", [(4.0, 25), (6.0, 12)])
def test_bits_of_the_per_substep_schedule(form, radius, nc):
    a, b = _sim(form, radius, nc), _sim(form, radius, nc)
    b.set_flight(False)
    a.step(25)
    b.step(25)
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    assert a.diag()["events"] == b.diag()["events"] > 0
    a.close()
    b.close()


def test_particles_that_the_box_rule_leaves_out_are_not_listed():
    # (the FP32 form listed every particle inside such a sphere for the exact test, and its substeps took
    # longer than the FP64 form's, whose collisions cost several times as much)
    us = {}
    for form in ("fp64", "fp32c"):
        sim = _sim(form, 6.0, 12)
        sim.step(20)
        sim.profile(True)
        sim.step(5)
        n, ms = sim.profile_read()["k_stream_near"]
        us[form] = ms / n * 1e3
        sim.close()
    assert us["fp32c"] < us["fp64"], us
