"""Which systems take the cooperative substeps: in the FP64 form not those whose active particles are far
more than its blocks hold in shared memory.  Both sides of the rule against the per-substep schedule,
and below it a system whose blocks hold more than their shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(form, nc, density=60, L=48):
    import brownian_gb300 as bg
    M = bg.displaced_mass(2.0, density)
    sim = bg.Simulation(L, L ** 3 * density, nc, n_sub=10, mass_colloid=M, sig_colloid=4.0, sigma=4.0,
                        I_colloid=0.4 * M * 4.0, v0=0.02, theta_deg=90.0, Dr=0.001, seed=5, max_per_cell=256,
                        init_gap=0.05, precision=bg.FP64 if form == "fp64" else bg.FP32C)
    sim.initialize(bg.INIT_PHYSICAL)
    sim.setup()
    return sim


# (about 256 expected active particles a sphere: 1,126 a block are the limit, 1,024 its shared memory)
@pytest.mark.parametrize("form,nc,one_kernel", [("fp64", 440, True), ("fp64", 600, False), ("fp32c", 600, True)])
def test_the_rule_by_active_particles(form, nc, one_kernel):
    a, b = _sim(form, nc), _sim(form, nc)
    b.set_flight(False)
    a.step(2)
    b.step(2)
    a.profile(True)
    a.step(1)
    kernels = set(a.profile_read())
    a.profile(False)
    b.step(1)
    assert ("k_rotdiff_step" in kernels) == one_kernel and ("k_stream_near_last" in kernels) != one_kernel, kernels
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()
