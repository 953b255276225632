"""A free-flight step's substeps in one cooperative kernel against the same steps launched
substep by substep (set_flight(False), whose parity with the oracle other tests check): the same
bits, the same wall-collision count, at the edges of what the kernel takes: two substeps, one
colloid, spheres whose reach passes the +-3 box rule, crowded cells, touching pairs, the corrected
rules, fast particles, and more active and pending particles than a block keeps in shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {
    "two_substeps": dict(n_sub=2, ndt=0.05),
    "one_colloid_odd_box": dict(L=(7, 8, 9), nc=1, density=15),
    "reach_beyond_the_box_rule": dict(L=(28, 27, 26), nc=10, radius=3.2, theta_deg=130.0),
    "crowded_cells": dict(L=(14, 13, 12), nc=80, radius=0.75, density=20, init_gap=0.02),
    "corrected_rules_small_spheres": dict(L=(12, 12, 12), nc=60, radius=0.5, density=20, physics=1),
    "strong_kick": dict(nc=10, v0=0.3, vmax=400.0),
    "shared_memory_overflows_fp64": dict(L=(48, 48, 48), nc=600, density=60, max_per_cell=256, steps=2, only="fp64"),
    "shared_memory_overflows_fp32c": dict(L=(48, 48, 48), nc=600, density=120, max_per_cell=512, steps=2, only="fp32c"),
}


def _sim(form, *, L=(20, 20, 20), nc=20, radius=2.0, density=10, steps=6, only=None, **kw):
    import brownian_gb300 as bg
    M = bg.displaced_mass(radius, density)
    p = dict(n_sub=10, v0=0.05, theta_deg=90.0, Dr=0.001, init_gap=0.3)
    p.update(kw)
    sim = bg.Simulation(L, int(np.prod(L) * density), nc, mass_colloid=M, sig_colloid=2 * radius, sigma=2 * radius,
                        I_colloid=0.4 * M * radius ** 2, seed=5,
                        precision=bg.FP64 if form == "fp64" else bg.FP32C, **p)
    sim.initialize(bg.INIT_PHYSICAL)
    sim.setup()
    return sim, steps


@pytest.mark.parametrize("form", ["fp64", "fp32c"])
@pytest.mark.parametrize("name", FORMS)
def test_one_kernel_substeps_give_the_same_bits(name, form):
    kw = FORMS[name]
    if kw.get("only", form) != form:
        pytest.skip("the other form's size")
    a, steps = _sim(form, **kw)
    b, _ = _sim(form, **kw)
    b.set_flight(False)
    a.step(steps)
    b.step(steps)
    sa, sb = a.get_state(), b.get_state()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
    da, db = a.diag(), b.diag()
    assert da["events"] == db["events"] > 0 and da["shell_records"] == db["shell_records"]
    assert np.array_equal(a.rotation_binning()[0], b.rotation_binning()[0])
    a.close()
    b.close()
