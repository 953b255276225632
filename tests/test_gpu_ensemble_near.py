"""The batched ensemble's substeps in one cooperative kernel, every system on blocks of its own,
against the batched per-substep schedule (whose systems' parity other tests check): the same bits
where systems share the SMs unevenly, have no colloids, need more than one launch, or include one
too crowded for it (the whole ensemble then takes a launch per stage)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (box, colloids, radius, Dr) of the systems
FORMS = {
    "uneven": [(10, 1, 2.0, 0.001), (24, 30, 2.0, 0.0), (12, 0, 2.0, 0.001), (11, 4, 1.5, 0.001)],
    "one_system": [(16, 5, 2.0, 0.001)],
    "two_launches": [(10, i % 3, 2.0, 0.001) for i in range(160)],
    "a_crowded_system": [(10, 3, 2.0, 0.001), (8, 40, 0.75, 0.001)],
}


def _params(i, L, nc, radius, Dr):
    import brownian_gb300 as bg
    M = bg.displaced_mass(radius, 10)
    return bg.make_params(L, L ** 3 * 10, nc, n_sub=6, mass_colloid=M, sig_colloid=2 * radius, sigma=2 * radius,
                          I_colloid=0.4 * M * radius ** 2, v0=0.05, theta_deg=90.0, Dr=Dr, seed=300 + i,
                          precision=bg.FP32C, sort_every=2, init_gap=0.05)


@pytest.mark.parametrize("name", FORMS)
def test_one_kernel_substeps_of_every_system_give_the_same_bits(name):
    import brownian_gb300 as bg
    params = [_params(i, *s) for i, s in enumerate(FORMS[name])]
    a, b = bg.Ensemble(params), bg.Ensemble(params)
    b.set_flight(False)
    for e in (a, b):
        for s in e:
            s.initialize(bg.INIT_PHYSICAL)
            s.setup()
    for on, k in ((True, 3), (False, 1), (True, 2)):
        a.set_flight(on)
        a.step(k)
        b.step(k)
        for r, (x, y) in enumerate(zip(a, b)):
            gx, gy = x.get_state(), y.get_state()
            for key in gx:
                assert np.array_equal(gx[key], gy[key]), (on, r, key)
    assert [s.diag()["events"] for s in a] == [s.diag()["events"] for s in b]
    # a system stepped alone goes on from there
    a[0].step(2)
    b[0].set_flight(False)
    b[0].step(2)
    assert np.array_equal(a[0].get_state()["pos_fl"], b[0].get_state()["pos_fl"])
    a.close()
    b.close()
