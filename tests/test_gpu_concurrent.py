"""Contexts and ensembles that step at the same time on one GPU, from their own streams and from their
own threads, give the bits that they give alone (each's cooperative kernel takes a block of every SM)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kw(form, L, nc, seed):
    import brownian_gb300 as bg
    M = bg.displaced_mass(2.0, 10)
    return dict(L=L, n_fluid=L ** 3 * 10, n_colloid=nc, n_sub=10, mass_colloid=M, sig_colloid=4.0, sigma=4.0,
                I_colloid=0.4 * M * 4.0, v0=0.05, theta_deg=90.0, Dr=0.001, seed=seed,
                precision=bg.FP64 if form == "fp64" else bg.FP32C)


SYSTEMS = [("fp64", 16, 8, 1), ("fp32c", 24, 30, 2), ("fp64", 24, 20, 3), ("fp32c", 14, 4, 4)]


def _sims():
    import brownian_gb300 as bg
    sims = [bg.Simulation(**_kw(*s)) for s in SYSTEMS]
    for s in sims:
        s.initialize(bg.INIT_PHYSICAL)
        s.setup()
    return sims


def _ens():
    import brownian_gb300 as bg
    e = bg.Ensemble([bg.make_params(**_kw("fp32c", L, nc, 9 + L)) for L, nc in ((16, 6), (20, 10), (12, 1))])
    for s in e:
        s.initialize(bg.INIT_PHYSICAL)
        s.setup()
    return e


def _same(a, b):
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k


def _alone():
    sims, e = _sims(), _ens()
    for s in sims:
        s.step(30)
    e.step(30)
    return sims, e


def test_steps_in_flight_on_several_streams():
    ref, ens = _alone()
    sims = _sims()
    for _ in range(3):
        for s in sims:
            s.step_async(10)
    for a, s in zip(ref, sims):
        s.sync()
        _same(a, s)
    for s in ref + sims:
        s.close()
    ens.close()


def test_steps_from_several_threads():
    ref, ref_e = _alone()
    sims, e = _sims(), _ens()
    failed = []

    def run(x):
        try:
            for _ in range(6):
                x.step(5)
        except Exception as err:
            failed.append(err)

    threads = [threading.Thread(target=run, args=(x,)) for x in [*sims, e]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for a, s in zip([*ref, *ref_e], [*sims, *e]):
        _same(a, s)
    for s in ref + sims:
        s.close()
    e.close()
    ref_e.close()
