"""Boxes that the free-flight step's reach spans: a sphere comes near a cell from both sides, a particle's
path leaves the nearest copy of a sphere for another, and a distance is not to the nearest copy.  The
free-flight schedules against the per-substep one, bit for bit, alone and in an ensemble."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# box, colloids, radius, density, substeps, time of a step
BOXES = [((18, 30, 8), 5, 3.0, 10, 10, 0.05), ((25, 11, 29), 1, 4.0, 10, 10, 0.2), ((18, 34, 34), 1, 4.0, 10, 2, 0.5),
         ((21, 10, 11), 2, 3.0, 20, 5, 0.1), ((25, 11, 27), 14, 2.0, 20, 4, 0.1), ((7, 31, 22), 24, 2.0, 20, 3, 0.05),
         ((15, 8, 10), 1, 3.0, 20, 10, 0.1), ((7, 7, 7), 1, 2.0, 10, 10, 0.1),
         ((9, 12, 14), 1, 2.0, 20, 5, 0.5), ((8, 8, 20), 2, 1.5, 40, 5, 0.5), ((10, 8, 9), 1, 4.0, 20, 10, 0.1),
         ((9, 12, 14), 1, 2.0, 20, 25, 0.5), ((8, 8, 20), 2, 1.5, 40, 25, 0.5)]


def _params(i, form, L, nc, radius, density, n_sub, ndt):
    import brownian_gb300 as bg
    M = bg.displaced_mass(radius, density)
    return (L, L[0] * L[1] * L[2] * density, nc), dict(
        n_sub=n_sub, ndt=ndt, mass_colloid=M, sig_colloid=2 * radius, sigma=2 * radius, I_colloid=0.4 * M * radius ** 2,
        v0=0.02, theta_deg=90.0, Dr=0.001, seed=40 + i, init_gap=0.05, precision=bg.FP64 if form == "fp64" else bg.FP32C)


def _start(s):
    import brownian_gb300 as bg
    s.initialize(bg.INIT_PHYSICAL)
    s.setup()
    return s


def _steps(sim, n):
    """n steps; the refusal, if there is one (two of the boxes: a sphere outruns its bound within a long step)."""
    import brownian_gb300 as bg
    try:
        sim.step(n)
    except bg.MPCDError as e:
        return str(e)
    return ""


def _same(a, b):
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    assert a.diag()["events"] == b.diag()["events"] > 0


@pytest.mark.parametrize("form", ("fp64", "fp32c"))
@pytest.mark.parametrize("i", range(len(BOXES)))
def test_bits_of_the_per_substep_schedule(form, i):
    import brownian_gb300 as bg
    size, kw = _params(i, form, *BOXES[i])
    a, b = (_start(bg.Simulation(*size, **kw)) for _ in range(2))
    b.set_flight(False)
    refused = [_steps(sim, 12) for sim in (a, b)]
    assert refused[0] == refused[1] and (not refused[0] or i in (8, 9)), refused
    if not refused[0]:
        _same(a, b)
    a.close()
    b.close()


def test_bits_in_an_ensemble():
    import brownian_gb300 as bg
    params = []
    for i, box in enumerate(BOXES):
        size, kw = _params(i, "fp32c", *box[:4], 10, 0.2)
        params.append(bg.make_params(*size, **kw))
    a, b = bg.Ensemble(params), bg.Ensemble(params)
    b.set_flight(False)
    for e in (a, b):
        for s in e:
            _start(s)
        e.step(12)
    for x, y in zip(a, b):
        _same(x, y)
    a.close()
    b.close()
