"""A free-flight step of the FP64 form with more particles near the spheres than there are records for
(N / 16 + 65,536): it is refused as every other overflow, no two particles share a record meanwhile, and
the simulation goes on from a new state with the bits of one that never met it."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L, N, RADIUS = 24, 552_960, 3.4


def _sim():
    """27 spheres on a lattice that they fill to a third (each within the 342 boxes about its own)."""
    import brownian_gb300 as bg
    M = bg.displaced_mass(RADIUS, 40)
    return bg.Simulation(L, N, 27, n_sub=2, mass_colloid=M, sig_colloid=0.1, sigma=2 * RADIUS, I_colloid=0.4 * M * RADIUS ** 2,
                         v0=0.0, theta_deg=90.0, Dr=0.0, seed=7, max_per_cell=256)


def _state(inside):
    """The fluid anywhere (a third of it inside the spheres), or in the gaps between them."""
    rng = np.random.default_rng(5)
    X = np.stack(np.meshgrid(*[np.arange(3) * 8.0 + 4.3] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = rng.uniform(0.01, L - 0.01, (N if inside else 2 * N, 3))
    if not inside:
        d = np.abs(pos - 4.3) % 8.0
        d = np.minimum(d, 8.0 - d)
        pos = pos[(d * d).sum(1) > (RADIUS + 0.05) ** 2][:N]
    assert len(pos) == N
    ra = np.zeros((27, 3))
    ra[:, 0] = 1.0
    return pos, rng.normal(0, 1, pos.shape), X, np.zeros((27, 3)), np.zeros((27, 3)), ra


def _steps(sim, flight, n):
    """n steps from the state in the gaps; the refusal, if there is one (a wall collision of the hottest of so
    many particles may exceed the displacement bound)."""
    import brownian_gb300 as bg
    sim.set_state(*_state(False))
    sim.setup()
    sim.set_flight(flight)
    try:
        sim.step(n)
    except bg.MPCDError as e:
        return str(e)
    return ""


@pytest.mark.parametrize("flight", (True, False))
def test_more_pending_particles_than_records(flight):
    import brownian_gb300 as bg
    a, b = _sim(), _sim()
    a.set_state(*_state(True))
    a.setup()
    a.set_flight(flight)
    with pytest.raises(bg.MPCDError) as e:
        a.step(3)
    # (which particles find no room depends on the order of the blocks, and so does what else the two steps
    # behind that one report: a range bit, 4 or 64, makes it code 4)
    bits = int(re.search(r"bits (0x[0-9a-f]+)", str(e.value))[1], 16)
    assert bits & 0x80 and e.value.code == (4 if bits & 0x44 else 3), str(e.value)
    _steps(b, flight, 3)  # (the draws are keyed by the step)
    refused = [_steps(s, flight, 4) for s in (a, b)]
    assert refused[0] == refused[1] and "event lists" not in refused[0], refused
    x, y = a.get_state(), b.get_state()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    a.close()
    b.close()
