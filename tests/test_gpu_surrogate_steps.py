"""The colloid-only step at the edges of its launches: one block of substeps up to 256 colloids and a
cluster beyond, and calls of one step against calls that mix the graphs of eight steps and of one (in
which the kernels overlap): the same bits.  The orientation, which runs beside the substeps, follows
its equations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sur(nc, seed, Dr=0.001):
    import brownian_gb300 as bg
    from brownian_gb300 import closure
    n1 = int(np.ceil(nc ** (1.0 / 3.0)))
    L = 6 * max(n1, 2)
    M = bg.displaced_mass(2.0, 10)
    p = bg.make_params(L, 1, nc, n_sub=10, mass_colloid=M, sig_colloid=4.0, sigma=4.0, I_colloid=0.4 * M * 4.0, v0=0.05,
                       theta_deg=90.0, Dr=Dr, seed=9)
    net = closure.Network(max_batch=64, seed=seed)
    net.set_normalisation(np.zeros(81), np.ones(81), np.zeros(6), np.full(6, 5.0))
    sur = closure.Surrogate(p, net)
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(n1)] * 3, indexing="ij"), -1).reshape(-1, 3)[:nc]
    pos = 6.0 * g + 1.0 + rng.uniform(0, 1.6, (nc, 3))
    ra = rng.normal(0, 1, (nc, 3))
    ra /= np.linalg.norm(ra, axis=1, keepdims=True)
    w = rng.normal(0, 0.04, (nc, 3))
    sur.set_state(pos, rng.normal(0, 0.05, (nc, 3)), w, ra)
    return sur, net, ra


@pytest.mark.parametrize("nc", [1, 33, 256, 257, 2048])
def test_steps_do_not_depend_on_how_they_are_called(nc):
    a, na, _ = _sur(nc, 3)
    b, nb, _ = _sur(nc, 3)
    a.step(17)
    for _ in range(17):
        b.step(1)
    sa, sb = a.get_state(), b.get_state()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
        assert np.all(np.isfinite(sa[k]))
    for s in (a, b, na, nb):
        s.close()


@pytest.mark.parametrize("nc", [40, 300])
def test_orientation_follows_omega(nc):
    sur, net, ra = _sur(nc, 4, Dr=0.0)
    w0 = sur.get_state()["ang_vel_colloid"]
    sur.step(1)
    st = sur.get_state()
    w1, n_sub, dt = st["ang_vel_colloid"], 10, 0.1 / 10
    r = sur.get_state()["ra"] * 0 + ra
    for l in range(n_sub):  # Omega moves in equal shares; the Euler matrix of Omega dt turns ra
        o = (w0 + (w1 - w0) * (l + 1) / n_sub) * dt
        s, c = np.sin(o), np.cos(o)
        (sx, sy, sz), (cx, cy, cz) = s.T, c.T
        m = np.array([[cy * cz, -cy * sz, sy],
                      [sx * sy * cz + cx * sz, -sx * sy * sz + cx * cz, -sx * cy],
                      [-cx * sy * cz + sx * sz, cx * sy * sz + sx * cz, cx * cy]])
        r = np.einsum("ijn,nj->ni", m, r)
        r /= np.linalg.norm(r, axis=1, keepdims=True)
    # ten rotations in FP32, each within a few 2^-22 (fast sine and cosine of small angles, 1e-7)
    assert np.allclose(st["ra"], r, atol=1e-5), np.abs(st["ra"] - r).max()
    sur.close()
    net.close()
