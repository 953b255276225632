"""Training's kernels at the edges of their tiles: 128 rows a CTA of the layers' products, stages of 64
rows and up to n_sm / 12 slices of the batch in the weight gradients' (a slice with one row, one stage
exactly, one row more), against the CPU restatement, and the same bits from the same call."""
import numpy as np
import pytest

from oracle import mlp_ref as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 768, 769, 5000])
def test_gradients_at_the_edges_of_the_tiles(n):
    import torch

    from brownian_gb300 import closure
    rng = np.random.default_rng(40 + n)
    net = closure.Network(max_batch=n, seed=1)
    p = rng.normal(0, 0.08, net.n_params).astype(np.float32)
    net.set_params(p)
    xm, xs = rng.normal(0, 1, M.IN).astype(np.float32), rng.uniform(0.5, 2, M.IN).astype(np.float32)
    ym, ys = rng.normal(0, 1, M.NY).astype(np.float32), rng.uniform(0.5, 2, M.NY).astype(np.float32)
    net.set_normalisation(xm, xs, ym, ys)
    x = (xm + xs * rng.normal(0, 1, (n, M.IN))).astype(np.float32)
    y = (ym + ys * rng.normal(0, 1, (n, M.NY))).astype(np.float32)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    loss, g = net.grad(xd.data_ptr(), yd.data_ptr(), n)
    again = net.grad(xd.data_ptr(), yd.data_ptr(), n)
    assert loss == again[0] and np.array_equal(g.view(np.int32), again[1].view(np.int32))
    lref, gref = M.loss_and_grad(p, x, y, xm, xs, ym, ys, bf16_emul=True)
    assert abs(loss - lref) <= 1e-5 * abs(lref)
    # both round to BF16 in the same places; where the order of an FP32 sum flips a rounding, that value is
    # off by up to 2^-8 of itself, and few rows average little of it away (the products one layer at a
    # time, as they were before, are off by the same 1.0e-3 of the norm at 64 rows of these)
    tol = 2.0 ** -8
    o = 0
    for k, m in M.DIMS:
        for size in (k * m, m):
            a, b = g[o:o + size], gref[o:o + size]
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b) + 1e-7, (o, size)
            o += size
    # a step moves every parameter by Adam's first step (lr times the gradient's sign, where it is not tiny)
    net.train_step(xd.data_ptr(), yd.data_ptr(), n, 1e-3)
    d = net.params() - p
    big = np.abs(g) > 1e-5
    assert np.allclose(d[big], -1e-3 * np.sign(g[big]), atol=2e-6)
    net.close()
