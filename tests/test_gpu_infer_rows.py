"""Inference at the edges of its row tiles (16, 32 and 64 rows a CTA, by how many CTAs the device
takes at once): a row's outputs do not depend on how many rows the call has, so every call must
leave the bits that the rows get elsewhere, nothing past its last row, and, at the first rows,
the CPU restatement's values."""
import numpy as np
import pytest

from oracle import mlp_ref as M

pytestmark = pytest.mark.gpu


def test_rows_do_not_depend_on_the_tile():
    import torch

    from brownian_gb300 import closure
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 64 * sm + 65
    rng = np.random.default_rng(7)
    net = closure.Network(max_batch=rows, seed=7)
    p = rng.normal(0, 0.08, net.n_params).astype(np.float32)
    net.set_params(p)
    xm, xs = rng.normal(0, 1, M.IN).astype(np.float32), rng.uniform(0.5, 2, M.IN).astype(np.float32)
    ym, ys = rng.normal(0, 1, M.NY).astype(np.float32), rng.uniform(0.5, 2, M.NY).astype(np.float32)
    net.set_normalisation(xm, xs, ym, ys)
    x = (xm + xs * rng.normal(0, 3, (rows, M.IN))).astype(np.float32)  # (some beyond the input clip)
    # an odd offset: the rows need no alignment beyond the element's
    buf = torch.zeros(rows * M.IN + 1, dtype=torch.float32, device="cuda")
    buf[1:] = torch.from_numpy(x.reshape(-1)).cuda()
    xd = buf[1:]
    whole = None
    for n in (rows, 64 * sm, 32 * sm + 1, 32 * sm, 16 * sm + 1, 16 * sm, 65, 64, 33, 17, 16, 15, 1):
        out = torch.full((rows * M.OUT + 1,), -77.0, dtype=torch.float32, device="cuda")
        net.forward(xd.data_ptr(), out[1:].data_ptr(), n)
        torch.cuda.synchronize()
        got = out[1:].cpu().numpy().reshape(rows, M.OUT)
        assert np.all(got[n:] == -77.0) and float(out[0]) == -77.0, n
        whole = got if whole is None else whole
        assert np.array_equal(got[:n].view(np.int32), whole[:n].view(np.int32)), n
    # 3e-4: the BF16 roundings that another order of the FP32 sums flips (as in the closure's tests)
    ref = M.forward(p, x[:500], xm, xs, ym, ys, bf16_emul=True)
    assert np.linalg.norm(whole[:500] - ref) <= 3e-4 * np.linalg.norm(ref)
    net.close()
