"""The FP64 free-flight pass's branch-free jump (kernels_fp64.cu, free_jump): n streaming steps of
one axis as the bit pattern of x plus n times the pattern difference of the first addition, where
that stays inside the binade of x and inside [2^-30 L, L) and the addition is no tie.  Restated
with 64-bit integers and checked bit for bit, wherever it says it applies, against n IEEE
additions x = mod(x + w, L) one by one."""
import numpy as np
import pytest

MANT, HIDDEN = np.int64(0xFFFFFFFFFFFFF), np.uint64(0x10000000000000)


def free_jump(x, w, n, L):
    bx, b1 = x.view(np.int64), (x + w).view(np.int64)
    aw = w.view(np.int64) & np.int64(0x7FFFFFFFFFFFFFFF)
    with np.errstate(over="ignore"):
        bn = bx + (b1 - bx) * np.int64(n)
    lo, hi = np.float64(np.ldexp(L, -30)).view(np.int64), np.float64(L).view(np.int64)
    inside = ((((b1 ^ bx) | (bn ^ bx)) >> 52) == 0) & ((bn & MANT) != 0)
    inside &= (bx >= lo) & (bn >= lo) & (bx < hi) & (bn < hi)
    sh = (bx >> 52) - (aw >> 52)
    mw = (aw & MANT).astype(np.uint64) | HIDDEN
    half = (mw << np.clip(64 - sh, 0, 63).astype(np.uint64)) == np.uint64(1 << 63)
    return inside & ~((sh >= 1) & (sh <= 53) & half), bn.view(np.float64)


def sequential(x, w, n, L):
    for _ in range(n):
        x = x + w
        q = (x - L * 0.5) / L
        t = np.trunc(q)
        t = np.where(np.abs(q - t) >= 0.5, t + np.sign(q), t)  # lround
        x = x - L * t
    return x


def cases(kind, L, rng):
    if kind == "thermal":
        return rng.uniform(0, L, 200000), rng.normal(0, 0.01, 200000)
    edge = 2.0 ** rng.integers(-32, int(np.log2(L)) + 1, 20000)
    if kind == "edges":  # binade edges and the box's, met exactly, by an ulp and by a few steps
        x = np.concatenate([edge, np.nextafter(edge, 0), np.nextafter(edge, 2 * L), edge - 0.01, np.full(2000, L)])
        w = rng.choice([0.02, -0.02, 1e-3, -1e-3, 1e-16, -1e-16, 0.0, 5e-324, 7.0, -7.0], x.size)
        return x, w
    x = rng.uniform(0.001, L, 50000)  # w = m u / 2 and m u / 4 for small and large m: ties among them
    u = np.spacing(x)
    m = rng.integers(-9, 10, x.size) + rng.choice([0.0, 2.0 ** 30, 2.0 ** 45], x.size)
    return x, m * u * rng.choice([0.5, 0.25], x.size)


@pytest.mark.parametrize("L", [7.0, 64.0, 53.0])
@pytest.mark.parametrize("n", [1, 10, 37])
@pytest.mark.parametrize("kind", ["thermal", "edges", "ties"])
def test_jump_equals_the_additions(kind, n, L):
    x, w = cases(kind, L, np.random.default_rng(n + int(L)))
    ok, got = free_jump(x, w, n, L)
    ref = sequential(x, w, n, L)
    assert np.array_equal(got[ok].view(np.int64), ref[ok].view(np.int64))
    if kind == "thermal" and n == 10 and L > 50:  # (the smaller the box, the more positions near its end)
        assert ok.mean() > 0.95  # what it leaves is the general routine's
