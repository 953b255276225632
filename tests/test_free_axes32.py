"""Two short forms of the FP32 free-flight pass (kernels_fp32c.cu) against what they stand for, restated
in Python: free_axes32's carry without rounding instructions (the offset leaves [0, 1) on the side it moves
to, the carried cells from the displacement) against floor's, and fix2's 32-bit steps against
the exact rounding of v 2^k and v^2 2^k, on random values and on the edges."""
from fractions import Fraction

import numpy as np
import pytest

F = np.float32


def fma(a, b, c):  # a b is exact in longdouble, and the sum nearly always
    return F(np.longdouble(a) * np.longdouble(b) + np.longdouble(c))


def by_floor(o, v, dt, n):
    k = 0
    for _ in range(n):
        o = fma(v, dt, o)
        f = np.floor(o)
        o = F(o - f)
        k += int(f)
        if o >= 1:
            o, k = F(0), k + 1
    return o, k


def by_side(o, v, dt, n):
    a = F(1) if v < 0 else F(-1)
    o0, top = o, F(0)
    for _ in range(n):
        o = fma(v, dt, o)
        if int(np.array(o).view(np.uint32)) >= 0x3F800000:
            o = F(o + a)
        top = max(top, o)
    k = int(np.rint(F(fma(v, F(n) * dt, o0) - o)))
    return None if not top < 1 else (o, k)


@pytest.mark.parametrize("n", [2, 10, 37])
def test_carry_by_side(n):
    rng = np.random.default_rng(n)
    dt = F(0.1) / F(10)
    ulp = F(2.0) ** -24
    o = np.concatenate([rng.uniform(0, 1, 2000), [0.0, 1 - 2.0 ** -24, 2.0 ** -149, 2.0 ** -30, 0.5] * 8]).astype(F)
    v = np.concatenate([rng.normal(0, 1, 1500), rng.uniform(-49, 49, 500),
                        np.repeat([1.0, -1.0, 100 * ulp, -100 * ulp, 0.0, -0.0, -50 * ulp, 49.9], 5)]).astype(F)
    taken = 0
    for a, b in zip(o, v):
        got = by_side(a, b, dt, n)
        if got is not None:
            taken += 1
            ref = by_floor(a, b, dt, n)
            assert got == ref, (a, b, got, ref)
    assert taken > 0.98 * len(o)


def fix2(v, k):
    b = int(np.array(v).view(np.uint32))
    e = (b >> 23) & 0xFF
    sh = e - 150 + k
    s = 158 - e - sh
    if not (0 <= sh <= 30 and 1 <= s <= 31):
        return None
    m = (b & 0x7FFFFF) | 0x800000
    f = (-m if b >> 31 else m) * (1 << sh)
    q = m * ((m << 8) & 0xFFFFFFFF)
    lo, hi = q & 0xFFFFFFFF, q >> 32
    low = ((hi << 32 | lo) >> s) & 0xFFFFFFFF
    rem = (lo << (32 - s)) & 0xFFFFFFFF
    r = ((hi >> s) << 32) | low
    return f, r + (1 if rem > 0x80000000 - (low & 1) else 0)


@pytest.mark.parametrize("k", [20, 40, 45, 52])
def test_fixed_point_terms(k):
    rng = np.random.default_rng(k)
    v = np.concatenate([rng.normal(0, 1, 3000), rng.normal(0, 0.01, 500), rng.uniform(-64, 64, 500),
                        [0.0, -0.0, 1.0, -1.0, 2.0 ** -11, 2.0 ** -12, 31.99999, 32.0, 1 + 2.0 ** -23, 3.5, 1.5,
                         2.0 ** -22, 1 - 2.0 ** -24, 1e-40]]).astype(F)
    for x in v:
        got = fix2(x, k)
        if got is None:
            continue
        fx = Fraction(float(x))
        # Fraction rounds half to even
        assert got[0] == round(fx * 2 ** k) and got[1] == round(fx * fx * 2 ** k), (x, k, got)
    if k == 45:
        assert np.mean([fix2(x, k) is not None for x in v[:3000]]) > 0.998
