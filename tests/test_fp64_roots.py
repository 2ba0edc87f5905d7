"""rsqrt_d and sqrt_d (komd_gb300/csrc/engine.cuh) restated in numpy from
their FP64 operations (fused ones through long double, whose 64-bit products of
these operands are exact enough to round once): seeds off by up to two FP32
ulps, as the hardware's approximations may be, still give results within 0.51
ulp of the real value."""
import numpy as np
import pytest

L = np.longdouble
pytestmark = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs 80-bit long double")


def fma(a, b, c):
    """a * b + c rounded once: the product split exactly into two doubles."""
    p = a * b
    def split(x):
        t = 134217729.0 * x
        hi = t - (t - x)
        return hi, x - hi
    ah, al = split(a)
    bh, bl = split(b)
    err = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    s = L(p) + L(c)   # 64 bits: |c| is 1 or far above the error term
    return np.float64(s + L(err))


def ulps(y, exact):
    return np.abs((L(y) - exact) / np.spacing(np.abs(y)).astype(L)).astype(float)


def args():
    rng = np.random.default_rng(4)
    x = np.concatenate([rng.uniform(0.01, 100.0, 100000), np.exp(rng.uniform(-80, 80, 100000)),
                        np.nextafter(2.0 ** np.arange(-100, 100.0), 4.0)])
    trunc = (x.view(np.int64) & ~((1 << 29) - 1)).view(np.float64).astype(np.float32)
    return x, trunc, 1.0 + rng.integers(-2, 3, x.size) * 2.0 ** -23


def test_reciprocal_root_and_root():
    x, t, off = args()
    y0 = (1.0 / np.sqrt(t.astype(np.float64)) * off).astype(np.float32).astype(np.float64)
    e = fma(-x, y0 * y0, np.ones_like(x))
    y = fma(y0 * e, fma(e, np.full_like(x, 0.375), np.full_like(x, 0.5)), y0)
    assert ulps(y, L(1) / np.sqrt(L(x))).max() < 0.51
    r = x * y
    r = fma(fma(-r, r, x), 0.5 * y, r)
    assert ulps(r, np.sqrt(L(x))).max() < 0.51
