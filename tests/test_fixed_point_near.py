"""The force accumulators' FP32 -> 64-bit fixed-point conversion below 2^20
(komd_gb300/csrc/atm_device.cuh, fix32_rn): half-integers off the sum with
1.5 2^22, the rest by one 32-bit conversion.  Restated in numpy with the same IEEE
operations and checked bit for bit against rounding x * 2^32."""
import numpy as np
import pytest

F = np.float32


def near(x):
    x = np.asarray(x, F)
    big = F(6291456.0)
    t = x + big
    rem = x - (t - big)
    scaled = rem * F(4294967296.0)
    assert (np.abs(scaled.astype(np.float64)) <= 2.0 ** 30).all()      # inside one 32-bit conversion
    lo = np.rint(scaled).astype(np.int64)
    h = big.view(np.int32).astype(np.int64) - t.view(np.int32).astype(np.int64)
    return h * -(2 ** 31) + lo


def direct(x):
    return np.rint(np.asarray(x, F).astype(np.float64) * 2.0 ** 32).astype(np.int64)


@pytest.mark.parametrize("lo,hi", [(0, 2 ** 32), (0x3a000000, 0x49800000), (0x2e000000, 0x3c000000)])
def test_random_bit_patterns(lo, hi):
    bits = np.random.default_rng(lo % 97).integers(lo, hi, size=2_000_000, dtype=np.uint64).astype(np.uint32)
    x = bits.view(F)
    x = x[np.isfinite(x)]
    x = x[np.abs(x) < 2.0 ** 20]
    x = np.concatenate([x, -x])
    assert x.size > 500_000 and np.array_equal(near(x), direct(x))


def test_edges():
    e = np.arange(-40, 20)
    x = np.concatenate([F(2.0) ** e, F(3.0) * F(2.0) ** (e - 2), F(2.0) ** e + F(0.25), np.arange(0, 64) * F(0.25)]).astype(F)
    x = np.concatenate([x, np.nextafter(x, F(np.inf)), np.nextafter(x, F(0)), [F(0), F(2 ** 20 - 0.0625), F(1e-38)]]).astype(F)
    x = x[np.abs(x) < 2.0 ** 20]
    x = np.concatenate([x, -x])
    assert np.array_equal(near(x), direct(x))
    assert near(F(2.0 ** -33)) == 0 and near(F(3 * 2.0 ** -33)) == 2   # ties to even
