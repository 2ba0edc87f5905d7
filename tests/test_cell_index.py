"""The binning's quotient (cell_index, kernels.cu) restated: truncating
x * (1 / cs) away from the integers, and the IEEE division near them, gives
the truncated IEEE quotient for every x and cs."""
import numpy as np
import pytest


def cell_index(x, cs, nd):
    t = x * (1.0 / cs)
    with np.errstate(invalid="ignore"):
        q0 = np.trunc(t)
    fr = t - q0
    fast = (q0 >= 0) & (q0 < 1e6) & (fr > 1e-9) & (fr < 1.0 - 1e-9)
    q = np.where(fast, q0, np.trunc(x / cs))
    return np.clip(q, 0, nd - 1), fast


@pytest.mark.parametrize("cs", [2.5, 2.7990000000000004, 1.0 / 3.0, 0.1, 67.3, 4.8])
def test_cell_index_is_the_truncated_quotient(cs):
    rng = np.random.default_rng(3)
    nd = 1 << 20
    k = rng.integers(0, nd + 2, 200000).astype(np.float64)
    edges = np.concatenate([k * cs, np.nextafter(k * cs, np.inf), np.nextafter(k * cs, -np.inf),
                            k * cs + cs * rng.uniform(-3e-9, 3e-9, k.size)])
    x = np.concatenate([edges, rng.uniform(-cs, (nd + 1) * cs, 400000), rng.uniform(0, 50 * cs, 400000), [0.0, -0.0]])
    q, fast = cell_index(x, cs, nd)
    assert np.array_equal(q, np.clip(np.trunc(x / cs), 0, nd - 1))
    assert fast[edges.size:].mean() > 0.9   # the rule matters: nearly every site takes the product
