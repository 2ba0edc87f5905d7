"""The device's own results of the scalar functions that test_fp64_roots,
test_fixed_point, test_fixed_point_near and test_cell_index restate in numpy."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    from komd_gb300 import build
    out = str(tmp_path_factory.mktemp("dev") / "libdevice_functions.so")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + build.ARCH +
                   ["-shared", os.path.join(ROOT, "tests", "device_functions.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _ulps(y, exact):
    return (np.abs(y.astype(np.longdouble) - exact) / np.spacing(np.abs(y)).astype(np.longdouble)).astype(float)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs a long double of 64 bits or more")
def test_roots_within_half_an_ulp(device):
    rng = np.random.default_rng(5)
    x = np.concatenate([rng.uniform(0.01, 100.0, 100000), np.exp(rng.uniform(-86, 86, 100000)),
                        np.nextafter(2.0 ** np.arange(-124, 124.0), 4.0), 2.0 ** np.arange(-125, 125.0)])
    y, s = np.empty_like(x), np.empty_like(x)
    assert device.roots(x.size, _ptr(x), _ptr(y), _ptr(s)) == 0
    root = np.sqrt(x.astype(np.longdouble))
    assert _ulps(y, 1 / root).max() < 0.51
    assert _ulps(s, root).max() < 0.51


def test_roots_outside_the_seed_range(device):
    x = np.array([0.0, np.inf, np.nan, -1.0, 1e-300, 5e-324, 1e300, 2.0 ** -126, 2.0 ** 126])
    y, s = np.empty_like(x), np.empty_like(x)
    assert device.roots(x.size, _ptr(x), _ptr(y), _ptr(s)) == 0
    with np.errstate(divide="ignore", invalid="ignore"):
        ry, rs = 1.0 / np.sqrt(x), np.sqrt(x)
    assert np.array_equal(np.isnan(y), np.isnan(ry)) and np.array_equal(np.isnan(s), np.isnan(rs))
    ok = ~np.isnan(rs)
    assert np.array_equal(s[ok], rs[ok])                                       # an IEEE root
    fin = ok & np.isfinite(ry)
    assert np.array_equal(y[ok & ~fin], ry[ok & ~fin]) and (np.abs(y[fin] - ry[fin]) <= 4e-16 * ry[fin]).all()


def test_fixed_point_is_the_rounded_product(device):
    rng = np.random.default_rng(6)
    e = np.arange(-40, 31)
    x = np.concatenate([2.0 ** e, 3.0 * 2.0 ** (e - 2), np.arange(0, 64) * 0.25, 2.0 ** 20 + np.arange(-8, 8) * 0.0625,
                        rng.uniform(-100, 100, 200000), rng.normal(0, 1, 200000) * 2.0 ** rng.integers(-40, 30, 200000)])
    x = x.astype(np.float32)
    x = np.concatenate([x, np.nextafter(x, np.float32(np.inf)), np.nextafter(x, np.float32(0)), -x])
    x = np.ascontiguousarray(x[np.abs(x) < 2.0 ** 31])
    q = np.empty(x.size, np.int64)
    assert device.fix(x.size, _ptr(x), _ptr(q)) == 0
    assert np.array_equal(q, np.rint(x.astype(np.float64) * 2.0 ** 32).astype(np.int64))
    x = np.full(4, np.nan, np.float32)
    q = np.empty(4, np.int64)
    assert device.fix(4, _ptr(x), _ptr(q)) == 0 and (q == 0).all()


@pytest.mark.parametrize("cs", [2.5, 2.7990000000000004, 4.8])
def test_cells_are_the_truncated_ieee_quotient(cs):
    """sites at, just below and just above every cell edge"""
    from komd_gb300 import gpu, lattice
    nd, low = 7, np.array([0.0, -3.1, 10.0])
    high = low + nd * cs + 0.3 * cs          # the last cell is stretched
    rng = np.random.default_rng(7)
    k = np.arange(nd + 1).astype(np.float64) * cs
    edge = np.concatenate([k, np.nextafter(k, np.inf), np.nextafter(k, -np.inf), k + 1e-9 * cs, k - 1e-9 * cs,
                           k + 3e-9 * cs])
    r = low + rng.choice(edge, (4000, 3))
    r = np.clip(r, low, high)
    n = len(r)
    s = lattice.System(r=r, v=np.zeros((n, 3)), m=np.ones(n), eps=np.ones(n), sig=np.ones(n),
                       mol_id=np.arange(n, dtype=np.uint64), low=low, high=high)
    g = gpu.GpuSystem(s, gpu.make_config(low, high, cs, cutoff=2.5))
    g.update_container()
    count, _ = g.cells()
    assert g.grid_dims() == (nd, nd, nd)
    g.close()
    b = np.clip(((r - low) / cs).astype(np.int64), 0, nd - 1) + 1
    want = np.bincount(b[:, 0] + (nd + 2) * (b[:, 1] + (nd + 2) * b[:, 2]), minlength=(nd + 2) ** 3)
    inner = np.zeros((nd + 2,) * 3, bool)
    inner[1:-1, 1:-1, 1:-1] = True
    assert np.array_equal(count[inner.ravel()], want[inner.ravel()])
