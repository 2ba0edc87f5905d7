"""The LJ pass over the Verlet rows: one site a warp for small systems, two above
32 sites per SM (4864 on 152 SMs).  Site counts on both sides of the line, odd ones
(half of the last warp empty) and rows of several passes, against FP64 sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _system(n, mixed):
    from komd_gb300 import lattice
    s = lattice.argon_fcc(11, rho=0.8442, t_star=1.0, seed=4, jitter=0.08)
    keep = np.sort(np.random.default_rng(n).choice(s.n, n, replace=False))
    r = s.r[keep]
    eps, sig = np.ones(n), np.ones(n)
    if mixed:
        eps[1::3] = 0.7
        sig[1::3] = 0.9
    return lattice.System(r=r, v=s.v[keep], m=np.ones(n), eps=eps, sig=sig, mol_id=np.arange(n, dtype=np.uint64),
                          low=s.low, high=s.high)


@pytest.mark.parametrize("n", [4864, 4865, 4899, 5324])
@pytest.mark.parametrize("mixed,cutoff", [(False, 2.5), (True, 2.5), (False, 4.0)])
def test_lj_rows_against_fp64(n, mixed, cutoff):
    from scipy.spatial import cKDTree
    from komd_gb300 import gpu
    s = _system(n, mixed)
    L = s.box
    cell = float(L[0]) / np.floor(float(L[0]) / (cutoff + 0.3))
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=cutoff, terms=gpu.TERM_LJ, dt=0.001, skin=0.3,
                                         virial_mode=gpu.VIRIAL_CORRECT))
    g.update_container()
    g.forces()
    r, _, f = g.download()
    g.close()
    pairs = cKDTree(np.mod(r - s.low, L), boxsize=L).query_pairs(cutoff + 1e-4, output_type="ndarray")
    i, j = pairs.T
    d = r[i] - r[j]
    d -= L * np.round(d / L)
    q = np.linalg.norm(d, axis=1)
    sg, ee = 0.5 * (s.sig[i] + s.sig[j]), np.sqrt(s.eps[i] * s.eps[j])
    x6 = (sg / q) ** 6
    mag = 24.0 * ee * (2.0 * x6 * x6 - x6) / q
    inside = q <= cutoff
    pf = np.where(inside, mag / q, 0.0)[:, None] * d
    ref = np.zeros_like(r)
    np.add.at(ref, i, pf)
    np.add.at(ref, j, -pf)
    # FP32 cell-local positions: 4 roundings of at most two cell edges in a difference; the
    # force's r^-13 turns them into 14 times that over r, its own arithmetic and the row sum add 64
    # roundings of the larger of its two terms; a pair within the first error of the cutoff may
    # count either way
    delta = 4 * EPS * 2 * cell
    big = 24.0 * ee * (2.0 * x6 * x6 + x6) / q
    tol_p = np.where(inside, big * (14 * delta / q + 64 * EPS), 0.0) + np.where(np.abs(q - cutoff) < 2 * delta, np.abs(mag), 0.0)
    tol = np.zeros(n)
    np.add.at(tol, i, tol_p)
    np.add.at(tol, j, tol_p)
    assert (np.abs(f - ref).max(1) <= tol).all()


@pytest.mark.parametrize("n", [4863, 4865, 4899])
def test_triplet_list_of_the_rows(n):
    """the neighbour list that the rows emit gives the descriptors and triplet forces of the list
    of per-step cells (both in FP32, summed in another order)"""
    from komd_gb300 import gpu, surrogate
    s = _system(n, False)
    cell = float(s.high[0]) / np.floor(float(s.high[0]) / 2.8)
    out = []
    for skin in (0.0, 0.3):
        g = gpu.GpuSystem(s, surrogate.physics_config(s, cell, skin=skin))
        g.update_container()
        g.forces()
        out.append(g.surrogate_sample())
        g.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-4 * np.abs(a).max()
