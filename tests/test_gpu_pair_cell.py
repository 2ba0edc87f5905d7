"""The per-step pair kernel (FP64 forces, FENE, the tabulated force) and the FP64
triplets against the FP64 oracle, where their shapes change: cells emptier
than a block's warps, neighbourhoods of several staging rounds, rows around a
warp's 32 entries, two species, molecules.  Bars as in test_gpu_parity: FP64
forces to 1e-12, FP32 forces to a relative RMSE of 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_rmse(a, b):
    return float(np.sqrt(((a - b) ** 2).sum(1).mean()) / np.sqrt((b ** 2).sum(1).mean()))


def _system(form):
    """(system, cell edge): sparse -- about one site per cell; liquid -- 18;
    crowded -- 76 (four staging rounds); molecules -- three-site, two species."""
    from komd_gb300 import lattice
    if form == "molecules":
        s = lattice.triatomic_sc(5, rho_site=0.3, t_star=0.5, seed=71, r0=0.97, theta0_deg=90.0)
        return s, 2.5
    if form == "sparse":
        s = lattice.argon_fcc(4, rho=0.07, t_star=0.7, seed=72, jitter=0.35)
        return s, 2.5
    s = lattice.argon_fcc(6 if form == "liquid" else 8, rho=0.8442, t_star=0.722, seed=73, jitter=0.05)
    return s, float(s.high[0]) / (4.0 if form == "liquid" else 3.0)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("form", ["sparse", "liquid", "crowded", "molecules"])
def test_cell_list_forces_match_oracle(oracle_lib, form, mixed):
    """LJ + FENE in both precisions, and the tabulated force."""
    from komd_gb300 import gpu
    s, cell = _system(form)
    if mixed:
        s.eps[::2], s.sig[::2] = 0.7, 0.95
    sim = oracle_lib.OracleSim(s, cell, 2.4, fene=True)
    sim.update_container()
    sim.forces()
    assert np.isfinite(sim.f).all()
    for precision, bar in ((gpu.FP64, 1e-12), (gpu.FP32, 1e-5)):
        g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.4, terms=gpu.TERM_LJ | gpu.TERM_FENE,
                                             precision=precision))
        g.update_container()
        g.forces()
        f = g.download()[2]
        u = g.measure(gpu.MEASURE_ENERGY)["u_lj"]
        g.close()
        assert rel_rmse(f, sim.f) < bar
        assert u == pytest.approx(sim.lj_out.u_total, rel=1e-11 if precision == gpu.FP64 else 2e-5)
    x = np.concatenate([[0.3], np.sort(np.random.default_rng(5).uniform(0.31, 2.2, 41))])   # uneven nodes, r beyond the last
    table = (x, 2.0 / x ** 2, 50.0, 0.25)
    sim = oracle_lib.OracleSim(s, cell, 2.4, lj=False, table=table)
    sim.update_container()
    sim.forces()
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.4, terms=gpu.TERM_TABULATED, precision=gpu.FP64))
    g.set_pair_table(*table)
    g.update_container()
    g.forces()
    assert rel_rmse(g.download()[2], sim.f) < 1e-12
    g.close()


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("form", ["sparse", "liquid", "crowded"])
def test_fp64_triplets_match_oracle(oracle_lib, form, full):
    """FP64 ATM forces in both triplet sets, energy and count in the full one
    (the oracle's compat sweep counts list entries, images among them); the
    cutoffs give vertices with no neighbour, with partly filled batches, and
    (crowded) with more than 32 neighbours and several batches each."""
    from komd_gb300 import gpu
    s, cell = _system(form)
    rc3 = 2.4 if form == "crowded" else 1.9
    sim = oracle_lib.OracleSim(s, cell, 2.4, nu=0.073, cutoff_atm=rc3, atm=True, atm_mode="full" if full else "compat")
    sim.update_container()
    sim.forces()
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.4, cutoff_3b=rc3, nu=0.073,
                                         terms=gpu.TERM_LJ | gpu.TERM_ATM, precision=gpu.FP64,
                                         atm_enum=gpu.ATM_ENUM_FULL if full else gpu.ATM_ENUM_COMPAT))
    g.update_container()
    g.forces()
    f = g.download()[2]
    o = g.measure(gpu.MEASURE_ENERGY)
    g.close()
    assert rel_rmse(f, sim.f) < 1e-12
    if full:
        assert o["triplets"] == sim.atm_out.triplets
        assert o["u_atm"] == pytest.approx(sim.atm_out.energy, rel=1e-11)


@pytest.mark.parametrize("form", ["sparse", "liquid", "crowded", "molecules"])
def test_verlet_list_forces_match_oracle(oracle_lib, form):
    """The Verlet list build where its units change: parts of few cells, cells
    with no or one site, neighbourhoods of several staging rounds, molecules
    (the same-molecule bit).  After 30 steps from the list, the forces are the
    oracle's at the engine's positions."""
    from komd_gb300 import gpu, lattice
    s, cell = _system(form)
    rc = 1.5 if form == "molecules" else 2.1   # every site pair in range lies in adjacent cells
    if form == "molecules":
        cell = float(s.high[0]) / 3.0
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=rc, terms=gpu.TERM_LJ, skin=0.3, dt=0.002,
                                         virial_mode=gpu.VIRIAL_CORRECT))
    g.update_container()
    g.forces()
    g.step(30)
    r, v, f = g.download()
    g.close()
    at = lattice.System(r=r, v=v, m=s.m, eps=s.eps, sig=s.sig, mol_id=s.mol_id, low=s.low, high=s.high)
    sim = oracle_lib.OracleSim(at, cell, rc)
    sim.update_container()
    sim.forces()
    assert rel_rmse(f, sim.f) < 1e-5


@pytest.mark.parametrize("nbins", [7, 250, 3001])
@pytest.mark.parametrize("form", ["sparse", "liquid", "crowded", "molecules"])
def test_rdf_counts_are_exact(form, nbins):
    """The cell path of the RDF against the reference's arithmetic on every
    ordered pair of centres: few and many bins (shared and global counts; 7
    does not divide max_r evenly), some staging rounds, parts of cells."""
    from komd_gb300 import gpu
    s, cell = _system(form)
    max_r, mol = 2.4, np.searchsorted(np.unique(s.mol_id), s.mol_id)
    L = s.high - s.low
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.4, terms=gpu.TERM_LJ))
    g.update_container()
    got = g.rdf_profile(max_r, nbins)
    r = g.download()[0]
    g.close()
    com = np.stack([np.bincount(mol, r[:, d]) for d in range(3)], 1) / np.bincount(mol)[:, None]
    dr, expect = max_r / nbins, np.zeros(nbins)
    for k in range(com.shape[0]):
        q = com[k] - com
        q -= L * np.round(q / L)
        rr = np.sqrt((q[:, 0] * q[:, 0] + q[:, 1] * q[:, 1]) + q[:, 2] * q[:, 2])
        rr = np.delete(rr, k)
        np.add.at(expect, np.minimum((rr[rr <= max_r] / dr).astype(np.int64), nbins - 1), 1.0)
    assert np.array_equal(got, expect)
