"""A second upload into an engine, with another number of sites: the learned term's
arrays follow the count, and a topology that names sites that are gone is dropped."""
import ctypes

import numpy as np
import pytest

from host_engine import host, host_library  # noqa: F401


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _upload(g, s):
    arrays = [np.ascontiguousarray(x, np.float64) for x in (s.r, s.v, s.m, s.eps, s.sig)]
    mid = np.ascontiguousarray(s.mol_id, np.uint64)
    g._check(g.L.komd_gpu_upload_sites(g.h, s.n, *[_ptr(x) for x in arrays], _ptr(mid)))
    g.n = s.n


def _steps(g):
    g.update_container()
    g.forces()
    g.step(1)
    g.step(9)


@pytest.mark.parametrize("kept", [648, 216])
def test_topology(host, kept):  # noqa: F811
    from komd_gb300 import gpu, lattice
    s = lattice.triatomic_count(216, rho_site=0.5, t_star=1.0, seed=5, aligned=True)   # 648 sites
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3.0, cutoff=1.6, dt=0.002,
                                         terms=gpu.TERM_LJ | gpu.TERM_BONDED))
    _steps(g)
    assert host.fake_count(b"k_bonded_mol") == 11
    host.fake_reset()
    _upload(g, lattice.System(r=s.r[:kept], v=s.v[:kept], m=s.m[:kept], eps=s.eps[:kept], sig=s.sig[:kept],
                              mol_id=s.mol_id[:kept], low=s.low, high=s.high))
    _steps(g)
    bonded = host.fake_count(b"k_bonded_mol") + host.fake_count(b"k_bonds") + host.fake_count(b"k_angles")
    assert bonded == (11 if kept == s.n else 0)
    g.close()


def _learned(s):
    from komd_gb300 import gpu, surrogate
    g = gpu.GpuSystem(s, surrogate.physics_config(s, 2.2, rc=2.0, skin=0.0,
                                                  terms=gpu.TERM_LJ | gpu.TERM_ATM | gpu.TERM_ATM_SURROGATE))
    model = dict(params=surrogate.init_params(1), fmean=np.zeros(32, np.float32), fstd=np.ones(32, np.float32),
                 e_scale=0.1, e_shift=0.0)
    g.surrogate_load(model, probe_every=0)
    return g


def _boxes():
    from komd_gb300 import lattice
    small = lattice.argon_fcc(4, rho=0.8442, t_star=0.722, seed=7, jitter=0.05)    # 256 sites
    keep = np.arange(0, small.n, 2)                                               # half of them, in the same box
    few = lattice.System(r=small.r[keep], v=small.v[keep], m=small.m[keep], eps=small.eps[keep], sig=small.sig[keep],
                         mol_id=small.mol_id[keep], low=small.low, high=small.high)
    return few, small


def test_learned_arrays_follow_the_count(host):  # noqa: F811
    few, many = _boxes()
    g = _learned(few)
    _steps(g)
    moments = 36 * 4   # bytes a site
    assert host.fake_live(moments * few.n) == 1
    _upload(g, many)
    _steps(g)
    assert host.fake_live(moments * many.n) == 1 and host.fake_live(moments * few.n) == 0
    g.close()


@pytest.mark.gpu
def test_learned_forces_after_a_second_upload():
    few, many = _boxes()
    a, b = _learned(few), _learned(many)
    _steps(a)
    _upload(a, many)
    for g in (a, b):
        g.update_container()
        g.forces()
    fa, fb = a.download()[2], b.download()[2]
    # the same FP32 terms, summed by atomics in any order
    assert np.isfinite(fa).all() and np.abs(fa - fb).max() < 1e-5 * np.abs(fb).max()
    a.step(9)
    a.close()
    b.close()


def _verlet(s):
    from komd_gb300 import gpu
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3.0, cutoff=2.5, cutoff_3b=2.0, nu=0.073,
                                         dt=0.005, terms=gpu.TERM_LJ | gpu.TERM_ATM, skin=0.3,
                                         atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL,
                                         virial_mode=gpu.VIRIAL_CORRECT))
    g.update_container()
    g.forces()
    return g


def _calls(g):
    for n in (9, 9, 3, 3, 3, 1, 1):   # graphs of four steps, of three and of one
        g.step(n)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["same", "fewer"])
def test_step_graphs_after_a_second_upload(form):
    from komd_gb300 import lattice
    s = lattice.argon_fcc(6, rho=0.8442, t_star=1.4, seed=9, jitter=0.05)
    a = _verlet(s)
    _calls(a)
    keep = np.arange(0, s.n, 1 if form == "same" else 2)
    t = lattice.System(r=s.r[keep], v=-s.v[keep], m=s.m[keep], eps=s.eps[keep], sig=s.sig[keep],
                       mol_id=s.mol_id[keep], low=s.low, high=s.high)
    _upload(a, t)
    a.update_container()
    a.forces()
    b = _verlet(t)
    for g in (a, b):
        _calls(g)
    assert all(np.isfinite(x).all() and np.array_equal(x, y) for x, y in zip(a.download(), b.download()))
    a.close()
    b.close()


@pytest.mark.gpu
def test_step_graphs_after_a_change_of_terms():
    from komd_gb300 import gpu, lattice
    s = lattice.argon_fcc(6, rho=0.8442, t_star=1.4, seed=9, jitter=0.05)
    a, b = _verlet(s), _verlet(s)
    for terms in (gpu.TERM_LJ, gpu.TERM_LJ | gpu.TERM_ATM):
        _calls(a)
        for _ in range(29):
            b.step(1)
        for g in (a, b):
            g.set_terms(terms)
    _calls(a)
    for _ in range(29):
        b.step(1)
    assert all(np.isfinite(x).all() and np.array_equal(x, y) for x, y in zip(a.download(), b.download()))
    a.close()
    b.close()
