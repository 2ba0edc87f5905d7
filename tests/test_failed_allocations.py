"""A device allocation that fails while an engine replaces buffers: the call says
so, no captured step graph that holds the replaced buffers is launched any more, and
the engine either goes on as before (the new buffers had not taken the old ones'
place yet) or refuses to run until sites are uploaded again."""
import ctypes

import numpy as np
import pytest

from host_engine import host, host_library  # noqa: F401

ERR_STATE, ERR_NOMEM = 4, 5


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _molecules():
    from komd_gb300 import gpu, lattice
    s = lattice.triatomic_count(216, rho_site=0.5, t_star=1.0, seed=5, aligned=True)
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3.0, cutoff=1.6, skin=0.2, dt=0.002,
                                         terms=gpu.TERM_LJ | gpu.TERM_BONDED, virial_mode=gpu.VIRIAL_CORRECT))
    return s, g


def _argon(**kw):
    from komd_gb300 import gpu, lattice
    s = lattice.argon_fcc(5, rho=0.8442, t_star=0.722, seed=3, jitter=0.05)
    kw = dict(dict(cutoff=2.5, cutoff_3b=2.0, nu=0.073), **kw)
    return s, gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3.0, **kw))


def _start(g):
    g.update_container()
    g.forces()
    g.step(1)
    g.step(9)


def _with_failures(host, call, after_failure):  # noqa: F811
    """call() with its first, second, ... allocation failing, until none is left;
    returns how many failed."""
    for k in range(200):
        host.fake_fail_malloc(k)
        rc = call()
        host.fake_fail_malloc(-1)
        if rc == 0:
            return k
        assert rc == ERR_NOMEM
        host.fake_reset()
        after_failure()
        assert host.fake_stale_launches() == 0
    raise AssertionError("the call never succeeds")


def test_topology(host):  # noqa: F811
    s, g = _molecules()
    _start(g)
    b, a = np.ascontiguousarray(s.bonds, np.int64), np.ascontiguousarray(s.angles, np.int64)

    def after():
        g.step(1)
        g.step(9)
        assert host.fake_count(b"k_bonded_mol") == 10   # the old topology

    n = _with_failures(host, lambda: host.komd_gpu_set_topology(g.h, len(b), _ptr(b), len(a), _ptr(a)), after)
    assert n == 5
    host.fake_reset()
    after()
    assert host.fake_stale_launches() == 0
    g.close()


def test_second_upload(host):  # noqa: F811
    from komd_gb300 import gpu
    full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
    s, g = _argon(terms=gpu.TERM_LJ | gpu.TERM_ATM, skin=0.1, **full)
    _start(g)
    arrays = [np.ascontiguousarray(x, np.float64) for x in (s.r, s.v, s.m, s.eps, s.sig)]
    mid = np.ascontiguousarray(s.mol_id, np.uint64)

    def after():
        for f in (lambda: g.step(1), lambda: g.step(9), g.forces, g.update_container, g.integrate0,
                  lambda: g.measure(gpu.MEASURE_ENERGY), g.download):
            with pytest.raises(gpu.KomdError) as e:
                f()
            assert e.value.code == ERR_STATE
        assert host.fake_direct() == 0 and host.fake_graph_launches() == 0

    n = _with_failures(host, lambda: host.komd_gpu_upload_sites(g.h, s.n, *[_ptr(x) for x in arrays], _ptr(mid)), after)
    assert n > 20
    host.fake_reset()
    _start(g)
    assert host.fake_stale_launches() == 0
    g.close()


def test_learned_model(host):  # noqa: F811
    from komd_gb300 import gpu, surrogate
    full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
    s, g = _argon(terms=gpu.TERM_LJ | gpu.TERM_ATM | gpu.TERM_ATM_SURROGATE, skin=0.1, **full)
    p = surrogate.init_params(1).astype(np.float32)
    fm, fs = np.zeros(32, np.float32), np.ones(32, np.float32)
    g.surrogate_load(dict(params=p, fmean=fm, fstd=fs, e_scale=1.0, e_shift=0.0), probe_every=0)
    _start(g)

    def after():   # no model: the exact form
        g.step(1)
        g.step(9)
        assert host.fake_count(b"k_sur_") == 0 and host.fake_count(b"k_lj_atm") > 0

    n = _with_failures(host, lambda: host.komd_gpu_surrogate_load(g.h, _ptr(p), _ptr(fm), _ptr(fs), ctypes.c_double(1.0),
                                                                 ctypes.c_double(0.0), 0, ctypes.c_double(1.0)), after)
    assert n > 10
    host.fake_reset()
    g.step(9)
    assert host.fake_count(b"k_sur_mlp") == 9 and host.fake_stale_launches() == 0
    g.close()


def test_pair_table_and_its_positions(host):  # noqa: F811
    from komd_gb300 import gpu
    s, g = _argon(terms=gpu.TERM_LJ)
    _start(g)

    def runs():
        g.step(1)
        g.step(9)

    n = _with_failures(host, lambda: host.komd_gpu_set_terms(g.h, gpu.TERM_LJ | gpu.TERM_TABULATED), runs)
    assert n == 3
    x = np.linspace(0.6, 2.5, 50)
    g.set_pair_table(x, 1.0 / x)
    runs()
    x2 = np.linspace(0.6, 2.5, 80)
    y2 = 1.0 / x2
    n = _with_failures(host, lambda: host.komd_gpu_set_pair_table(g.h, 80, _ptr(x2), _ptr(y2), ctypes.c_double(1.0),
                                                                 ctypes.c_double(0.0)), runs)
    assert n == 3
    g.close()
