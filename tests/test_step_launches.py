"""What a call of komd_gpu_step launches (on the CPU: host code alone, no kernel
runs), and that calls of any length give the state of single steps (on the GPU)."""
import numpy as np
import pytest

from host_engine import host, host_library  # noqa: F401

FORMS = ["verlet_lj", "verlet_lj_atm", "verlet_switch", "verlet_molecules", "verlet_learned", "cells_lj",
         "cells_fp64_atm", "cells_fp32_full", "cells_compat_limit", "cells_learned", "cells_table", "thermostat",
         "thermostat_full"]


def engine(form):
    from komd_gb300 import gpu, lattice, surrogate
    if form == "verlet_molecules":
        s = lattice.triatomic_count(216, rho_site=0.5, t_star=1.0, seed=5, aligned=True)
        kw = dict(cutoff=1.6, terms=gpu.TERM_LJ | gpu.TERM_BONDED, bond_k=300.0, angle_k=50.0, angle_theta0=1.91,
                  dt=0.002, skin=0.2, virial_mode=gpu.VIRIAL_CORRECT)
    else:
        s = lattice.argon_fcc(6, rho=0.8442, t_star=0.722, seed=9, jitter=0.05)
        full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
        lj, atm = gpu.TERM_LJ, gpu.TERM_LJ | gpu.TERM_ATM
        learned = dict(terms=atm | gpu.TERM_ATM_SURROGATE, **full)
        kw = {"verlet_lj": dict(terms=lj, skin=0.3, virial_mode=gpu.VIRIAL_CORRECT),
              "verlet_lj_atm": dict(terms=atm, skin=0.3, **full),
              "verlet_switch": dict(terms=atm, skin=0.3, switch_width=0.3, **full),
              "verlet_learned": dict(skin=0.3, **learned),
              "cells_lj": dict(terms=lj),
              "cells_fp64_atm": dict(terms=atm, precision=gpu.FP64),
              "cells_fp32_full": dict(terms=atm, **full),
              "cells_compat_limit": dict(terms=atm | gpu.TERM_LIMIT, limit=20.0),
              "cells_learned": learned,
              "cells_table": dict(terms=gpu.TERM_TABULATED, precision=gpu.FP64),
              "thermostat": dict(terms=lj, thermostat=1, temperature_target=1.2),
              "thermostat_full": dict(terms=atm, skin=0.3, thermostat=1, temperature_target=1.2, **full)}[form]
        kw = dict(dict(cutoff=2.5, cutoff_3b=2.0, nu=0.073, dt=0.005), **kw)
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3.0, **kw))
    if form == "cells_table":
        x = np.linspace(0.6, 2.5, 50)
        g.set_pair_table(x, 24.0 * (2.0 * x ** -13 - x ** -7))
    g.update_container()
    if form.endswith("learned"):
        x, _, _ = g.surrogate_sample()
        g.surrogate_load(dict(params=surrogate.init_params(1), fmean=x.mean(0).astype(np.float32),
                              fstd=(x.std(0) + 1e-6).astype(np.float32), e_scale=1.0, e_shift=0.0), probe_every=0)
    g.forces()
    return g


@pytest.mark.parametrize("form", FORMS)
def test_short_calls_are_graphs(host, form):  # noqa: F811
    """A step of a small system is shorter than the launches of its kernels one by
    one: a call of a few steps that comes again is launched as graphs, captured once."""
    g = engine(form)
    for n in (1, 2, 3, 4):
        g.step(n)
        g.step(n)
        host.fake_reset()
        for _ in range(3):
            g.step(n)
        assert host.fake_direct() == 0 and host.fake_captures() == 0
        assert host.fake_replayed() > 0 and host.fake_stale_launches() == 0
        assert host.fake_graph_launches() <= 3 * n
    g.close()


@pytest.mark.parametrize("form", FORMS + ["bonds_by_atomics", "learned_probed", "no_table"])
def test_reported_kernels_are_those_launched(host, form):  # noqa: F811
    from komd_gb300 import gpu
    g = engine({"bonds_by_atomics": "verlet_molecules", "learned_probed": "verlet_learned",
                "no_table": "cells_lj"}.get(form, form))
    if form == "bonds_by_atomics":   # one chain of all sites
        b = np.array([[k, k + 1] for k in range(g.n - 1)], np.int64)
        g._check(g.L.komd_gpu_set_topology(g.h, len(b), b.ctypes.data, 0, None))
    if form == "learned_probed":
        g.surrogate_load(dict(params=np.zeros(6337, np.float32), fmean=np.zeros(32, np.float32),
                              fstd=np.ones(32, np.float32), e_scale=1.0, e_shift=0.0), probe_every=3,
                         probe_threshold=1e9)
        g.step(4)
    if form == "no_table":
        g.set_terms(gpu.TERM_LJ | gpu.TERM_TABULATED)
    probes = lambda: g.surrogate_status()["probes"] if form == "learned_probed" else 0  # noqa: E731
    for profiling in (False, True):
        g.set_profiling(profiling)
        for n in (1, 2, 3, 4, 5, 9, 22):
            host.fake_reset()
            before, said = probes(), g.step_kernels(n)
            assert n != 1 or said == g.kernels_per_step()
            g.step(n)
            # a probe: the exact triplets and their flush, the learned term's four, the comparison
            assert host.fake_direct() + host.fake_replayed() == said + 7 * (probes() - before)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [f for f in FORMS if not f.endswith("learned")])
def test_calls_equal_single_steps(form):
    for n in (2, 3, 4, 9):
        a, b = engine(form), engine(form)
        for _ in range(3):   # directly, captured, replayed
            a.step(n)
            for _ in range(n):
                b.step(1)
        assert all(np.isfinite(p).all() and np.array_equal(p, q) for p, q in zip(a.download(), b.download()))
        a.close()
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [f for f in FORMS if f.endswith("learned")])
def test_learned_boundary_between_two_steps(form):
    """The pass between two steps with the learned term.  Both start from forces
    without it, so the positions before it are the same bit for bit, so are the
    network's outputs, and only the order of the FP32 atomics that sum the forces is
    free: at most 64 roundings of a sum of 64 pair shares, which the drift carries into
    the positions with dt^2 / m (m = 1).  A missing or doubled learned force would be
    some thousand times that."""
    from komd_gb300 import gpu
    a, b = engine(form), engine(form)
    for g in (a, b):
        g.set_terms(gpu.TERM_LJ)
        g.update_container()
        g.forces()
        g.set_terms(gpu.TERM_LJ | gpu.TERM_ATM | gpu.TERM_ATM_SURROGATE)
    a.step(2)
    b.step(1)
    top = np.abs(b.download()[2]).max()
    b.step(1)
    (ra, va, fa), (rb, _, _) = a.download(), b.download()
    assert all(np.isfinite(x).all() for x in (ra, va, fa))
    assert np.abs(ra - rb).max() <= 0.005 ** 2 * 64 * 64 * 2.0 ** -24 * top
    a.close()
    b.close()
