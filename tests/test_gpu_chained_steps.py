"""Several steps in one call share a pass at every step boundary (the end of one
step with the drift of the next); one step per call does not.  Both give the
same state bit for bit, list rebuilds on the way included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = ["verlet_lj", "verlet_lj_atm", "verlet_atm2b_limit", "verlet_molecules", "cells_fp64", "cells_fp32_full",
         "cells_compat", "cells_table", "thermostat"]


def _engine(form):
    from komd_gb300 import gpu, lattice
    if form == "verlet_molecules":
        s = lattice.triatomic_count(216, rho_site=0.5, t_star=1.0, seed=5, aligned=True)
        cell = float(s.high[0]) / 3.0
        kw = dict(cutoff=1.6, terms=gpu.TERM_LJ | gpu.TERM_BONDED, bond_k=300.0, angle_k=50.0, angle_theta0=1.91,
                  dt=0.002, skin=0.2, virial_mode=gpu.VIRIAL_CORRECT)
    else:
        s = lattice.argon_fcc(6, rho=0.8442, t_star=1.4, seed=9, jitter=0.05)
        cell = float(s.high[0]) / 3.0
        full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
        lj, atm = gpu.TERM_LJ, gpu.TERM_LJ | gpu.TERM_ATM
        kw = {"verlet_lj": dict(terms=lj, skin=0.3, virial_mode=gpu.VIRIAL_CORRECT),
              "verlet_lj_atm": dict(terms=atm, skin=0.3, **full),
              "verlet_atm2b_limit": dict(terms=atm | gpu.TERM_ATM2B | gpu.TERM_LIMIT, limit=30.0, skin=0.3, **full),
              "cells_fp64": dict(terms=atm, precision=gpu.FP64),
              "cells_fp32_full": dict(terms=atm, **full),
              "cells_compat": dict(terms=atm | gpu.TERM_LIMIT, limit=20.0),
              "cells_table": dict(terms=gpu.TERM_TABULATED, precision=gpu.FP64),
              "thermostat": dict(terms=lj, skin=0.3, virial_mode=gpu.VIRIAL_CORRECT, thermostat=1,
                                 temperature_target=1.2)}[form]
        kw = dict(dict(cutoff=2.5, cutoff_3b=2.0, nu=0.073, dt=0.005), **kw)
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, **kw))
    if form == "cells_table":
        x = np.linspace(0.6, 2.5, 50)
        g.set_pair_table(x, 24.0 * (2.0 * x ** -13 - x ** -7))
    g.update_container()
    g.forces()
    return g


@pytest.mark.parametrize("form", FORMS)
def test_steps_in_one_call_equal_single_steps(form):
    a, b = _engine(form), _engine(form)
    for n in (2, 1, 37, 3):
        a.step(n)
        for _ in range(n):
            b.step(1)
        for x, y in zip(a.download(), b.download()):
            assert np.isfinite(x).all() and np.array_equal(x, y)
    a.close()
    b.close()
