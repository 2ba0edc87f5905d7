"""A position that is not finite stays with its own site in the FP32 passes: the
forces of all others are those of the system without that site."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP32_FORCE_RMSE = 1e-5   # the repository's bar for FP32 forces
FORMS = ["rows_one_a_warp", "rows_two_a_warp", "rows_two_a_warp_mixed", "half", "half_mixed", "half_switch", "full_rows",
         "cells_lj", "cells_compat", "cells_full"]


def _system(form):
    from komd_gb300 import lattice
    s = lattice.argon_fcc(11 if "two_a_warp" in form else 6, rho=0.8442, t_star=0.722, seed=4, jitter=0.05)
    if form.endswith("mixed"):
        s.eps[1::3] = 0.7
        s.sig[1::3] = 0.9
    return s


def _engine(form, s):
    from komd_gb300 import gpu
    lj, atm = gpu.TERM_LJ, gpu.TERM_LJ | gpu.TERM_ATM
    full = dict(atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)
    kw = {"rows": dict(terms=lj, skin=0.3, virial_mode=gpu.VIRIAL_CORRECT),
          "half": dict(terms=atm, skin=0.3, **full),
          "full_rows": dict(terms=atm | gpu.TERM_LIMIT, limit=1e6, skin=0.3, **full),
          "cells_lj": dict(terms=lj), "cells_compat": dict(terms=atm), "cells_full": dict(terms=atm, **full)}
    kw = kw["rows" if form.startswith("rows") else "half" if form.startswith("half") else form]
    if form == "half_switch":
        kw["switch_width"] = 0.3
    cell = float(s.high[0]) / np.floor(float(s.high[0]) / 2.8)
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, cell, cutoff=2.5, cutoff_3b=2.0, nu=0.073, dt=0.001, **kw))
    g.update_container()
    g.forces()
    return g


def _without(s, r, gone):
    from komd_gb300 import lattice
    keep = np.arange(s.n) != gone
    return keep, lattice.System(r=r[keep], v=s.v[keep], m=s.m[keep], eps=s.eps[keep], sig=s.sig[keep],
                                mol_id=s.mol_id[keep], low=s.low, high=s.high)


def _off_the_cutoffs(s, r):
    """sites whose forces no pair within 5e-6 of a cutoff can change (the positions'
    FP32 roundings, 4 of two cell edges, may put it on either side)"""
    from scipy.spatial import cKDTree
    L = s.high - s.low
    q = np.mod(r - s.low, L)
    ok = np.ones(s.n, bool)
    tree = cKDTree(q, boxsize=L)
    for cut, reach in ((2.5, 0.0), (2.0, 2.1)):   # a triplet's third site is within the cutoff of both
        pairs = tree.query_pairs(cut + 5e-6, output_type="ndarray")
        d = q[pairs[:, 0]] - q[pairs[:, 1]]
        d -= L * np.round(d / L)
        for k in pairs[np.abs(np.linalg.norm(d, axis=1) - cut) < 5e-6].ravel():
            ok[tree.query_ball_point(q[k], reach)] = False
            ok[k] = False
    return ok


def _check(form, s, r, f, gone):
    keep, rest = _without(s, r, gone)
    ref = _engine(form, rest)
    fr = ref.download()[2]
    ref.close()
    assert np.isfinite(f[keep]).all()
    ok = _off_the_cutoffs(rest, rest.r)
    assert ok.mean() > 0.5
    d = np.abs(f[keep] - fr)[ok]
    assert np.sqrt((d ** 2).sum(1).mean() / (fr ** 2).sum(1).mean()) < FP32_FORCE_RMSE
    # nobody is off alone: 14 times the distance's error (4 roundings of two edges of 2.8)
    # over a distance of 0.9 in each of 12 close pairs of the largest force
    assert d.max() < 12 * 14 * (4 * 2.0 ** -24 * 5.6) / 0.9 * np.abs(fr).max()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("form", FORMS)
def test_other_sites_do_not_see_it(form, value):
    from komd_gb300 import gpu
    s = _system(form)
    gone = s.n // 2
    g = _engine(form, s)
    r, v, f = g.download()
    r[gone, 1] = value
    try:   # a step from the caller's positions: a Verlet list is not built again
        g.step_host(1, r, v, f)
    except gpu.KomdError as e:
        assert e.code == 6   # ERR_NONFINITE: the site's own velocity
    r, v, f = g.download()
    assert not np.isfinite(r[gone, 1]) and np.isfinite(np.delete(r, gone, 0)).all()
    _check(form, s, r, f, gone)
    g.set_state(r, v)      # and with the list built over it
    g.update_container()
    g.forces()
    r, v, f = g.download()
    _check(form, s, r, f, gone)
    g.close()
