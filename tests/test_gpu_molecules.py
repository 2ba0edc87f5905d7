"""Molecules of several sites on the device: bonded forces molecule by molecule, and
the wrap on steps that keep the cells, where an FP32 estimate of the centre of
mass decides which molecules need the FP64 one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _reference(r, bonds, angles, kb, r0, ka, th0):
    """FP64 forces, and a bound per site on the FP32 evaluation's error: each term's
    differences, norms and products are within 32 roundings of its force scale
    (kb (r + r0); ka pi / sin(theta) (1/|u| + 1/|v|)), the angle's conditioned by
    1 / sin(theta)^2."""
    f, tol = np.zeros_like(r), np.zeros(len(r))
    for i, j in bonds:
        d = r[i] - r[j]
        q = np.linalg.norm(d)
        g = -kb * (q - r0) / q * d
        f[i] += g
        f[j] -= g
        tol[[i, j]] += 32 * EPS * kb * (q + r0)
    for i, j, k in angles:
        u, v = r[i] - r[j], r[k] - r[j]
        nu, nv = np.linalg.norm(u), np.linalg.norm(v)
        cs = u @ v / (nu * nv)
        sn = np.sqrt(1 - cs * cs)
        pre = ka * (np.arccos(cs) - th0) / sn
        fi = pre * (v / (nu * nv) - cs * u / nu ** 2)
        fk = pre * (u / (nu * nv) - cs * v / nv ** 2)
        f[i] += fi
        f[k] += fk
        f[j] -= fi + fk
        tol[[i, j, k]] += 32 * EPS * ka * np.pi / sn ** 3 * (1 / nu + 1 / nv)
    return f, tol


def _graph(form, n, rng):
    """pairs of bonded sites and chains' angles of n sites"""
    if form == "random":                  # one component, terms given twice
        bonds = [tuple(rng.choice(n, 2, replace=False)) for _ in range(200)]
        return bonds + [bonds[0][::-1]], [tuple(rng.choice(n, 3, replace=False)) for _ in range(90)]
    if form == "interleaved":             # small components whose ranges overlap
        return [(k, k + n // 2) for k in range(n // 2)], []
    if form == "one_bond":
        return [(n - 1, n - 2)], []
    if form == "one_angle":
        return [], [(2, 0, 1)]
    size = {"pairs": 2, "triples": 3, "nines": 9, "tens": 10}[form]   # 17 terms a component of ten: one too many
    runs = [np.arange(k, k + size) for k in range(1, n - size, size + (size == 3))]   # triples: a free site between
    bonds = [(x[q + 1], x[q]) for x in runs for q in range(size - 1)]
    return bonds, [(x[q], x[q + 1], x[q + 2]) for x in runs for q in range(size - 2)]


@pytest.mark.parametrize("form", ["one_bond", "one_angle", "pairs", "triples", "nines", "tens", "interleaved",
                                  "random"])
def test_bonded_forces_of_any_graph(form):
    from komd_gb300 import gpu, lattice
    s = lattice.argon_fcc(5, rho=0.4, t_star=1.0, seed=2, jitter=0.1)
    bonds, angles = _graph(form, s.n, np.random.default_rng(3))
    bonds = np.array(bonds, np.int64).reshape(-1, 2)

    def bent(i, j, k):
        u, v = s.r[i] - s.r[j], s.r[k] - s.r[j]
        return np.linalg.norm(np.cross(u, v)) > 0.4 * np.linalg.norm(u) * np.linalg.norm(v)
    angles = np.array([t for t in angles if bent(*t)], np.int64).reshape(-1, 3)
    s.bonds, s.angles = bonds, angles
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, float(s.high[0]) / 3, cutoff=1.0, terms=gpu.TERM_BONDED,
                                         bond_k=80.0, bond_r0=1.1, angle_k=30.0, angle_theta0=1.9))
    g.update_container()
    g.forces()
    r, _, f = g.download()
    ref, tol = _reference(r, bonds, angles, 80.0, 1.1, 30.0, 1.9)
    assert (np.abs(f - ref).max(1) <= tol).all()
    g.close()


@pytest.mark.parametrize("sites", [1, 3, 5])
def test_wrap_at_the_faces_without_a_rebuild(sites):
    """centres of mass that come to lie within 1e-10 to 1e-3 of a face, on both sides: each
    is inside the domain after the step, and moved by whole box lengths only"""
    from komd_gb300 import gpu, lattice
    n_mol, L, dt = 96, 24.0, 1e-3
    rng = np.random.default_rng(sites)
    n = n_mol * sites
    m = rng.uniform(0.7, 2.3, n)
    mol = np.repeat(np.arange(n_mol), sites).astype(np.uint64)
    com = np.stack(np.meshgrid(*[np.arange(5) * 4.0 + 4.0] * 3), -1).reshape(-1, 3)[:n_mol] + rng.uniform(-1, 1, (n_mol, 3))
    off = rng.uniform(-0.4, 0.4, (n_mol, sites, 3))
    mm = m.reshape(n_mol, sites, 1)
    off -= (off * mm).sum(1, keepdims=True) / mm.sum(1, keepdims=True)
    gap = np.where(rng.random(n_mol) < 0.5, -1, 1) * 10.0 ** rng.uniform(-10, -3, n_mol)
    com[np.arange(n_mol), np.arange(n_mol) % 3] = np.where(np.arange(n_mol) % 2, L, 0.0) + gap
    v = np.repeat(rng.uniform(-1, 1, (n_mol, 3)), sites, 0)
    r = (com[:, None, :] + off).reshape(n, 3) - v * dt
    s = lattice.System(r=r, v=v, m=m, eps=np.full(n, 1e-12), sig=np.full(n, 0.05), mol_id=mol, low=np.zeros(3),
                       high=np.full(3, L))
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, 4.0, cutoff=0.06, terms=gpu.TERM_LJ, dt=dt, skin=1.0,
                                         virial_mode=gpu.VIRIAL_CORRECT))
    g.update_container()
    g.forces()
    g.step(1)
    a = g.download()[0]
    got = np.zeros((n_mol, 3))
    for q in range(sites):
        got += a[q::sites] * m[q::sites, None]
    tot = m[0::sites].copy()
    for q in range(1, sites):
        tot = tot + m[q::sites]
    got /= tot[:, None]
    assert ((got >= 0.0) & (got <= L)).all()
    free = r + v * dt
    k = np.round((a - free) / L)
    assert np.abs(a - free - k * L).max() < 1e-12
    assert (k != 0).any() and (np.abs(k) <= 1).all()
    g.close()


@pytest.mark.parametrize("bonded", [False, True])
def test_steps_without_a_pair_term(bonded):
    """the forces start from a clearing, not from a pair kernel, in every step"""
    from komd_gb300 import gpu, lattice
    s = lattice.argon_fcc(3, rho=0.4, t_star=1.0, seed=2, jitter=0.1)
    if bonded:
        s.bonds = np.array([(k, k + 1) for k in range(0, s.n, 2)], np.int64)
    cfg = gpu.make_config(s.low, s.high, float(s.high[0]) / 3, cutoff=1.0, terms=gpu.TERM_BONDED, dt=1e-3,
                          bond_k=80.0, bond_r0=1.1, angle_k=30.0, angle_theta0=1.9)
    a, b = gpu.GpuSystem(s, cfg), gpu.GpuSystem(s, cfg)
    for g in (a, b):
        g.update_container()
        g.forces()
    a.step(9)
    for _ in range(9):
        b.step(1)
    for x, y in zip(a.download(), b.download()):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    assert np.any(a.download()[2]) == bonded
    a.close()
    b.close()
