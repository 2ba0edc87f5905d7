"""Performance cases of the engine: what its users have it do, through komd_gb300.gpu.

Each case is a production interval as a user's program runs it: some MD steps
from a prepared system, the observables of the interval and the state back on
the host.  The kinds:

  stock      KoMD's stock program: LJ + FENE + Limit (+ ATM with the reference's
             triplet set and sign), per-step cells, the velocity-scaling
             thermostat; per-call hooks as Simulation::run makes them, or whole
             intervals per call (`fused`)
  fp64       LJ (+ ATM) with FP64 forces on per-step cells: the reference's precision
  verlet     LJ (+ ATM) with FP32 forces on the Verlet list: production runs;
             `host`: state in the caller's buffers, one call per step;
             `switch`: the smooth cutoffs
  molecules  flexible 3-site molecules, bonds and angles, Verlet list
  ibi        the tabulated force of an IBI iteration with its RDF samples
  replicas   many small uneven systems advanced by one graph
  learned    LJ + the learned three-body term
  fit        force-matched training of that term

FP32 forces give trajectories of single precision, so those come back as
float32; positions and velocities are the state a run keeps (forces follow from
them).  FP64 runs return r, v and f as they are.
"""
import functools
import itertools
import math

import numpy as np
import torch

from komd_gb300 import gpu, lattice, surrogate

NU, RHO, T_STAR = 0.073, 0.8442, 0.722
T_KELVIN = T_STAR * lattice.T_STAR_TO_K
BOND = dict(bond_k=1000.0, bond_r0=1.0, angle_k=100.0, angle_theta0=math.radians(109.47))


def listed():
    return [
        # a small melt of FENE molecules in the stock program, a call per hook: latency and launches
        dict(name="stock_hooks_fene_1k5", kind="stock", n=1536, fene=True, atm=False, fused=False, steps=10),
        # the stock program on LJ + ATM argon (one cutoff of 2.0 for both, cells of 2.0)
        dict(name="stock_lj_atm_32k", kind="stock", n=32000, fene=False, atm=True, fused=True, steps=10),
        # the reference's precision, on its small plain-LJ system and on LJ + ATM
        dict(name="fp64_lj_4k", kind="fp64", n=4000, atm=False, steps=10),
        dict(name="fp64_lj_atm_32k", kind="fp64", n=32000, atm=True, steps=10),
        # FP32 production: the small system, where launches count, and the largest
        dict(name="verlet_lj_4k", kind="verlet", n=4000, atm=False, skin=0.3, switch=0.0, host=False, steps=100),
        dict(name="verlet_lj_atm_256k", kind="verlet", n=256000, atm=True, skin=0.6, switch=0.0, host=False, steps=50),
        # a program that keeps the state itself and calls once per step (odd count: vacancies in the lattice)
        dict(name="host_lj_atm_31k", kind="verlet", n=31013, atm=True, skin=0.4, switch=0.0, host=True, steps=20),
        # the multi-site workload
        dict(name="molecules_300k", kind="molecules", n=300000, skin=0.3, steps=20),
        # one IBI sampling interval
        dict(name="ibi_32k", kind="ibi", n=32000, nodes=200, steps=10),
        # a state-point scan: uneven boxes of 2000 to 20000 atoms
        dict(name="replicas_48", kind="replicas", count=48, boxes=2027, skin=0.3, steps=20),
        # the learned three-body term, run and trained
        dict(name="learned_32k", kind="learned", n=32000, skin=0.3, steps=20),
        dict(name="fit_120", kind="fit", snaps=120, batch=4, epochs=1),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stock", "stock", "fp64", "fp64", "verlet", "verlet", "verlet", "molecules", "ibi", "replicas",
                       "learned", "fit"])
    if kind == "stock":
        fene = rng.random() < 0.5
        n = 3 * _spread(rng, 150, 4000) if fene else _spread(rng, 1000, 32000)
        return dict(kind=kind, n=n, fene=fene, atm=not fene and rng.random() < 0.7, fused=rng.random() < 0.5, steps=10)
    if kind == "fp64":
        return dict(kind=kind, n=_spread(rng, 1000, 30000), atm=rng.random() < 0.6, steps=10)
    if kind == "verlet":
        return dict(kind=kind, n=_spread(rng, 2000, 250000), atm=rng.random() < 0.7, skin=rng.choice([0.3, 0.4, 0.6]),
                    switch=rng.choice([0.0, 0.0, 0.3]), host=rng.random() < 0.3, steps=20)
    if kind == "molecules":
        return dict(kind=kind, n=3 * _spread(rng, 3000, 90000), skin=rng.choice([0.3, 0.4]), steps=20)
    if kind == "ibi":
        return dict(kind=kind, n=_spread(rng, 1000, 31000), nodes=rng.choice([100, 200, 333]), steps=10)
    if kind == "replicas":
        return dict(kind=kind, count=rng.randint(3, 47), boxes=rng.randrange(1 << 30), skin=rng.choice([0.3, 0.4]), steps=20)
    if kind == "learned":
        return dict(kind=kind, n=_spread(rng, 2000, 31000), skin=rng.choice([0.3, 0.4]), steps=20)
    return dict(kind=kind, snaps=10 * rng.randint(2, 11), batch=rng.choice([2, 4]), epochs=1)


# ---- systems ---------------------------------------------------------------
def _argon(n, seed, rho=RHO, t_star=T_STAR):
    """n argon atoms on an FCC lattice with thermal displacements, trimmed to n by seed."""
    s = lattice.trimmed_fcc(n, rho, t_star, seed)
    rng = np.random.default_rng(seed + 1)
    s.r = np.mod(s.r + rng.normal(0.0, 0.04, s.r.shape), s.high)
    return s


def _fene_melt(n, seed):
    side = max(4, math.ceil((n / 3) ** (1 / 3) - 1e-9))
    s = lattice.triatomic_sc(side, rho_site=0.25, t_star=0.5, seed=seed, r0=0.97, theta0_deg=90.0)
    keep = min(n, s.n) // 3 * 3   # ragged: the last molecules of the lattice left out
    return lattice.System(r=s.r[:keep], v=s.v[:keep], m=s.m[:keep], eps=s.eps[:keep], sig=s.sig[:keep],
                          mol_id=s.mol_id[:keep], low=s.low, high=s.high)


def _cell(s, reach):
    side = float(np.min(s.high - s.low))
    return side / math.floor(side / reach)


def _system(case, seed):
    """The system and the engine configuration's keywords."""
    k = case["kind"]
    if k == "stock":
        s = _fene_melt(case["n"], seed) if case["fene"] else _argon(case["n"], seed)
        rc = 2.5 if case["fene"] else 2.0
        terms = gpu.TERM_LJ | gpu.TERM_FENE | gpu.TERM_LIMIT | (gpu.TERM_ATM if case["atm"] else 0)
        return s, dict(cell_size=rc, cutoff=rc, nu=NU, dt=0.002 if case["fene"] else 0.005, terms=terms, limit=20.0,
                       thermostat=1 if case["fused"] else 0, temperature_target=T_KELVIN)
    if k == "molecules":
        s = lattice.triatomic_count(case["n"] // 3, rho_site=0.8, t_star=1.0, seed=seed, aligned=True)
        return s, dict(cell_size=_cell(s, 4.5 + case["skin"]), cutoff=2.5, dt=0.002, skin=case["skin"],
                       terms=gpu.TERM_LJ | gpu.TERM_BONDED, virial_mode=gpu.VIRIAL_CORRECT, **BOND)
    s = _argon(case["n"], seed)
    if k == "ibi":
        return s, dict(cell_size=_cell(s, 2.5), cutoff=2.5, terms=gpu.TERM_TABULATED, precision=gpu.FP64)
    skin = case.get("skin", 0.0)
    terms = gpu.TERM_LJ | (gpu.TERM_ATM if k == "learned" or case["atm"] else 0)
    return s, dict(cell_size=_cell(s, 2.5 + skin), cutoff=2.5, cutoff_3b=2.0, nu=NU,
                   terms=terms | (gpu.TERM_ATM_SURROGATE if k == "learned" else 0),
                   precision=gpu.FP64 if k == "fp64" else gpu.FP32, skin=skin, switch_width=case.get("switch", 0.0),
                   atm_sign=gpu.ATM_SIGN_PHYSICAL, atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT)


def _replicas(case, seed):
    """The boxes (sizes and state points) are the case's; what is in them comes from the seed."""
    for k, (_, n, rho, t_star) in enumerate(lattice.replica_specs(case["count"], case["boxes"])):
        yield _argon(n, 1000 * seed + k, rho, t_star)


def _table(nodes):
    """An IBI force table: the LJ force on `nodes` nodes."""
    x = np.linspace(0.6, 2.5, nodes)
    return x, 24.0 * (2.0 * x ** -13 - x ** -7)


@functools.lru_cache(None)
def _model():
    """A network of the learned term with gentle forces (a step's cost does not depend on the weights)."""
    return dict(params=surrogate.init_params(1), fmean=np.full(gpu.SUR_NFEAT, 0.5, np.float32),
                fstd=np.full(gpu.SUR_NFEAT, 2.0, np.float32), e_scale=0.1, e_shift=0.0)


def _engine(s, kw, case):
    g = gpu.GpuSystem(s, gpu.make_config(s.low, s.high, **kw))
    if case["kind"] == "ibi":
        g.set_pair_table(*_table(case["nodes"]))
    if case["kind"] == "learned":
        g.surrogate_load(_model(), probe_every=0)
    g.update_container()
    g.forces()
    return g


def prepare(case, seed):
    k = case["kind"]
    if k == "fit":
        data = surrogate.capture(n_points=case["snaps"] // 10, snaps_per_point=10, ncell=5, equil=10, every=2,
                                 seed=seed)
        return dict(case=case, data=data, scale=surrogate.scaling(data), params=surrogate.init_params(seed))
    if k == "replicas":
        reps = [_engine(s, dict(cell_size=_cell(s, 2.5 + case["skin"]), cutoff=2.5, cutoff_3b=2.0, nu=NU,
                                terms=gpu.TERM_LJ | gpu.TERM_ATM, skin=case["skin"], atm_sign=gpu.ATM_SIGN_PHYSICAL,
                                atm_enum=gpu.ATM_ENUM_FULL, virial_mode=gpu.VIRIAL_CORRECT), case)
                for s in _replicas(case, seed)]
        return dict(case=case, reps=reps, batch=gpu.Batch(reps, n_streams=4, steps_per_graph=5))
    s, kw = _system(case, seed)
    st = dict(case=case, g=_engine(s, kw, case))
    if case.get("host"):   # the caller's own (pinned) state, as a coupled program keeps it
        st["buf"] = [torch.from_numpy(np.ascontiguousarray(x)).pin_memory().numpy()
                     for x in (s.r, s.v, np.zeros_like(s.r))]
    return st


# ---- one pass --------------------------------------------------------------
_SENSORS = gpu.MEASURE_TEMPERATURE | gpu.MEASURE_ENERGY | gpu.MEASURE_PRESSURE


def _state32(r, v):
    return {"r": r.astype(np.float32), "v": v.astype(np.float32)}


def _observed(o, atm):
    out = {"u_lj": o["u_lj"], "temperature": o["temperature"], "pressure": o["pressure"].astype(np.float32)}
    return dict(out, u_atm=o["u_atm"]) if atm else out


def run(state):
    case = state["case"]
    k, steps = case["kind"], case.get("steps")
    if k == "fit":
        c = state["scale"]
        p, loss = state["data"].fit(state["params"], c["fmean"], c["fstd"], c["e_scale"], c["e_shift"], c["f2"],
                                    case["epochs"], snaps_per_batch=case["batch"], lr=3e-3, lr_end=5e-5)
        return {"params": p, "loss": loss}
    if k == "replicas":
        b = state["batch"]
        b.step(steps // b.steps_per_graph)
        obs = b.measure(_SENSORS)
        down = [g.download() for g in state["reps"]]
        return dict(_state32(np.concatenate([d[0] for d in down]), np.concatenate([d[1] for d in down])),
                    u_lj=np.array([o["u_lj"] for o in obs], np.float32),
                    u_atm=np.array([o["u_atm"] for o in obs], np.float32))
    g = state["g"]
    if k == "stock":
        if case["fused"]:
            g.step(steps)
        else:   # Simulation::run's loop body, a call per hook
            for _ in range(steps):
                g.integrate0()
                g.update_container()
                g.forces()
                g.integrate1()
                g.scale_velocities(math.sqrt(T_KELVIN / g.measure(gpu.MEASURE_TEMPERATURE)["temperature"]))
        o = g.measure(_SENSORS)
        r, v, _ = g.download()
        return dict(_state32(r, v), **_observed(o, case["atm"]))
    if k == "ibi":
        rdf = np.zeros(100)
        for _ in range(steps // 5):   # the profiler samples every few steps
            g.step(5)
            rdf += g.rdf_profile(2.5, 100)
        r, v, f = g.download()
        return {"r": r, "v": v, "f": f, "rdf": rdf}
    if case.get("host"):
        r, v, f = state["buf"]
        for _ in range(steps):
            g.step_host(1, r, v, f)
        return _state32(r, v)
    g.step(steps)
    if k == "learned":
        return _state32(*g.download()[:2])
    o = g.measure(_SENSORS)
    r, v, f = g.download()
    if k == "fp64":
        return {"r": r, "v": v, "f": f, "u_lj": o["u_lj"], "pressure": o["pressure"]}
    return dict(_state32(r, v), **_observed(o, case.get("atm")))


def work(case):
    """The state in and out once, 40 operations a pair and 200 a triplet (the reference's formulation)."""
    k = case["kind"]
    if k == "fit":   # network forward, backward and weight gradients, and two passes over 27 neighbours a site
        n = 500 * case["snaps"] * case["epochs"]
        return {"bytes": n * (27 * 16 + 4 * 72), "flops": n * (6 * 2 * 6144 + 27 * 4 * 260)}
    n = 11000 * case["count"] if k == "replicas" else case["n"]
    rho = {"molecules": 0.8}.get(k, 0.25 if case.get("fene") else RHO)
    rc = 2.0 if k == "stock" and not case["fene"] else 2.5
    pairs = n * rho * 2.094 * rc ** 3
    atm = k in ("replicas", "learned") or case.get("atm")
    per_step = 40 * pairs + (200 * 41 * n if atm else 0)
    return {"bytes": n * 120.0, "flops": case["steps"] * float(per_step)}


# ---- 64 bits ---------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cells_of(x, low, L, nd, cs):
    """Cell of each position: edges cs, the last cell stretched (clamped)."""
    q = torch.floor((x - low) / cs).long()
    q = torch.minimum(q.clamp(min=0), torch.tensor(nd, device=x.device) - 1)
    return q[:, 0] + nd[0] * (q[:, 1] + nd[1] * q[:, 2])


def _pairs(r, cell, nd, L, rmax):
    """Every pair of sites in adjacent (periodic) cells with r2 <= rmax^2, once:
    i, j and r_i - r_j through the cells' periodic shift."""
    dev, n = r.device, r.shape[0]
    ncell = nd[0] * nd[1] * nd[2]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    slot = torch.empty_like(order)
    slot[order] = torch.arange(n, device=dev)
    c3 = torch.stack([cell % nd[0], (cell // nd[0]) % nd[1], cell // (nd[0] * nd[1])], 1)
    out = []
    for off in itertools.product((-1, 0, 1), repeat=3):
        if off < (0, 0, 0):
            continue
        q = c3 + torch.tensor(off, device=dev)
        ndt = torch.tensor(nd, device=dev)
        shift = torch.where(q < 0, -L, torch.where(q >= ndt, L, torch.zeros_like(L)))
        q = q % ndt
        qc = q[:, 0] + nd[0] * (q[:, 1] + nd[1] * q[:, 2])
        m = count[qc]
        i = torch.repeat_interleave(torch.arange(n, device=dev), m)
        first = torch.cumsum(m, 0) - m
        js = start[qc][i] + torch.arange(i.shape[0], device=dev) - first[i]
        if off == (0, 0, 0):
            keep = js > slot[i]
            i, js = i[keep], js[keep]
        j = order[js]
        d = r[i] - (r[j] + shift[i])
        keep = (d * d).sum(1) <= rmax * rmax
        out.append((i[keep], j[keep], d[keep]))
    return [torch.cat(t) for t in zip(*out)]


def _smooth(x, rc, width):
    """The smooth cutoff's S and dS/dx at squared distance x."""
    if not width:
        return torch.ones_like(x), torch.zeros_like(x)
    iw = 1.0 / (rc * rc - (rc - width) ** 2)
    t = ((rc * rc - x) * iw).clamp(0, 1)
    return t * t * (3 - 2 * t), -6 * t * (1 - t) * iw


def _outer(w, d):
    """sum w d (x) d: XX XY YY XZ YZ ZZ."""
    return torch.stack([(w * d[:, a] * d[:, b]).sum() for a, b in ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))])


def _atm(i, j, d, n, rc, nu, width, allowed=None):
    """V, forces -grad V and virial of the triplets with all sides inside rc (allowed: a filter on the three sites)."""
    near = (d * d).sum(1) <= rc * rc
    i, j, d = i[near], j[near], d[near]
    # each triplet from the vertex that owns two of its sides: sides as directed pairs low -> high
    swap = i > j
    i, j, d = torch.where(swap, j, i), torch.where(swap, i, j), torch.where(swap[:, None], -d, d)
    order = torch.argsort(i, stable=True)
    i, j, d = i[order], j[order], d[order]
    cnt = torch.bincount(i, minlength=n)
    end = torch.cumsum(cnt, 0)
    p = torch.arange(i.shape[0], device=i.device)
    rest = end[i] - p - 1                       # later pairs of the same vertex
    a = torch.repeat_interleave(p, rest)
    b = a + 1 + torch.arange(a.shape[0], device=i.device) - (torch.cumsum(rest, 0) - rest)[a]
    c = d[b] - d[a]                             # r_ja - r_jb
    keep = (c * c).sum(1) <= rc * rc
    if allowed is not None:
        keep &= allowed(i[a], j[a], j[b])
    a, b, c = a[keep], b[keep], c[keep]
    A, B, C = (d[a] ** 2).sum(1), (d[b] ** 2).sum(1), (c * c).sum(1)
    s2 = 1.0 / (A * B * C)
    s = torch.sqrt(s2)
    t1, t2, t3 = A + B - C, A - B + C, B + C - A
    P = t1 * t2 * t3
    s5 = s2 * s2 * s
    V = nu * (s2 * s + 0.375 * P * s5)
    dP = (-t1 * t2 + t1 * t3 + t2 * t3, t1 * t2 - t1 * t3 + t2 * t3, t1 * t2 + t1 * t3 - t2 * t3)
    g = [nu * s5 * (0.375 * dP[q] - 1.5 * other - 0.9375 * P / X) for q, (X, other) in
         enumerate(((A, B * C), (B, A * C), (C, A * B)))]
    if width:
        S = [_smooth(X, rc, width) for X in (A, B, C)]
        g = [(g[q] * S[q][0] + V * S[q][1]) * S[(q + 1) % 3][0] * S[(q + 2) % 3][0] for q in range(3)]
        V = V * S[0][0] * S[1][0] * S[2][0]
    f = torch.zeros(n, 3, dtype=d.dtype, device=d.device)
    fa, fb, fc = -2 * g[0][:, None] * d[a], -2 * g[1][:, None] * d[b], -2 * g[2][:, None] * c
    f.index_add_(0, i[a], fa + fb)
    f.index_add_(0, j[a], fc - fa)
    f.index_add_(0, j[b], -fc - fb)
    vir = _outer(-2 * g[0], d[a]) + _outer(-2 * g[1], d[b]) + _outer(-2 * g[2], c)
    return V.sum(), f, vir


def _learned(i, j, d, n, rc, model):
    """Energy and forces of the learned three-body term."""
    near = (d * d).sum(1) < rc * rc
    i, j, d = i[near], j[near], d[near]
    i, j, d = torch.cat([i, j]), torch.cat([j, i]), torch.cat([-d, d]).requires_grad_()   # d = r_j - r_i
    r = torch.sqrt((d * d).sum(1))
    u, fc = d / r[:, None], 0.5 * (torch.cos(math.pi * r / rc) + 1)
    one = dict(dtype=d.dtype, device=d.device)
    mu = 0.85 + torch.arange(16, **one) * (1.15 / 15)
    G = torch.exp(-50.0 * (r[:, None] - mu) ** 2) * fc[:, None]
    feats = [torch.zeros(n, 16, **one).index_add(0, i, G)]
    inv = [[], [], [], []]
    for c in range(4):
        gc = (torch.exp(-(r - (1.05 + 0.25 * c)) ** 2 / (2 * 0.15 ** 2)) * fc)[:, None] * u
        m1 = torch.zeros(n, 3, **one).index_add(0, i, gc)
        m2 = torch.zeros(n, 9, **one).index_add(0, i, (gc[:, :, None] * u[:, None, :]).reshape(-1, 9)).view(n, 3, 3)
        inv[0].append((m1 * m1).sum(1))
        inv[1].append((m2 * m2).sum((1, 2)))
        inv[2].append(torch.einsum("ni,nij,nj->n", m1, m2, m1))
        inv[3].append(torch.einsum("nij,njk,nki->n", m2, m2, m2))
    x = torch.cat(feats + [torch.stack(q, 1) for q in inv], 1)
    p = torch.tensor(model["params"], **one)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [2048, 64, 4096, 64, 64, 1])
    x = (x - torch.tensor(model["fmean"], **one)) / torch.tensor(model["fstd"], **one)
    h = torch.tanh(torch.tanh(x @ w1.view(64, 32).T + b1) @ w2.view(64, 64).T + b2)
    E = (model["e_scale"] * (h @ w3 + b3) + model["e_shift"]).sum()
    g, = torch.autograd.grad(E, d)
    f = torch.zeros(n, 3, **one)
    f.index_add_(0, i, g)
    f.index_add_(0, j, -g)
    return E.detach(), f


class _Exact:
    """The same system, stepped in 64 bits."""

    def __init__(self, s, kw, case):
        def t(x):
            return torch.as_tensor(np.asarray(x), device=_dev())
        self.kw, self.case, self.n = kw, case, s.n
        self.r, self.v = t(s.r).clone(), t(s.v).clone()
        self.low, self.L = t(s.low), t(s.high - s.low)
        _, mol = np.unique(s.mol_id, return_inverse=True)
        self.mol, self.single = t(mol), s.n == mol.max() + 1
        self.size = torch.bincount(self.mol).double()
        self.bonds, self.angles = t(s.bonds), t(s.angles)
        self.terms = kw["terms"]
        self.forces()

    def _com(self):
        z = torch.zeros(self.size.shape[0], 3, dtype=torch.float64, device=self.r.device)
        return z.index_add_(0, self.mol, self.r) / self.size[:, None]

    def _wrap(self):
        com = self._com()
        off = torch.where(com < self.low, self.L, torch.where(com > self.low + self.L, -self.L, torch.zeros_like(com)))
        self.r = self.r + off[self.mol]

    def forces(self):
        self._wrap()
        kw, n = self.kw, self.n
        listed_cells = not self.single and not kw.get("skin")   # molecules by their centre, as the cells bin them
        cs = kw["cell_size"] if self.single or listed_cells else kw["cutoff"]
        Lh = [float(x) for x in self.L]
        nd = [int(math.floor(x / cs)) for x in Lh]
        if listed_cells or self.single:
            pos, r = self._com()[self.mol], self.r
        else:
            r = self.low + torch.remainder(self.r - self.low, self.L)
            pos, cs = r, Lh[0] / nd[0]
        cell = _cells_of(pos, self.low, self.L, nd, cs)
        reach = kw["cutoff"]
        width = kw.get("switch_width", 0.0)
        i, j, d = _pairs(r, cell, nd, self.L, reach)
        r2 = (d * d).sum(1)
        f = torch.zeros_like(self.r)
        self.u_lj = self.u_atm = torch.zeros((), dtype=torch.float64)
        self.w = torch.zeros(6, dtype=torch.float64, device=r.device)

        def add(i, j, fp):
            f.index_add_(0, i, fp)
            f.index_add_(0, j, -fp)
        if self.terms & gpu.TERM_LJ:
            other = self.mol[i] != self.mol[j]
            li, lj, ld, x = i[other], j[other], d[other], r2[other]
            s6 = x ** -3
            u, fac = 4 * (s6 * s6 - s6), 24 * (2 * s6 * s6 - s6) / x
            S, dS = _smooth(x, reach, width)
            fac, u = fac * S - 2 * u * dS, u * S
            add(li, lj, ld * fac[:, None])
            self.u_lj = u.sum()
            self.w = self.w + _outer(fac, ld)
        if self.terms & gpu.TERM_FENE and not self.single:   # every pair of a molecule, no cutoff
            a, b = np.triu_indices(3, 1)
            base = torch.arange(0, n, 3, device=r.device)[:, None]
            fi, fj = (base + torch.as_tensor(a, device=r.device)).reshape(-1), (base + torch.as_tensor(b, device=r.device)).reshape(-1)
            fd = self.r[fi] - self.r[fj]
            q = (fd * fd).sum(1, keepdim=True) / 2.25
            add(fi, fj, torch.where(q >= 1, -1e30 / fd, -fd * 30.0 / (1 - q)))
        if self.terms & gpu.TERM_TABULATED:
            x, y = (torch.as_tensor(t, device=r.device) for t in _table(self.case["nodes"]))
            rr = torch.sqrt(r2)
            k = (torch.searchsorted(x, rr) - 1).clamp(0, x.shape[0] - 2)
            F = y[k] + (y[k + 1] - y[k]) / (x[k + 1] - x[k]) * (rr - x[k])
            F = torch.where(rr > x[-1], torch.zeros_like(F), torch.where(rr < x[0], torch.full_like(F, 1e6), F))
            add(i, j, d / rr[:, None] * F[:, None])
        if self.terms & gpu.TERM_BONDED:
            a, b = self.bonds[:, 0], self.bonds[:, 1]
            bd = self.r[a] - self.r[b]
            l = torch.sqrt((bd * bd).sum(1))
            fs = -kw["bond_k"] * (l - kw["bond_r0"]) / l
            add(a, b, bd * fs[:, None])
            self.w = self.w + _outer(fs, bd)
            a, c, b = self.angles.T
            u, w = self.r[a] - self.r[c], self.r[b] - self.r[c]
            iu, iw = (u * u).sum(1) ** -0.5, (w * w).sum(1) ** -0.5
            cs_ = (u * w).sum(1) * iu * iw
            pre = kw["angle_k"] * (torch.arccos(cs_) - kw["angle_theta0"]) / torch.sqrt(1 - cs_ * cs_)
            fu = pre[:, None] * (w * (iu * iw)[:, None] - u * (cs_ * iu * iu)[:, None])
            fw = pre[:, None] * (u * (iu * iw)[:, None] - w * (cs_ * iw * iw)[:, None])
            add(a, c, fu)
            add(b, c, fw)
            self.w = self.w + torch.stack([(u[:, p] * fu[:, q] + w[:, p] * fw[:, q]).sum()
                                           for p, q in ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))])
        if self.terms & gpu.TERM_LIMIT:
            f = f.clamp(-kw["limit"], kw["limit"])
        if self.terms & gpu.TERM_ATM_SURROGATE:
            f = f + _learned(i, j, d, n, kw["cutoff_3b"], _model())[1]
        elif self.terms & gpu.TERM_ATM:
            stock = self.case["kind"] == "stock"

            def allowed(a, b, c):   # the reference's triplets: the three cells all equal or all distinct
                x, y, z = cell[a], cell[b], cell[c]
                return ((x == y) & (y == z)) | ((x != y) & (y != z) & (x != z))
            self.u_atm, fa, wa = _atm(i, j, d, n, kw.get("cutoff_3b") or kw["cutoff"], kw["nu"], width,
                                      allowed if stock else None)
            f = f + (-fa if stock else fa)   # the stock program adds +grad V
            self.w = self.w + wa
        self.f = f

    def temperature(self):
        inside = ((self.r >= self.low) & (self.r <= self.low + self.L)).all(1)   # the sensor's sites
        return float((self.v[inside] ** 2).sum()) / (3 * int(inside.sum())) * lattice.T_STAR_TO_K

    def step(self, count):
        dt = self.kw.get("dt", 0.005)
        for _ in range(count):
            self.v = self.v + self.f * (0.5 * dt)
            self.r = self.r + self.v * dt
            self.forces()
            self.v = self.v + self.f * (0.5 * dt)
            if self.case["kind"] == "stock":
                self.v = self.v * math.sqrt(T_KELVIN / self.temperature())

    def pressure(self):
        return (_outer(torch.ones(self.n, dtype=torch.float64, device=self.r.device), self.v) + self.w).cpu().numpy()

    def rdf(self):
        """Ordered pairs in 100 bins to 2.5."""
        com = self.r
        nd = [int(math.floor(float(x) / 2.5)) for x in self.L]
        cell = _cells_of(com, self.low, self.L, nd, self.kw["cell_size"])
        d = _pairs(com, cell, nd, self.L, 2.5)[2]
        b = torch.floor(torch.sqrt((d * d).sum(1)) / 0.025).long().clamp(max=99)
        return 2.0 * torch.bincount(b, minlength=100).double().cpu().numpy()


def exact(case, seed):
    k = case["kind"]
    if k == "fit":   # an epoch of Adam on tensor-core gradients has no short restatement
        return None
    if k == "replicas":
        kw = dict(cutoff=2.5, cutoff_3b=2.0, nu=NU, terms=gpu.TERM_LJ | gpu.TERM_ATM, skin=case["skin"])
        r, v, u, ua = [], [], [], []
        for s in _replicas(case, seed):
            e = _Exact(s, dict(kw, cell_size=_cell(s, 2.5)), case)
            e.step(case["steps"])
            r.append(e.r.cpu().numpy())
            v.append(e.v.cpu().numpy())
            u.append(float(e.u_lj))
            ua.append(float(e.u_atm))
        return {"r": np.concatenate(r), "v": np.concatenate(v), "u_lj": np.array(u), "u_atm": np.array(ua)}
    s, kw = _system(case, seed)
    e = _Exact(s, kw, case)
    if k == "ibi":
        rdf = np.zeros(100)
        for _ in range(case["steps"] // 5):
            e.step(5)
            rdf += e.rdf()
        return {"r": e.r.cpu().numpy(), "v": e.v.cpu().numpy(), "f": e.f.cpu().numpy(), "rdf": rdf}
    e.step(case["steps"])
    out = {"r": e.r.cpu().numpy(), "v": e.v.cpu().numpy()}
    if k == "learned" or case.get("host"):
        return out
    u = {"u_lj": float(e.u_lj), "pressure": None if k == "stock" else e.pressure()}
    if k == "fp64":
        return dict(out, f=e.f.cpu().numpy(), **u)
    return dict(out, temperature=e.temperature(), **u, **({"u_atm": float(e.u_atm)} if case.get("atm") else {}))
