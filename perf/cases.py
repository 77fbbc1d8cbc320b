"""Performance cases of the framework: what its users have it do, through its
public entry points (gomc_gb300.engine).

Each case is one kind of call at one size:

  move      one proposed molecule move scored through the reference-shaped
            interfaces (MoleculeInter, MolReciprocal): the smallest call
  trials    one CBMC trial set of a Lennard-Jones particle (RemoveMol,
            ParticleInter, AddMol)
  chain     a segment of one translate/rotate Markov chain on the device
  replicas  a segment of many chains batched on one GPU, mixed precision
  mp        a segment with the MultiParticle move in the mix
  gemc      a segment of the two-box Gibbs-ensemble run
  forces    forces, reciprocal sums and energy, torques (MultiParticle::CalcEn)
  total     SystemTotal: every energy term of a box from its coordinates
  volume    the energies of a trial volume (VolumeTransfer::CalcEn)
  virial    the pressure's virial

Systems are the repository's own: SPC/E-geometry waters at 1 g/cm^3 on a
seeded lattice (256 to 20,000 molecules, Rcut 9 or 10 A, Ewald tolerance
1e-5) and single-site LJ spheres (sigma 3.73 A, epsilon 148 K, Rcut 12 A).
"""
import math

import numpy as np
import torch

from gomc_gb300 import engine
from gomc_gb300.config import SimConfig
from gomc_gb300.systems import (lj_sphere_box, spce_water_box,
                                water_box_length)

TEMP, TOL = 298.0, 1e-5
SCALES = (0.3, 0.3, 0.02, 0.01 * math.pi)
LJ_EPS, LJ_SIG, LJ_RCUT = 148.0, 3.73, 12.0
QQ = 167103.208067979  # e^2 / (4 pi eps0 kB A) in K


def listed():
    return [
        # a host program that keeps its own move loop scores one move per
        # call on the 256-water configuration: latency and launches
        dict(name="move_w256", kind="move", n=256, rcut=9.0),
        # one CBMC first-atom trial set (CBMC_First 10) in the 2,400-sphere
        # liquid box of the Gibbs-ensemble configuration
        dict(name="trials_lj2400", kind="trials", n=2400, trials=10),
        # the 256-water FP64 configuration run on the device, and the
        # 8,000-water system that the headline metric is quoted on
        dict(name="chain_w256", kind="chain", n=256, rcut=9.0, moves=1000),
        dict(name="chain_w8000", kind="chain", n=8000, rcut=10.0, moves=500),
        # mixed precision: replicas of the 8,000-water system that fill the
        # GPU, and jobs of uneven size as a serving round holds them
        dict(name="replicas_36x8000", kind="replicas", lo=8000, hi=8000,
             count=36, cluster=8, rcut=10.0, moves=100),
        dict(name="replicas_uneven12", kind="replicas", lo=500, hi=20000,
             count=12, cluster=0, rcut=9.0, moves=100),
        # translate / rotate / MultiParticle 0.495 / 0.495 / 0.01
        dict(name="mp_w8000", kind="mp", n=8000, rcut=10.0, moves=1000),
        # Gibbs-ensemble NVT of 2,400 + 300 LJ spheres, FP64
        dict(name="gemc_lj2700", kind="gemc", n0=2400, n1=300, l0=40.0,
             l1=90.0, mixed=False, moves=1000),
        # a host-side MultiParticle move: forces and torques of one state
        dict(name="forces_w8000", kind="forces", n=8000, rcut=10.0),
        # the energy check of the largest box a job may have
        dict(name="total_w20000", kind="total", n=20000, rcut=10.0),
        # a volume move of an odd-sized box
        dict(name="volume_w2001", kind="volume", n=2001, rcut=9.0,
             scale=1.013),
        # a pressure sample of the headline system
        dict(name="virial_w8000", kind="virial", n=8000, rcut=10.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["move", "trials", "chain", "replicas", "mp", "gemc",
                       "forces", "total", "volume", "virial"])
    rcut = rng.choice([9.0, 9.5, 10.0])
    if kind == "move":
        return dict(kind=kind, n=_log_int(rng, 256, 8000), rcut=rcut)
    if kind == "trials":
        return dict(kind=kind, n=_log_int(rng, 300, 2400),
                    trials=_log_int(rng, 4, 200))
    if kind == "chain":
        return dict(kind=kind, n=_log_int(rng, 256, 8000), rcut=rcut,
                    moves=rng.randrange(100, 500))
    if kind == "replicas":
        lo = _log_int(rng, 500, 4000)
        return dict(kind=kind, lo=lo, hi=rng.randrange(lo, 8000),
                    count=rng.randrange(2, 17), cluster=0, rcut=rcut,
                    moves=rng.randrange(50, 100))
    if kind == "mp":
        return dict(kind=kind, n=_log_int(rng, 256, 8000), rcut=rcut,
                    moves=rng.randrange(500, 1000))
    if kind == "gemc":
        return dict(kind=kind, n0=rng.randrange(1600, 2400),
                    n1=rng.randrange(100, 300), l0=40.0,
                    l1=round(rng.uniform(70.0, 90.0), 2),
                    mixed=rng.random() < 0.5, moves=rng.randrange(200, 1000))
    if kind == "volume":
        return dict(kind=kind, n=_log_int(rng, 256, 8000), rcut=rcut,
                    scale=round(rng.uniform(0.985, 1.015), 4))
    hi = 20000 if kind == "total" else 8000
    return dict(kind=kind, n=_log_int(rng, 256, hi), rcut=rcut)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _edge(n):
    """Edge of n waters at 1 g/cm^3 (19.7 A for 256, 62.1 A for 8,000)."""
    return round(water_box_length(n), 1)


def _water(n, seed):
    """Seeded-lattice waters, each molecule displaced by up to 0.3 A."""
    s = spce_water_box(n, _edge(n), seed=seed)
    rng = np.random.default_rng(seed + 1)
    s.pos[:] = np.mod(s.pos + np.repeat(rng.uniform(-0.3, 0.3, (n, 3)), 3, 0),
                      s.box[0])
    return s


def _cfg(case):
    return SimConfig(temperature=TEMP, rcut=case["rcut"], tolerance=TOL)


def _lj(n, edge, seed):
    # non-overlapping at any fill of the boxes above
    return lj_sphere_box(n, edge, seed=seed, epsilon=LJ_EPS, sigma=LJ_SIG,
                         min_sep=2.4, name="LJ")


def _lj_edge(n):
    return round(40.0 * (n / 2400.0) ** (1.0 / 3.0), 2) if n > 900 else 30.0


def _sizes(case):
    lo, hi, c = case["lo"], case["hi"], case["count"]
    return [int(round(lo * (hi / lo) ** (i / max(c - 1, 1))))
            for i in range(c)]


def _cluster(n, rcut):
    """CTAs per chain as the job server picks them (2,048 k-vectors each)."""
    k = _k_count(_edge(n), rcut)
    return next((c for c in (2, 4, 8) if k <= 2048 * c), 16)


def _proposal(s, seed):
    """A displaced, rotated copy of one molecule."""
    rng = np.random.default_rng(seed + 2)
    m = int(rng.integers(s.n_mol))
    L = s.box[0]
    p = s.pos[3 * m:3 * m + 3]
    p = p[0] + (p - p[0] - L * np.round((p - p[0]) / L))
    c = p.mean(0)
    a = rng.uniform(-0.3, 0.3)
    rot = np.array([[math.cos(a), -math.sin(a), 0.0],
                    [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])
    return m, np.mod((p - c) @ rot.T + c + rng.uniform(-0.3, 0.3, 3), L)


def _trial_set(case, s, seed):
    rng = np.random.default_rng(seed + 3)
    return int(rng.integers(s.n_mol)), rng.random((case["trials"], 3)) * s.box


def _scaled(case, s):
    """Molecules moved with their first atoms to an edge scaled by `scale`."""
    L = s.box[0]
    L2 = L * case["scale"]
    p = s.pos.reshape(-1, 3, 3)
    d = p - p[:, :1]
    d -= L * np.round(d / L)
    q = np.mod(p[:, :1] * case["scale"] + d, L2).reshape(-1, 3)
    q[q >= L2] = 0.0
    return np.array([L2] * 3), q


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gemc":
        s0 = _lj(case["n0"], case["l0"], seed)
        s1 = _lj(case["n1"], case["l1"], seed + 7)
        g = engine.Gemc(s0.pos, s1.pos, s0.box, s1.box, LJ_EPS, LJ_SIG, 12.0,
                        150.0, LJ_RCUT, seed & 0xFFFFFFF, (0.8, 0.01, 0.19),
                        100, 10, precision=int(case["mixed"]))
        return dict(case=case, gemc=g)
    if kind == "replicas":
        boxes, same = [], None
        for i, n in enumerate(_sizes(case)):
            # equal replicas start from one configuration
            if same is None or n != same.n_mol:
                same = _water(n, seed + i)
            b = engine.Box(same, _cfg(case), precision=engine.GB_MIXED)
            b.mc_init((seed + i) & 0xFFFFFFF, (0.5, 0.5, 0.0), 1000,
                      scales=SCALES, recompute_freq=10000,
                      cluster_size=case["cluster"] or _cluster(n, case["rcut"]))
            boxes.append(b)
        return dict(case=case, boxes=boxes, step=0)
    if kind == "trials":
        s = _lj(case["n"], _lj_edge(case["n"]), seed)
        cfg = SimConfig(temperature=150.0, rcut=LJ_RCUT, ewald=False,
                        electrostatic=False)
        m, trials = _trial_set(case, s, seed)
        return dict(case=case, box=engine.Box(s, cfg), mol=m, trials=trials)
    s = _water(case["n"], seed)
    box = engine.Box(s, _cfg(case))
    st = dict(case=case, box=box, step=0)
    if kind in ("chain", "mp"):
        frac = (0.5, 0.5, 0.0) if kind == "chain" else (0.495, 0.495, 0.01)
        box.mc_init(seed & 0xFFFFFFF, frac, 1000, scales=SCALES)
    elif kind == "move":
        st["mol"], st["new"] = _proposal(s, seed)
        st["en"], st["ew"] = engine.CalculateEnergy(box), engine.Ewald(box)
    elif kind == "volume":
        st["edges"], st["xyz"] = _scaled(case, s)
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "gemc":
        g = st["gemc"]
        g.run(case["moves"])
        s = g.state()
        xyz, com, lookup = g.coords()
        return dict(energy=s["energy"], axes=s["axes"], counts=s["counts"],
                    xyz=xyz, lookup=lookup)
    if kind == "replicas":
        engine.mc_run_batch(st["boxes"], st["step"], case["moves"])
        st["step"] += case["moves"]
        return dict(energy=np.stack([b.energy() for b in st["boxes"]]),
                    xyz=np.concatenate([b.coords() for b in st["boxes"]]))
    box = st["box"]
    if kind == "trials":
        box.cell_remove_mol(st["mol"])
        ov, en, re = box.particle_inter(st["mol"], 0, st["trials"])
        box.cell_add_mol(st["mol"])
        return dict(en=en, overlap=ov)
    if kind in ("chain", "mp"):
        box.mc_run(st["step"], case["moves"])
        st["step"] += case["moves"]
        return dict(energy=box.energy(), xyz=box.coords())
    if kind == "move":
        ov, lj, re = st["en"].MoleculeInter(st["new"], st["mol"])
        dr = st["ew"].MolReciprocal(st["new"], st["mol"])
        return dict(overlap=ov, de=np.array([lj, re, dr]))
    if kind == "forces":
        aF, mF, lj, re = box.box_force()
        box.box_reciprocal_sums()
        rec = box.box_reciprocal()
        aR, mR = box.box_force_reciprocal()
        tq = box.calculate_torque()
        return dict(energy=np.array([lj, re, rec]), aF=aF, mF=mF, aR=aR,
                    mR=mR, tq=tq)
    if kind == "total":
        t = box.system_total()
        # a job that checks its energies keeps the refreshed structure
        # factors with them
        sr, si = box.sums_new()
        return dict(energy=np.array([t[k] for k in ("inter", "real", "recip",
                                                    "self", "correction")]),
                    sr=sr, si=si)
    if kind == "volume":
        lj, re = box.box_inter_coords(st["edges"], st["xyz"])
        box.recip_init(st["edges"])
        box.box_reciprocal_setup_coords(st["xyz"])
        return dict(energy=np.array([lj, re, box.box_reciprocal(True)]))
    return dict(virial=box.virial())


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _k_count(edge, rcut):
    kc = -2.0 * math.log(TOL) / rcut
    return 2.0 / 3.0 * math.pi * (kc * edge / (2.0 * math.pi)) ** 3


def _water_work(n, rcut):
    """(atoms, k-vectors, in-cutoff pairs) of n waters."""
    e = _edge(n)
    cut = 4.0 / 3.0 * math.pi * rcut ** 3 * 3 * n / e ** 3
    return 3 * n, _k_count(e, rcut), 3 * n * cut / 2.0


def work(case):
    kind = case["kind"]
    if kind == "gemc":
        n0, n1 = case["n0"], case["n1"]
        cut = 4.0 / 3.0 * math.pi * LJ_RCUT ** 3
        d0, d1 = cut * n0 / case["l0"] ** 3, cut * n1 / case["l1"] ** 3
        per = 0.8 * 2 * d0 + 0.19 * 10 * (d0 + d1) + 0.01 * (n0 * d0 + n1 * d1)
        return dict(bytes=2 * 24 * (n0 + n1), flops=case["moves"] * per * 20)
    if kind == "trials":
        cut = 4.0 / 3.0 * math.pi * LJ_RCUT ** 3 * case["n"] / \
            _lj_edge(case["n"]) ** 3
        return dict(bytes=24 * (case["n"] + case["trials"]),
                    flops=case["trials"] * cut * 20)
    sizes = _sizes(case) if kind == "replicas" else [case["n"]]
    total = dict(bytes=0.0, flops=0.0)
    for n in sizes:
        atoms, k, pairs = _water_work(n, case["rcut"])
        per_move = 49 * k + 6 * 2 * pairs / atoms * 33
        sums = atoms * 2 * k * 2  # one multiply-add per atom, k and part
        if kind in ("chain", "replicas", "mp", "move"):
            moves = case.get("moves", 1)
            total["flops"] += moves * per_move
            total["bytes"] += (2 * 24 * atoms + 40 * k) if kind != "move" \
                else 24 * atoms + 56 * k
            if kind == "mp":  # two states' forces and one set of sums
                total["flops"] += 0.01 * moves * (
                    2 * (3 * sums + pairs * 60) + sums)
        elif kind == "forces":
            total["flops"] += 4 * sums + pairs * 60
            total["bytes"] += 24 * atoms * 3 + 24 * n * 3 + 56 * k
        elif kind == "virial":
            total["flops"] += 3 * sums + pairs * 40
            total["bytes"] += 24 * atoms + 56 * k
        else:
            total["flops"] += sums + pairs * 33
            total["bytes"] += 24 * atoms + 40 * k
    return total


# ---------------------------------------------------------------------------
# The same in 64 bits, without the framework
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Pairs:
    """All in-cutoff pairs of different molecules, rows in chunks."""

    def __init__(self, pos, q, kind, mol, edge, rcut, alpha, sig, eps):
        d = _dev()
        self.x = torch.as_tensor(np.asarray(pos), dtype=torch.float64,
                                 device=d)
        self.q = torch.as_tensor(q, dtype=torch.float64, device=d)
        self.kind = torch.as_tensor(np.asarray(kind), device=d)
        self.mol = torch.as_tensor(np.asarray(mol), device=d)
        self.L, self.rc, self.al = float(edge), rcut, alpha
        self.sig, self.eps = sig, eps

    def rows(self):
        n = self.x.shape[0]
        step = max(1, 30_000_000 // n)
        for i0 in range(0, n, step):
            yield slice(i0, min(n, i0 + step))

    def table(self, sl, x=None):
        """(i, j, r2, dr) of the pairs of rows `sl` (or points x)."""
        xi = self.x[sl] if x is None else x
        dr = xi[:, None, :] - self.x[None, :, :]
        dr -= self.L * torch.round(dr / self.L)
        r2 = (dr * dr).sum(-1)
        keep = r2 < self.rc * self.rc
        if x is None:
            keep &= self.mol[sl][:, None] != self.mol[None, :]
        i, j = keep.nonzero(as_tuple=True)
        return i, j, r2[i, j], dr[i, j]

    def lj(self, r2):
        s3 = (self.sig * self.sig / r2) ** 3
        return 4 * self.eps * (s3 * s3 - s3)

    def lj_vir(self, r2):
        s3 = (self.sig * self.sig / r2) ** 3
        return 24 * self.eps * (2 * s3 * s3 - s3) / r2

    def coul(self, r2):
        r = r2.sqrt()
        return torch.erfc(self.al * r) / r

    def coul_vir(self, r2):
        r = r2.sqrt()
        return (torch.erfc(self.al * r) / r + 2 * self.al / math.sqrt(math.pi)
                * torch.exp(-self.al * self.al * r2)) / r2


def _water_pairs(s, pos, edge, rcut):
    return _Pairs(pos, s.atom_charge, s.atom_kind, s.atom_mol, edge, rcut,
                  math.sqrt(-math.log(TOL)) / rcut, s.kinds[0].sigma,
                  s.kinds[0].epsilon)


class _Recip:
    """k-vectors in the reference's order and exp(i k r) by axis."""

    def __init__(self, edge, rcut):
        al2 = -math.log(TOL) / rcut ** 2
        kc = -2.0 * math.log(TOL) / rcut
        c = 2.0 * math.pi / edge
        m = int(kc * edge / (2 * math.pi)) + 1
        g = np.arange(-m, m + 1)
        n = np.stack(np.meshgrid(np.arange(m + 1), g, g, indexing="ij"),
                     -1).reshape(-1, 3)
        half = (n[:, 0] > 0) | (n[:, 1] > 0) | ((n[:, 1] == 0) & (n[:, 2] > 0))
        k2 = ((c * n) ** 2).sum(1)
        n = n[half & (k2 < kc * kc)]
        k2 = ((c * n) ** 2).sum(1)
        d = _dev()
        self.pre = torch.as_tensor(
            QQ * np.exp(-k2 / (4 * al2)) / (k2 * edge ** 3 / (4 * math.pi)),
            device=d)
        self.k2 = torch.as_tensor(k2, device=d)
        self.n = torch.as_tensor(n, device=d)
        self.c, self.m, self.al2, self.edge = c, m, al2, edge
        # columns (n_y, n_z): k-vector = row n_x of column `col`
        key = n[:, 1] * 1000 + n[:, 2]
        u, col = np.unique(key, return_inverse=True)
        self.ny = torch.as_tensor(np.round(u / 1000).astype(np.int64),
                                  device=d)
        self.nz = torch.as_tensor(
            (u - 1000 * np.round(u / 1000)).astype(np.int64), device=d)
        self.col = torch.as_tensor(col, device=d)

    def phases(self, x):
        """exp(i n t) of one axis, [n_points, 2 m + 1], n = -m..m."""
        t = x / self.edge
        n = torch.arange(-self.m, self.m + 1, device=x.device)
        f = n[None, :] * t[:, None]
        f = (f - torch.round(f)) * (2 * math.pi)
        return torch.complex(torch.cos(f), torch.sin(f))

    def chunks(self, x):
        step = max(1, 60_000_000 // max(1, self.ny.shape[0]))
        for a in range(0, x.shape[0], step):
            xs = x[a:a + step]
            ex = self.phases(xs[:, 0])[:, self.m:]
            yz = self.phases(xs[:, 1])[:, self.m + self.ny] * \
                self.phases(xs[:, 2])[:, self.m + self.nz]
            yield slice(a, a + xs.shape[0]), ex, yz

    def sums(self, x, q):
        s = 0
        for sl, ex, yz in self.chunks(x):
            s = s + (ex * q[sl, None]).T @ yz
        return s[self.n[:, 0], self.col]

    def energy(self, s):
        return float((self.pre * (s.real ** 2 + s.imag ** 2)).sum())

    def force(self, x, q, s):
        """2 q sum_k pre (sin(k r) S_R - cos(k r) S_I) k."""
        out = torch.empty_like(x)
        kv = self.c * self.n.to(torch.float64)
        for sl, ex, yz in self.chunks(x):
            for d in range(3):
                c = torch.zeros(self.m + 1, self.ny.shape[0],
                                dtype=torch.complex128, device=x.device)
                c[self.n[:, 0], self.col] = self.pre * kv[:, d] * s.conj()
                f = ((ex @ c) * yz).sum(1).imag
                out[sl, d] = 2 * q[sl] * f
        return out


def _intra(p, al):
    """Same-molecule pairs of waters: (i, j, dr, r) with i != j."""
    x = p.x.view(-1, 3, 3)
    d = x[:, :, None, :] - x[:, None, :, :]
    d = d - p.L * torch.round(d / p.L)
    qq = p.q.view(-1, 3)[:, :, None] * p.q.view(-1, 3)[:, None, :]
    off = ~torch.eye(3, dtype=torch.bool, device=x.device)
    return d, qq * off, (d * d).sum(-1).sqrt() + (~off).double()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gemc", "replicas", "chain", "mp"):
        return None  # the state after many accepted and rejected moves
    if kind == "trials":
        s = _lj(case["n"], _lj_edge(case["n"]), seed)
        m, trials = _trial_set(case, s, seed)
        keep = np.arange(s.n_mol) != m
        p = _Pairs(s.pos[keep], s.atom_charge[keep], s.atom_kind[keep],
                   s.atom_mol[keep], s.box[0], LJ_RCUT, 0.0, LJ_SIG, LJ_EPS)
        x = torch.as_tensor(trials, device=_dev())
        i, j, r2, _ = p.table(None, x)
        en = torch.zeros(len(trials), dtype=torch.float64, device=_dev())
        return dict(en=en.index_add(0, i, p.lj(r2)), overlap=None)
    s = _water(case["n"], seed)
    edge, rcut = float(s.box[0]), case["rcut"]
    pos = s.pos
    if kind == "volume":
        edges, pos = _scaled(case, s)
        edge = float(edges[0])
    p = _water_pairs(s, pos, edge, rcut)
    al = p.al
    if kind == "move":
        m, new = _proposal(s, seed)
        own = slice(3 * m, 3 * m + 3)
        q0 = p.q[own]
        lj = re = 0.0
        rec = _Recip(edge, rcut)
        xn = torch.as_tensor(new, device=_dev())
        for sign, x in ((-1.0, p.x[own]), (1.0, xn)):
            i, j, r2, _ = p.table(None, x)
            other = p.mol[j] != m
            i, j, r2 = i[other], j[other], r2[other]
            oo = (i == 0) & (p.kind[j] == 0)
            lj = lj + sign * p.lj(r2[oo]).sum()
            re = re + sign * (QQ * q0[i] * p.q[j] * p.coul(r2)).sum()
        s0 = rec.sums(p.x, p.q)
        s1 = s0 + rec.sums(xn, q0) - rec.sums(p.x[own], q0)
        dr = (rec.pre * ((s1 - s0) * (s1 + s0).conj()).real).sum()
        return dict(overlap=None, de=torch.stack([lj, re, dr]))
    lj = re = 0.0
    vir = torch.zeros(2, 3, dtype=torch.float64, device=_dev())
    aF = torch.zeros_like(p.x)
    x3 = p.x.view(-1, 3, 3)
    un = x3[:, :1] + (x3 - x3[:, :1]
                      - edge * torch.round((x3 - x3[:, :1]) / edge))
    com = un.mean(1)
    for sl in p.rows():
        i, j, r2, dr = p.table(sl)
        i = i + sl.start
        oo = (p.kind[i] == 0) & (p.kind[j] == 0)
        qq = p.q[i] * p.q[j]
        lj = lj + 0.5 * p.lj(r2[oo]).sum()
        re = re + 0.5 * QQ * (qq * p.coul(r2)).sum()
        if kind in ("forces", "virial"):
            fl = torch.where(oo, p.lj_vir(r2), torch.zeros_like(r2))
            fc = QQ * qq * p.coul_vir(r2)
            if kind == "forces":
                aF.index_add_(0, i, dr * (fl + fc)[:, None])
            else:
                cc = com[p.mol[i]] - com[p.mol[j]]
                cc = cc - edge * torch.round(cc / edge)
                for k, f in enumerate((fl, fc)):
                    vir[k] += 0.5 * (f[:, None] * dr * cc).sum(0)
    rec = _Recip(edge, rcut)
    sk = rec.sums(p.x, p.q)
    e_rec = rec.energy(sk)
    if kind == "volume":
        return dict(energy=np.array([float(lj), float(re), e_rec]))
    d, qq, r = _intra(p, al)
    if kind == "total":
        corr = -0.5 * QQ * float((qq * torch.erf(al * r) / r).sum())
        self_e = -QQ * al / math.sqrt(math.pi) * float((p.q ** 2).sum())
        return dict(energy=np.array([float(lj), float(re), e_rec, self_e,
                                     corr]), sr=sk.real, si=sk.imag)
    aR = rec.force(p.x, p.q, sk)
    if kind == "virial":
        k2, kv = rec.k2, rec.c * rec.n.to(torch.float64)
        w = rec.pre * (sk.real ** 2 + sk.imag ** 2)
        w = (w[:, None] * (1 - 2 * (0.25 / rec.al2 + 1 / k2)[:, None]
                           * kv * kv)).sum(0)
        w = w - (aR * (un - com[:, None]).reshape(-1, 3)).sum(0)
        t = torch.cat([vir, w[None]])
        return dict(virial=torch.cat([t.sum(1), t.sum()[None], t.reshape(-1),
                                      t.sum(0)]))
    f = QQ * qq * (torch.erf(al * r) / r - 2 * al / math.sqrt(math.pi)
                   * torch.exp(-al * al * r * r)) / r ** 2
    aR = aR - (f[..., None] * d).sum(2).reshape(-1, 3)
    both = (aF + aR).view(-1, 3, 3)
    tq = torch.linalg.cross(un - com[:, None], both).sum(1)
    return dict(energy=np.array([float(lj), float(re), e_rec]), aF=aF,
                mF=aF.view(-1, 3, 3).sum(1), aR=aR,
                mR=aR.view(-1, 3, 3).sum(1), tq=tq)
