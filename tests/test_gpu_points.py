"""One-molecule and one-atom calls (MoleculeInter, MolReciprocal, the swap
deltas, ParticleInter) against the oracle, at the edges of their tiling: one
to sixteen and more positions a call, molecules of one to eight sites,
positions on the box edges, a Coulomb cutoff below Rcut, a Mie exponent,
no Ewald sum, and a molecule taken out of the grid.

Bar: 1e-10 of the box's own term (of at least 1 K), as in the other FP64
tests of energy differences.
"""
import numpy as np
import pytest

from gomc_gb300.config import SimConfig
from gomc_gb300.systems import AtomKind, MolSystem, MoleculeType
from tests.test_gpu_box_sums import CASES, mixture

pytestmark = pytest.mark.gpu

REL = 1e-10


@pytest.fixture(scope="module")
def gb():
    from gomc_gb300 import engine
    engine.lib(build_if_missing=True)
    return engine


@pytest.mark.parametrize("name", sorted(CASES))
def test_points_against_oracle(gb, name):
    from oracle import oracle as orc
    counts, edges, opt = CASES[name]
    cfg = SimConfig(**{**dict(temperature=298.0, rcut=9.0, tolerance=1e-5),
                       **opt})
    s = mixture(counts, edges, 11, cfg.electrostatic)
    box, ref = gb.Box(s, cfg), orc.OracleBox(s, cfg)
    box.system_total()
    tot = ref.system_total()
    scale = {k: max(abs(tot[k]), 1.0) for k in ("inter", "real", "recip")}
    rng = np.random.default_rng(3)
    L = np.asarray(edges)

    def near(got, want, k):
        assert abs(got - want) <= REL * max(scale[k], abs(want)), (k, got, want)

    lens = np.diff(s.mol_start)
    picks = {int(np.argmax(lens == n)) for n in np.unique(lens)} | {s.n_mol - 1}
    for m in sorted(picks):
        old = ref.coords()[s.mol_start[m]:s.mol_start[m + 1]]
        for shift in (rng.uniform(-0.3, 0.3, 3), -old[0], L / 2):
            new = np.mod(old + shift, L)
            ov, lj, re = box.molecule_inter(m, new)
            o, l, r = ref.molecule_inter(m, new)
            assert ov == o
            near(lj, l, "inter")
            near(re, r, "real")
            if cfg.ewald:
                near(box.mol_reciprocal(m, new), ref.mol_reciprocal(m, new),
                     "recip")
                near(box.swap_dest_recip(m, new), ref.swap_dest_recip(m, new),
                     "recip")
                near(box.swap_source_recip(m, old),
                     ref.swap_source_recip(m, old), "recip")
    m = s.n_mol // 2
    box.cell_remove_mol(m)
    ref.cell_remove_mol(m)
    for n in (1, 16, 17, 200):
        t = rng.random((n, 3)) * L
        t[0] = 0.0
        t[-1, 1] = L[1]
        ov, lj, re = box.particle_inter(m, 0, t)
        for i in range(n):
            o, l, r = ref.particle_inter(m, 0, t[i])
            assert bool(ov[i]) == bool(o)
            near(lj[i], l, "inter")
            near(re[i], r, "real")
    box.cell_add_mol(m)
    box.close()


def chains(length, n, edge, seed):
    """n zigzag chains of `length` charged sites, 6 A apart."""
    rng = np.random.default_rng(seed)
    per = int(edge / 6.0)
    i = np.arange(length)
    one = np.stack([1.1 * (i % 16), 0.9 * (i // 16), 0.4 * (i % 2)], -1)
    q = np.where(i % 2, 0.3, -0.3)
    at = np.arange(n)
    origin = np.stack([0 * at, at % per, at // per], -1) * 6.0
    pos = origin[:, None] + one + rng.uniform(-.05, .05, (n, length, 3))
    kinds = [AtomKind("A", 40.0, 2.6, 12.0), AtomKind("B", 0.0, 1.0, 12.0)]
    kind = (i % 2).astype(np.int32)
    t = MoleculeType("CH", ["X%d" % j for j in i], kind.tolist(), q.tolist())
    return MolSystem(np.full(3, edge), kinds, [t],
                     np.mod(pos.reshape(-1, 3), edge), np.tile(kind, n),
                     np.tile(q, n), np.repeat(at, length).astype(np.int32),
                     (np.arange(n + 1) * length).astype(np.int32),
                     np.zeros(n, np.int32))


# sites: the last of the 16-position call, the first beyond it, the first
# whose positions need one CTA each, the largest molecule
@pytest.mark.parametrize("length", [16, 17, 32, 33, 64])
def test_long_molecules_against_oracle(gb, length):
    from oracle import oracle as orc
    edge = 36.0
    cfg = SimConfig(temperature=298.0, rcut=9.0, tolerance=1e-5)
    s = chains(length, 12, edge, 2)
    box, ref = gb.Box(s, cfg), orc.OracleBox(s, cfg)
    box.system_total()
    tot = ref.system_total()
    rng = np.random.default_rng(4)
    for m in (0, 11):
        old = ref.coords()[s.mol_start[m]:s.mol_start[m + 1]]
        for shift in (rng.uniform(-0.3, 0.3, 3), np.array([3.0, 18.0, 15.0])):
            new = np.mod(old + shift, edge)
            got = box.molecule_inter(m, new) + (box.mol_reciprocal(m, new),)
            want = ref.molecule_inter(m, new) + (ref.mol_reciprocal(m, new),)
            assert got[0] == want[0]
            for g, w, k in zip(got[1:], want[1:], ("inter", "real", "recip")):
                assert abs(g - w) <= REL * max(abs(tot[k]), abs(w), 1.0), (k, g, w)
    box.close()


def test_lj_term_to_the_last_bits(gb):
    """One pair's 12-6 energy over r^2 from 0.25 to 81 A^2, powers of two and
    their neighbours among them, against exact rational arithmetic.

    Separations are multiples of 2^-20 A along one axis, so r^2 is exact.  With
    sigma^2 / r^2 within a unit of the last place (2u, u = 2^-53), its third power
    has 3 x 2 + 2 = 8 u, the sixth 2 x 8 + 1 = 17 u, and the difference and the
    factor epsilon one each: 19 u of the two terms' sum."""
    from fractions import Fraction
    sigma, eps, edge, rc = 2.9, 70.0, 64.0, 9.0
    s = MolSystem(np.full(3, edge), [AtomKind("A", eps, sigma, 12.0)],
                  [MoleculeType("T", ["X"], [0], [0.0])],
                  np.array([[16.0, 16.0, 16.0], [60.0, 60.0, 60.0]]),
                  np.zeros(2, np.int32), np.zeros(2),
                  np.arange(2, dtype=np.int32), np.arange(3, dtype=np.int32),
                  np.zeros(2, np.int32))
    cfg = SimConfig(temperature=298.0, rcut=rc, ewald=False,
                    electrostatic=False)
    box = gb.Box(s, cfg)
    box.cell_remove_mol(1)
    unit = 2.0 ** -20
    pow2 = np.concatenate([np.sqrt(2.0 ** k) * (1 + np.arange(-8, 8) * 2.0 ** -20)
                           for k in range(-2, 7)])
    rng = np.random.default_rng(6)
    r = np.concatenate([pow2, rng.uniform(0.5, rc - 0.01, 1500)])
    r = np.rint(r / unit) * unit
    en = np.concatenate([
        box.particle_inter(1, 0, np.stack([16.0 + c, 0 * c + 16.0, 0 * c + 16.0],
                                          -1))[1]
        for c in np.array_split(r, 8)])
    e4 = Fraction(4.0 * eps)
    s2 = Fraction(sigma * sigma)
    for d, got in zip(r, en):
        x = (s2 / Fraction(d) ** 2) ** 3
        bar = 19 * Fraction(1, 2 ** 53) * e4 * (x * x + x)
        assert abs(Fraction(got) - e4 * (x * x - x)) <= bar, (d, got)
    box.close()


@pytest.mark.parametrize("tol", [1e-5, 1e-10])
def test_ewald_term_to_the_last_bits(gb, tol):
    """One pair's real-space Ewald energy near the cutoff, where the segment
    polynomial bends most, against 40 digits.

    r^2 is exact (as above) and the charge product is taken as the call rounds
    it.  The polynomial interpolates to 1.1e-16 of the value, its constant term,
    last step and the product with the charges round by 1.1e-16 each, and the
    lower terms, a fifth of the value at most, by a fifth of that."""
    mp = pytest.importorskip("mpmath")
    import math
    mp.mp.dps = 40
    edge, rc, qa, qb = 64.0, 10.0, 0.75, -0.5
    s = MolSystem(np.full(3, edge), [AtomKind("A", 0.0, 2.9, 12.0)],
                  [MoleculeType("T", ["X"], [0], [qa])],
                  np.array([[16.0, 16.0, 16.0], [60.0, 60.0, 60.0]]),
                  np.zeros(2, np.int32), np.array([qa, qb]),
                  np.arange(2, dtype=np.int32), np.arange(3, dtype=np.int32),
                  np.zeros(2, np.int32))
    box = gb.Box(s, SimConfig(temperature=298.0, rcut=rc, tolerance=tol))
    box.cell_remove_mol(1)
    unit = 2.0 ** -20
    r = np.rint(np.random.default_rng(9).uniform(8.5, 9.99, 16384) / unit) * unit
    re = np.concatenate([
        box.particle_inter(1, 0, np.stack([16.0 + c, 0 * c + 16.0, 0 * c + 16.0],
                                          -1))[2]
        for c in np.array_split(r, 64)])
    alpha = mp.mpf(math.sqrt(-math.log(tol)) / rc)
    qq = mp.mpf((qb * 167103.208067979) * qa)
    bar = (1.1 + 3 * 1.1 + 0.2 * 1.1) * 1e-16
    for d, got in zip(r, re):
        want = qq * mp.erfc(alpha * mp.mpf(d)) / mp.mpf(d)
        assert abs(mp.mpf(got) - want) <= bar * abs(want), d
    box.close()


@pytest.mark.parametrize("n", [64, 65, 151, 152, 153, 256])
def test_trial_counts_agree(gb, n):
    """A trial's energies do not depend on how many others the call has (and so
    on how many CTAs a trial gets) beyond the order of its sums: 1e-13 of the
    sum of the terms' sizes, some 400 terms in FP64."""
    s = mixture((301, 230, 17), (27.3, 31.1, 64.7), 11)
    box = gb.Box(s, SimConfig(temperature=298.0, rcut=9.0, tolerance=1e-5))
    box.cell_remove_mol(3)
    t = np.random.default_rng(5).random((n, 3)) * s.box
    ov, lj, re = box.particle_inter(3, 0, t)
    for i in range(0, n, 7):
        o, l, r = box.particle_inter(3, 0, t[i:i + 1])
        assert o[0] == ov[i]
        assert abs(l[0] - lj[i]) <= 1e-13 * max(abs(l[0]), 1e3)
        assert abs(r[0] - re[i]) <= 1e-13 * max(abs(r[0]), 1e5)
    box.close()
