"""The box-wide walks and sums -- BoxInter, BoxForce, VirialCalc, the
structure factor and the reciprocal forces -- against the oracle, where their
tiling can go wrong: boxes of three cells per axis, edges that differ (one
five times the others), one molecule, atom counts around the warp, batch and
tile sizes, molecules of one to eight sites, a Coulomb cutoff below Rcut, a
Mie exponent other than 12, and no Ewald sum.

Bar: 1e-10 of the largest value of each output (of at least 1 K), the bar of
the other FP64 tests.
"""
import numpy as np
import pytest

from gomc_gb300.config import SimConfig
from gomc_gb300.systems import AtomKind, MolSystem, MoleculeType

pytestmark = pytest.mark.gpu

REL = 1e-10


def mixture(counts, box, seed, charged=True):
    """counts[t] molecules of type t (1, 3 and 8 sites) on a jittered grid of
    at least 3.3 A, randomly assigned to its points."""
    rng = np.random.default_rng(seed)
    box = np.asarray(box, dtype=np.float64)
    kinds = [AtomKind("A", 70.0, 2.9, 12.0), AtomKind("H", 0.0, 1.0, 12.0),
             AtomKind("M", 45.0, 2.7, 14.0)]
    sites = [np.zeros((1, 3)),
             np.array([[0, 0, 0], [0.8, 0.55, 0], [-0.8, 0.55, 0.1]]),
             np.array([[x, y, z] for x in (-.4, .4) for y in (-.4, .4)
                       for z in (-.4, .4)], dtype=np.float64)]
    akind = [[2], [0, 1, 1], [0, 1, 1, 1, 1, 1, 1, 2]]
    q = [[0.35], [-0.8, 0.4, 0.4], [-0.7, .1, .1, .1, .1, .1, .1, 0.0]]
    if not charged:
        q = [[0.0] * len(c) for c in q]
    types = [MoleculeType("T%d" % t, ["X%d" % i for i in range(len(s))],
                          akind[t], q[t]) for t, s in enumerate(sites)]
    n = np.maximum((box / 3.3).astype(int), 1)
    grid = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"),
                    -1).reshape(-1, 3)
    pick = grid[rng.permutation(len(grid))[:sum(counts)]]
    centre = (pick + 0.5) * (box / n) + rng.uniform(-0.2, 0.2, pick.shape)
    pos, kind, chg, mol, start, mtype = [], [], [], [], [0], []
    order = rng.permutation(np.repeat(np.arange(3), counts))
    for m, t in enumerate(order):
        a = rng.uniform(0, 2 * np.pi)
        rot = np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0],
                        [0, 0, 1.0]])
        pos.append(np.mod(centre[m] + sites[t] @ rot.T, box))
        kind += akind[t]
        chg += q[t]
        mol += [m] * len(akind[t])
        start.append(start[-1] + len(akind[t]))
        mtype.append(t)
    return MolSystem(box, kinds, types, np.concatenate(pos),
                     np.array(kind, np.int32), np.array(chg),
                     np.array(mol, np.int32), np.array(start, np.int32),
                     np.array(mtype, np.int32))


# molecules by type, edges, configuration
CASES = {
    "one_molecule": ((0, 0, 1), (20.0, 20.0, 20.0), {}),
    "three_cells": ((60, 40, 3), (20.0, 23.1, 26.9), {}),
    "odd_edges": ((301, 230, 17), (27.3, 31.1, 64.7), {}),
    "coulomb_cut": ((100, 99, 1), (28.0, 28.0, 29.5),
                    dict(rcut=9.0, rcut_coulomb=7.5)),
    "no_ewald": ((128, 64, 5), (30.0, 27.5, 33.0), dict(ewald=False)),
    "neutral": ((257, 100, 0), (31.0, 30.0, 36.0),
                dict(ewald=False, electrostatic=False)),
    "tile_128": ((128, 0, 0), (24.0, 24.0, 24.0), {}),
    "tile_129": ((129, 0, 0), (24.0, 24.0, 24.0), {}),
    "many_sites": ((1, 900, 301), (45.0, 47.0, 49.0), {}),
    # |n_z| and |n_x| to 41: more columns than one tile of the product has
    "long_z": ((0, 60, 1), (20.0, 20.5, 101.0), {}),
    "long_x": ((0, 60, 1), (101.0, 20.5, 20.0), {}),
    # 33,024 atoms: more than one batch of the product, a molecule across it
    "two_batches": ((32700, 100, 3), (109.0, 109.0, 110.0),
                    dict(rcut=12.0, tolerance=1e-2)),
}


@pytest.fixture(scope="module")
def gb():
    from gomc_gb300 import engine
    engine.lib(build_if_missing=True)
    return engine


def near(got, ref):
    ref = np.asarray(ref, dtype=np.float64)
    np.testing.assert_allclose(np.asarray(got).reshape(ref.shape), ref, rtol=0,
                               atol=REL * max(np.abs(ref).max(), 1.0))


@pytest.mark.parametrize("name", sorted(CASES))
def test_against_oracle(gb, name):
    from oracle import oracle as orc
    counts, edges, opt = CASES[name]
    cfg = SimConfig(**{**dict(temperature=298.0, rcut=9.0, tolerance=1e-5),
                       **opt})
    s = mixture(counts, edges, 5, cfg.electrostatic)
    box, ref = gb.Box(s, cfg), orc.OracleBox(s, cfg)
    st, rt = box.system_total(), ref.system_total()
    for k in ("inter", "real", "recip", "self", "correction", "total"):
        near(st[k], rt[k])
    aF, mF, lj, re = box.box_force()
    rF = ref.box_force()
    near(aF, rF[0])
    near(mF, rF[1])
    near(lj, rF[2])
    near(re, rF[3])
    if cfg.ewald:
        near(box.sums_new(), ref.sum_new())
        box.copy_recip()
        ref.copy_recip()
        aR, mR = box.box_force_reciprocal()
        rR = ref.box_force_recip()
        near(aR, rR[0])
        near(mR, rR[1])
    near(box.virial(), ref.virial())
    box.close()


def test_cutoff_to_the_last_bit(gb):
    """216 isolated pairs whose r^2 is within a few units of the last place of
    Rcut^2: each is inside or outside as the oracle's unfused r^2 has it (one
    pair's terms are 1e-3 of the sums)."""
    from oracle import oracle as orc
    rng = np.random.default_rng(8)
    edge, rc = 180.0, 9.0
    g = np.arange(6) * 30.0 + 8.0
    a = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    v = rng.normal(size=a.shape)
    v *= rc / np.linalg.norm(v, axis=1)[:, None]
    pos = np.mod(np.concatenate([a, a + v]), edge)
    n = len(pos)
    s = MolSystem(np.full(3, edge), [AtomKind("A", 70.0, 2.9, 12.0)],
                  [MoleculeType("T", ["X"], [0], [0.0])], pos,
                  np.zeros(n, np.int32), np.zeros(n),
                  np.arange(n, dtype=np.int32),
                  np.arange(n + 1, dtype=np.int32), np.zeros(n, np.int32))
    cfg = SimConfig(temperature=298.0, rcut=rc, ewald=False,
                    electrostatic=False)
    box, ref = gb.Box(s, cfg), orc.OracleBox(s, cfg)
    want = ref.system_total()["inter"]
    one = abs(4 * 70.0 * (2.9 / rc) ** 6)
    assert 20 * one < abs(want) < 196 * one  # some pairs on each side
    near(box.system_total()["inter"], want)
    aF, mF, lj, _ = box.box_force()
    rF = ref.box_force()
    near(aF, rF[0])
    near(lj, rF[2])
    near(box.virial(), ref.virial())
    box.close()


# column tiles of 16, 32, 48 and 64, and two of 48
@pytest.mark.parametrize("edge,tol,kmax", [
    (20.0, 1e-3, (4, 7)), (50.0, 1e-3, (8, 15)), (50.0, 1e-5, (16, 23)),
    (70.0, 1e-5, (24, 31)), (97.0, 1e-5, (32, 47))])
def test_structure_factor_digits(gb, edge, tol, kmax):
    """Every digit product of the structure factor counts: 64 single charges
    against extended precision.

    A product of a y-z and an x factor, numbers below 1 to 2^-54 each (2^-55
    off), misses the digit products i + j >= 7, six of at most 2^14 2^-68, five
    of 2^8 times less and so on, 6.03 2^-54 in all: with the rounding of its
    phases within 2^-51 of the charge unit (a power of two above the charges).
    An atom has four in each part of a sum.  A digit product left out moves each
    by up to 64 x 128 x 2^-60 and more."""
    s = mixture((64, 0, 0), (edge,) * 3, 3)
    cfg = SimConfig(temperature=298.0, rcut=9.0, tolerance=tol)
    box = gb.Box(s, cfg)
    assert kmax[0] <= box.num_kvectors()[1] <= kmax[1]
    box.system_total()
    sr, si = box.sums_new()
    kv = box.kvectors()
    n = np.rint(np.stack([kv[c] for c in ("kx", "ky", "kz")], 1) * edge /
                (2 * np.pi)).astype(np.longdouble)
    turns = np.asarray(box.coords(), np.longdouble) / np.longdouble(edge)
    t = n @ turns.T
    a = (t - np.rint(t)) * np.longdouble("6.28318530717958647692528676655900577")
    q = s.atom_charge.astype(np.longdouble)
    bar = 4 * 2.0 ** -51 * 64 * 0.5  # 64 charges below 2^-1
    assert np.abs(sr - np.cos(a) @ q).max() <= bar
    assert np.abs(si - np.sin(a) @ q).max() <= bar
    box.close()


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_charge_that_is_not_finite(gb, value):
    """An infinite charge or one that is not a number shows in every sum and
    force it enters, and in no other."""
    from oracle import oracle as orc
    s = mixture((60, 40, 3), (20.0, 23.1, 26.9), 5)
    s.atom_charge[17] = value
    cfg = SimConfig(temperature=298.0, rcut=9.0, tolerance=1e-5)
    box, ref = gb.Box(s, cfg), orc.OracleBox(s, cfg)
    st, rt = box.system_total(), ref.system_total()
    for k in ("inter", "real", "recip", "self", "correction", "total"):
        assert np.isfinite(st[k]) == np.isfinite(rt[k]), k
    near(st["inter"], rt["inter"])
    for got, want in zip(box.sums_new(), ref.sum_new()):
        assert not np.isfinite(want).any() and not np.isfinite(got).any()
    box.copy_recip()
    ref.copy_recip()
    for got, want in zip(box.box_force_reciprocal() + box.box_force()[:2],
                         ref.box_force_recip()[:2] + ref.box_force()[:2]):
        np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
    np.testing.assert_array_equal(np.isfinite(box.virial()),
                                  np.isfinite(ref.virial()))
    box.close()


def test_structure_factor_of_unequal_charges(gb):
    """Two charges of 2 among 2,998 a thousand times smaller: a term is within
    2^-51 of the power of two above the charges of its own size (four terms an
    atom and part, as above), and the sum is rounded once for each size."""
    n, edge = 3000, 44.0
    rng = np.random.default_rng(2)
    q = np.where(np.arange(n) % 2, 1e-3, -1e-3)
    q[[5, 1700]] = 2.0, -2.0
    s = MolSystem(np.full(3, edge), [AtomKind("A", 0.0, 2.9, 12.0)],
                  [MoleculeType("T", ["X"], [0], [0.0])],
                  rng.random((n, 3)) * edge, np.zeros(n, np.int32), q,
                  np.arange(n, dtype=np.int32),
                  np.arange(n + 1, dtype=np.int32), np.zeros(n, np.int32))
    box = gb.Box(s, SimConfig(temperature=298.0, rcut=9.0, tolerance=1e-5))
    box.system_total()
    sr, si = box.sums_new()
    kv = box.kvectors()
    pick = rng.permutation(len(sr))[:1500]
    k = np.rint(np.stack([kv[c] for c in ("kx", "ky", "kz")], 1)[pick] * edge /
                (2 * np.pi)).astype(np.longdouble)
    turns = np.asarray(box.coords(), np.longdouble) / np.longdouble(edge)
    t = k @ turns.T
    a = (t - np.rint(t)) * np.longdouble("6.28318530717958647692528676655900577")
    ql = q.astype(np.longdouble)
    bar = 2.0 ** -49 * (2 * 4.0 + 2998 * 2.0 ** -9) + 2 * 2.0 ** -53 * 4.1
    assert np.abs(sr[pick] - np.cos(a) @ ql).max() <= bar
    assert np.abs(si[pick] - np.sin(a) @ ql).max() <= bar
    box.close()
