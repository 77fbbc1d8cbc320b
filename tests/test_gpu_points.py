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
