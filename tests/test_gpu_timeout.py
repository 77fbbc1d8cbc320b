"""Bounded device-side waits of the FP64 chain (gb_mc_set_wait_limit).

A wait that gives up must not fault or hang the GPU: with the limit cut to
one poll, the chain's waits (grid barrier, partials, the next context, the
decision word) run out long before the other CTAs arrive, gb_mc_run returns
GB_ERR_TIMEOUT, the box's coordinates and running energies are those before
the call, and after gb_mc_init the same box runs the reference's move
sequence exactly as a fresh box does.
"""
import numpy as np
import pytest

from tests.golden_util import config_of, load, move_fractions, system_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    from gomc_gb300 import engine
    engine.lib(build_if_missing=True)
    return engine


def test_wait_limit_times_out_and_box_recovers(gb):
    from gomc_gb300._lib import GbError
    z, meta = load("c0_water")
    sysm, cfg = system_of(z, meta), config_of(meta)
    seed = meta["config"]["random_seed"]
    frac = move_fractions(meta)
    adj = meta["config"]["adj_steps"]
    box = gb.Box(sysm, cfg)
    x0, e0 = box.coords(), box.energy()
    box.mc_init(seed, frac, adj)
    box.mc_set_wait_limit(1)
    with pytest.raises(GbError) as err:
        box.mc_run(0, 200)
    assert err.value.code == 5  # GB_ERR_TIMEOUT
    np.testing.assert_array_equal(box.coords(), x0)
    np.testing.assert_array_equal(box.energy(), e0)

    box.mc_init(seed, frac, adj)  # the default limit, the error cleared
    r = box.mc_run(0, 200, trace=True)
    fresh = gb.Box(sysm, cfg)
    fresh.mc_init(seed, frac, adj)
    rf = fresh.mc_run(0, 200, trace=True)
    for key in ("kind", "mol", "accepted"):
        np.testing.assert_array_equal(r[key], rf[key])
    np.testing.assert_array_equal(r["de"], rf["de"])
    np.testing.assert_array_equal(box.coords(), fresh.coords())
    np.testing.assert_array_equal(box.energy(), fresh.energy())
    box.close()
    fresh.close()


def test_wait_limit_rejects_out_of_range(gb):
    from gomc_gb300._lib import GbError
    z, meta = load("c0_water")
    box = gb.Box(system_of(z, meta), config_of(meta))
    with pytest.raises(GbError):
        box.mc_set_wait_limit(10)  # no loop yet: GB_ERR_STATE
    box.mc_init(meta["config"]["random_seed"], move_fractions(meta),
                meta["config"]["adj_steps"])
    with pytest.raises(GbError):
        box.mc_set_wait_limit(-1)
    box.mc_set_wait_limit(0)
    box.close()


def test_ewald_sums_report_a_wait_that_gives_up(gb):
    """One poll for the waits of the box-wide Ewald sums: every call that uses
    them says so, nothing incomplete is kept, and with the default back the box
    gives what it gave before."""
    from gomc_gb300._lib import GbError
    z, meta = load("c0_water")
    sysm, cfg = system_of(z, meta), config_of(meta)
    box = gb.Box(sysm, cfg)
    x0 = box.coords()
    box.recip_init(box.edges())

    def volume():
        box.box_reciprocal_setup_coords(x0)
        return box.box_reciprocal(True)

    def forces():
        box.box_reciprocal_sums()
        return box.box_force_reciprocal()

    calls = [lambda: list(box.system_total().values()),
             box.box_reciprocal_setup, box.box_reciprocal_sums,
             lambda: box.box_reciprocal_sums(x0), volume, forces, box.virial,
             lambda: box.set_coords(x0)]

    def values(r):
        return [] if r is None else list(r) if isinstance(r, tuple) else [r]

    for f in calls:  # the last one wraps the molecules by their centres
        f()
    want = [values(f()) for f in calls]
    ref, e0 = box.kvectors(), box.energy()
    for i, f in enumerate(calls + [box.box_force_reciprocal]):
        box.set_wait_limit(1)
        with pytest.raises(GbError) as err:
            f()
        assert err.value.code == 5, i  # GB_ERR_TIMEOUT
        np.testing.assert_array_equal(box.energy(), e0)
        kv = box.kvectors()
        for k in ("sumRref", "sumIref"):
            np.testing.assert_array_equal(kv[k], ref[k])
        # still reported, without another wait
        assert pytest.raises(GbError, box.box_inter).value.code == 5
        box.set_wait_limit(0)
        box.box_inter()
    for f, w in zip(calls, want):
        for a, b in zip(values(f()), w):
            np.testing.assert_array_equal(a, b)
    with pytest.raises(GbError):
        box.set_wait_limit(-1)
    box.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_multiparticle_move_with_a_wait_that_gives_up(gb, precision):
    from gomc_gb300._lib import GbError
    z, meta = load("c0_water")
    sysm, cfg = system_of(z, meta), config_of(meta)
    box = gb.Box(sysm, cfg, precision=precision)
    x0 = box.coords()
    box.mc_init(7, [0.0, 0.0, 1.0], 100)
    box.set_wait_limit(1)
    with pytest.raises(GbError) as err:
        box.mc_run(0, 4)
    assert err.value.code == 5
    np.testing.assert_array_equal(box.coords(), x0)
    box.set_wait_limit(0)
    box.mc_init(7, [0.0, 0.0, 1.0], 100)
    r = box.mc_run(0, 8, trace=True)
    fresh = gb.Box(sysm, cfg, precision=precision)
    fresh.mc_init(7, [0.0, 0.0, 1.0], 100)
    f = fresh.mc_run(0, 8, trace=True)
    np.testing.assert_array_equal(r["accepted"], f["accepted"])
    np.testing.assert_array_equal(box.coords(), fresh.coords())
    box.close()
    fresh.close()
