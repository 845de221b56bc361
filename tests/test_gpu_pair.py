"""Tabulated pair potential (TForcePair) and the Berendsen thermostat on the GPU,
against the reference's own outputs (tests/golden).

FP64 mode (the plain-FP64 Lennard-Jones configuration): forces within 1e-10
eV/A and the trajectory within 1e-9 A of the reference.  FP32 mode: the
norm-wise relative force error <= 1e-5.
"""
import os

import numpy as np
import pytest

from conftest import TABLES, load_case, nbr_set

pytestmark = pytest.mark.gpu

LJ = os.path.join(TABLES, "pair.lj.argon")


def lj_context(omdg, d, fp64, rebuild_every=1):
    from objectmd_gb300 import inputs

    ctx = omdg.Context(0)
    ctx.set_box(d["box_lo"], d["box_hi"])
    ctx.set_atoms(d["x0"], d["v0"], masses=[inputs.md_mass("argon")], znum=[18.0])
    ctx.add_pair_table(LJ, fp64=fp64)
    ctx.set_neighbor(0.3, rebuild_every)
    return ctx


@pytest.mark.parametrize("fp64", [True, False])
def test_lj_static_matches_reference(omdg_lib, fp64):
    d = load_case("lj_ar_500")
    with lj_context(omdg_lib, d, fp64) as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
        mine = nbr_set(*ctx.neighbors())
    if fp64:
        assert np.abs(st["f"] - d["f"]).max() < 1e-10
        assert np.abs(st["pot"] - d["pot"]).max() < 1e-12
    else:
        rel = np.linalg.norm(st["f"] - d["f"]) / np.linalg.norm(d["f"])
        assert rel <= 1e-5, rel
    assert mine == set(map(tuple, d["nbr"].tolist()))


def test_lj_fp64_nve_trajectory_matches_reference(omdg_lib):
    """50 steps, dt 1 fs, FP64 end to end (plain LJ configuration)."""
    d = load_case("lj_ar_nve")
    with lj_context(omdg_lib, d, True) as ctx:
        ctx.set_timestep(float(d["dt"]))
        ctx.step(int(d["steps"]))
        st = ctx.get_state()
        kin, pot = ctx.ledger_history()
    L = d["box_hi"] - d["box_lo"]
    dx = st["x"] - d["x"]
    dx -= np.round(dx / L) * L
    assert np.abs(dx).max() < 1e-9
    np.testing.assert_allclose(kin, d["ledger"][1:1 + len(kin), 1], rtol=1e-9)
    np.testing.assert_allclose(pot, d["ledger"][1:1 + len(pot), 2], rtol=1e-9)


def run_thermostat(omdg_lib, d, count_ghosts):
    from objectmd_gb300 import inputs

    ctx = omdg_lib.Context(0)
    ctx.set_box(d["box_lo"], d["box_hi"])
    ctx.set_atoms(d["x0"], d["v0"], masses=[inputs.md_mass("aluminum")], znum=[13.0])
    ctx.add_eam(os.path.join(TABLES, "eam.aluminum5000"))
    ctx.set_neighbor(0.3, 1)
    ctx.set_timestep(float(d["dt"]))
    ctx.set_thermostat(float(d["tcontrol"][0]), float(d["tcontrol"][1]))
    ctx.set_compat("thermostat_counts_ghosts", count_ghosts)
    ctx.step(int(d["steps"]))
    kin, pot = ctx.ledger_history()
    st = ctx.get_state()
    ctx.close()
    return kin, st


def test_berendsen_thermostat_matches_reference(omdg_lib):
    """TempController(300 K, 0.05 ps) on EAM Al starting at 600 K, 20 steps, with
    the reference's temperature divisor (owners plus ghost images)."""
    d = load_case("eam_al_tc")
    kin, st = run_thermostat(omdg_lib, d, True)
    np.testing.assert_allclose(kin, d["ledger"][1:1 + len(kin), 1], rtol=1e-6)
    assert np.abs(st["v"] - d["v"]).max() < 1e-4 * np.abs(d["v"]).max()


def test_berendsen_thermostat_default_counts_owners(omdg_lib, oracle_lib):
    """Default divisor: the box's own atoms; against an FP64 oracle replay."""
    from conftest import TABLES as T
    from objectmd_gb300 import inputs

    oc = oracle_lib
    d = load_case("eam_al_tc")
    kin, st = run_thermostat(omdg_lib, d, False)
    tab = os.path.join(T, "eam.aluminum5000")
    phi, ed, em = (oc.Table.from_file(tab, s) for s in ("PAIR", "EDENS", "EMBED"))
    box = oc.make_box(d["box_lo"], d["box_hi"], (1, 1, 1))
    x = oc.wrap(box, d["x0"])
    v = d["v0"].copy()
    n = len(x)
    mass = np.full(n, inputs.md_mass("aluminum"))
    f = np.zeros((n, 3))
    dt, (tset, tau) = float(d["dt"]), d["tcontrol"]
    ref = []
    for step in range(int(d["steps"])):
        oc.vv_kick_drift(x, v, f, mass, dt)
        x = oc.wrap(box, x)
        f = oc.eam(box, x, oc.neighbors(box, x, phi.max_range() + 0.3), phi, ed, em)[0]
        oc.vv_kick(v, f, mass, dt)
        k = oc.kinetic(v, mass)
        ref.append(k)
        if step:
            v *= oc.berendsen_factor(dt, tau, tset, (2.0 / 3.0) / 8.61734279e-05 * k / n)
    np.testing.assert_allclose(kin, ref, rtol=1e-6)


def _lj(omdg, x, types, ntypes, lo, hi, pairs):
    from objectmd_gb300 import inputs

    ctx = omdg.Context(0)
    ctx.set_box(lo, hi)
    ctx.set_atoms(x, types=types, masses=[inputs.md_mass("argon")] * ntypes, znum=[18.0] * ntypes)
    for a, b in pairs:
        ctx.add_pair_table(LJ, a, b, fp64=True)
    ctx.set_neighbor(0.3, 1)
    return ctx


# The FP64 pass takes 32, 16 or 8 lanes an atom by the box's size (1,216 and
# 3,040 atoms on 152 SMs); untyped and typed, against the oracle.
@pytest.mark.parametrize("ncell,ntypes", [(4, 1), (6, 2), (7, 1), (8, 2), (9, 1), (10, 2)])
def test_fp64_pair_lanes_match_oracle(omdg_lib, oracle_lib, ncell, ntypes):
    from objectmd_gb300 import inputs

    oc = oracle_lib
    x, _, (lo, hi) = inputs.lj_argon(ncell=ncell)
    x = inputs.perturb(x, 0.15, 7, lo, hi)
    types = np.random.default_rng(8).integers(0, ntypes, len(x)).astype(np.int32)
    phi = oc.Table.from_file(LJ, "")
    nb = oc.neighbors(oc.make_box(lo, hi, (1, 1, 1)), x, phi.max_range() + 0.3)
    off, j, _ = nb
    f, e = oc.pair_table(oc.make_box(lo, hi, (1, 1, 1)), x, nb, phi)[:2]
    with _lj(omdg_lib, x, types, ntypes, lo, hi, [(0, 0), (0, 1), (1, 1)][:1 if ntypes == 1 else 3]) as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
    assert np.abs(st["f"] - f).max() < 1e-10
    assert np.abs(st["pot"] - e).max() < 1e-12 + 2.0 ** -23 * np.abs(e).max()


# A pair closer than the first knot is refused (treader.cpp:199-218), and so is a
# pair moved onto one point without a rebuild of the list in between.
@pytest.mark.parametrize("gap,later", [(1.9, None), (0.5, None), (3.0, 1.95), (2.1, 1.95), (2.01, 0.0)])
def test_fp64_pair_below_the_first_knot(omdg_lib, gap, later):
    lo, hi = np.zeros(3), np.full(3, 40.0)
    x = np.array([[10.0, 10.0, 10.0], [10.0 + gap, 10.0, 10.0]])
    with _lj(omdg_lib, x, np.zeros(2, np.int32), 1, lo, hi, [(0, 0)]) as ctx:
        if later is None:
            with pytest.raises(omdg_lib.OMDGError) as err:
                ctx.compute_forces()
            assert err.value.code == omdg_lib.OMDG_ERANGE
        else:
            ctx.set_neighbor(20.0 if later == 0.0 else 3.0, 0)
            ctx.compute_forces()
            x[1, 0] = 10.0 + later
            ctx.set_positions(x)
            with pytest.raises(omdg_lib.OMDGError) as err:
                ctx.compute_forces()
            assert err.value.code in (omdg_lib.OMDG_ERANGE, omdg_lib.OMDG_EOVERLAP)


# Typed FP32 pairs in a box large enough for the compacted rows (256 atoms a
# SM and more), dilute and half and half, one and two type pairs, a number of
# atoms that leaves the last warp ragged, against the oracle.
@pytest.mark.parametrize("share,pairs,lanes", [(0.001, [(0, 1)], 8), (0.5, [(0, 1), (1, 1)], 4),
                                               (0.02, [(1, 1), (0, 1)], 32)])
def test_typed_pair_in_a_large_box_matches_oracle(omdg_lib, oracle_lib, share, pairs, lanes):
    from objectmd_gb300 import inputs

    oc = oracle_lib
    x, _, (lo, hi) = inputs.lj_argon(ncell=22)
    x = inputs.perturb(x, 0.15, 9, lo, hi)[:-5]
    n = len(x)
    types = (np.random.default_rng(10).uniform(size=n) < share).astype(np.int32)
    phi = oc.Table.from_file(LJ, "")
    box = oc.make_box(lo, hi, (1, 1, 1))
    nb = oc.neighbors(box, x, phi.max_range() + 0.3)
    f, e, w = np.zeros((n, 3)), np.zeros(n), np.zeros(n)
    for a, b in pairs:
        oc.pair_table_typed(box, x, types, a, b, nb, phi, f, e, w)
    with omdg_lib.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_atoms(x, types=types, masses=[inputs.md_mass("argon")] * 2, znum=[18.0] * 2)
        for a, b in pairs:
            ctx.add_pair_table(LJ, a, b)
        ctx.set_neighbor(0.3, 1)
        ctx.set_launch("pair_lanes", lanes)
        ctx.compute_forces()
        st = ctx.get_state()
    assert np.linalg.norm(st["f"] - f) / np.linalg.norm(f) <= 1e-5
    assert np.array_equal(np.abs(st["f"]).sum(1) == 0.0, np.abs(f).sum(1) == 0.0)
    # the table ends in a jump (it is not shifted): a pair within FP32's
    # rounding of the cutoff may fall on either side of it
    off, j, code = nb
    i = np.repeat(np.arange(n), np.diff(off))
    shift = np.stack([code % 3 - 1, code // 3 % 3 - 1, code // 9 - 1], 1) * (np.asarray(hi) - lo)
    r = np.linalg.norm(x[i] - x[j] - shift, axis=1)
    clear = np.ones(n, dtype=bool)
    clear[i[np.abs(r - phi.max_range()) < 4e-6]] = False
    assert clear.mean() > 0.99
    assert np.abs(st["pot"] - e)[clear].max() <= 2e-6
