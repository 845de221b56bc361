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


def dimers(r, direction, spacing):
    """Pairs at distances r along a direction, on a grid; returns the positions
    (first atoms, then second ones) and the box."""
    n = len(r)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * spacing + 1.0
    d = np.asarray(direction, dtype=np.float64)
    return np.vstack([grid, grid + np.asarray(r)[:, None] * d / np.linalg.norm(d)]), np.zeros(3), np.full(3, side * spacing)


def dimer_forces(omdg, table, x, lo, hi):
    with omdg.Context(0) as ctx:
        ctx.set_box(lo, hi, (False, False, False))
        ctx.set_atoms(x, masses=[39.948], znum=[18.0])
        ctx.add_pair_table(str(table), fp64=True)
        ctx.set_neighbor(0.3, 1)
        ctx.compute_forces()
        return ctx.get_state()["f"]


def plain_table(path, off, dr, values):
    lines = ["#$ NumberOfData %d" % len(values), "#$ Spacing %.17g" % dr, "#$ Offset %.17g" % off, "#$ Format PLAIN",
             "#$ --"] + ["%.17g" % v for v in values]
    path.write_text("\n".join(lines) + "\n")


# Distances within 2e-4 of a segment of a knot, where FP32 may name the wrong
# segment, in a table of measured values (LJ with noise of 1e-4 eV): the slope's
# cubic term jumps from segment to segment, so the neighbouring segment's slope
# is off by 1e-8 eV/A.  Allowed: the FP64 rounding of the four operations of the
# slope (each at most its largest term's, eight ulps in all), and that of r and
# of its offset from the knot (four ulps of r) times the curvature.
def test_fp64_pair_next_to_the_knots(omdg_lib, oracle_lib, tmp_path):
    oc = oracle_lib
    rng = np.random.default_rng(21)
    n, off, rc = 5000, 2.0, 8.5125
    dr = (rc - off) / (n - 1)
    at = off + dr * np.arange(n)
    s6 = (3.405 / at) ** 6
    plain_table(tmp_path / "noisy", off, dr, 4 * 0.0104 * (s6 * s6 - s6) + 1e-4 * rng.standard_normal(n))
    t = oc.Table.from_file(str(tmp_path / "noisy"), "")
    knot = rng.integers(1, n - 2, 1000)
    x, lo, hi = dimers(off + dr * (knot + rng.uniform(1e-6, 2e-4, 1000) * rng.choice([-1.0, 1.0], 1000)), (1, 0, 0), 20.0)
    f = dimer_forces(omdg_lib, tmp_path / "noisy", x, lo, hi)
    r = x[1000:, 0] - x[:1000, 0]
    k = ((r - off) / dr).astype(int)
    d = np.longdouble(r) - np.longdouble(off) - k * np.longdouble(dr)
    c3, c2, c1 = 3 * t.a[k] * d * d, 2 * t.b[k] * d, np.longdouble(t.c[k])
    tol = 8 * 2.0 ** -53 * (abs(c3) + abs(c2) + abs(c1)) + 4 * 2.0 ** -53 * r * abs(2 * t.b[k] + 6 * t.a[k] * d)
    assert (np.abs(f[:1000, 0] - (c3 + c2 + c1)) <= tol).all()
    assert np.array_equal(f[:1000], -f[1000:])


# The root and its reciprocal over the range of distances, against numpy's: in a
# table of phi = r a pair's force is its unit vector, r^2's rounding (an ulp, half
# of it in the root), the reciprocal's, and three products'.
@pytest.mark.parametrize("direction", [(1, 0, 0), (0.3, -1.1, 0.7)])
def test_fp64_pair_unit_vectors(omdg_lib, oracle_lib, tmp_path, direction):
    n, off, rc = 2000, 1e-3, 40.0
    dr = (rc - off) / (n - 1)
    plain_table(tmp_path / "line", off, dr, off + dr * np.arange(n))
    r = np.exp(np.random.default_rng(22).uniform(np.log(0.01), np.log(39.9), 500))
    x, lo, hi = dimers(r, direction, 90.0)
    f = dimer_forces(omdg_lib, tmp_path / "line", x, lo, hi)
    t = oracle_lib.Table.from_file(str(tmp_path / "line"), "")
    slope = np.abs(np.array([t.read(q)[1] for q in r]) - 1.0).max()  # the table's own rounding
    d = np.longdouble(x[500:]) - np.longdouble(x[:500])
    u = d / np.sqrt((d * d).sum(1))[:, None]
    assert np.abs(f[:500] - u).max() <= 6 * 2.0 ** -53 + 2 * slope


# The thermostat's factor from one root estimate, against the formula in extended
# precision: atoms without neighbours, whose velocities only it changes.  Allowed:
# the three roundings of its quotients (half an ulp each, in an argument whose
# root halves them) and the root's, 4 x 2^-53; the velocities' product one more.
@pytest.mark.parametrize("target,tau", [(300.0, 0.1), (0.0, 0.5), (5000.0, 0.02), (90.0, 10.0)])
def test_thermostat_factor(omdg_lib, target, tau):
    rng = np.random.default_rng(23)
    x, lo, hi = dimers(np.full(32, 15.0), (0, 0, 1), 40.0)
    v = rng.standard_normal(x.shape)
    dt, n = 0.001, len(x)
    with omdg_lib.Context(0) as ctx:
        ctx.set_box(lo, hi, (False, False, False))
        ctx.set_atoms(x, v, masses=[39.948], znum=[18.0])
        ctx.add_pair_table(LJ)
        ctx.set_neighbor(0.3, 0)
        ctx.set_timestep(dt)
        ctx.set_thermostat(target, tau)
        last = None
        for step in range(6):
            ctx.step(1)
            now, kin = ctx.get_state()["v"], ctx.ledger()["kinetic"]
            if step:
                T = np.longdouble(2.0 / 3.0 / 8.61734279e-05) * np.longdouble(kin) / n
                want = np.sqrt(1 + np.longdouble(dt) / np.longdouble(tau) * (np.longdouble(target) / T - 1))
                assert np.abs(now / (last * want) - 1).max() <= 6 * 2.0 ** -53, step
            last = now
