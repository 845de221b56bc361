"""Row overflow in the three-body passes and in replicas.

As in test_gpu_overflow.py: atoms driven toward the centre lengthen the rows
past a tight capacity inside queued steps, and the recovered run has to be the
run with ample rows, bit for bit.  Here the rebuild is the conditional node of
a box above 32,768 atoms, in the graph of eight steps with joined kicks and
drifts, or the kernels of every step in a small box; the rows have reverse
slots (stale for the entries that an overflowing row dropped) and centres past
the register path, which queue.  A recovery rebuilds every replica, an
ensemble with ample rows only those that moved: another order of the sums, and
positions to 1e-5 A as in the other replica tests.
"""
import os

import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu

TERSOFF = os.path.join(TABLES, "tersoff.silicon27")
SW = os.path.join(TABLES, "sw.silicon")


def converging_silicon(ncell, radius, rate, seed=61):
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=0.05, temp=300.0, seed_pos=seed,
                                            seed_vel=seed + 1)
    d = x - 0.5 * (np.asarray(lo) + np.asarray(hi))
    inner = np.linalg.norm(d, axis=1) < radius
    v = v.copy()
    v[inner] -= rate * d[inner]
    return x, v, lo, hi


def context(omdg, kind, x, v, lo, hi, capacity):
    from objectmd_gb300 import inputs

    ctx = omdg.Context(0)
    ctx.set_box(lo, hi)
    ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
    if kind == "sw":
        ctx.add_sw(SW)
    else:
        ctx.add_tersoff(TERSOFF)
    if capacity:
        ctx.set_launch("nbr_capacity", capacity)
    ctx.set_neighbor(0.3, 0)
    ctx.set_timestep(0.0005)
    return ctx


def longest(ctx):
    return int(np.diff(ctx.neighbors()[0]).max())


@pytest.mark.parametrize("kind,ncell", [("tersoff", 17), ("tersoff", 6), ("sw", 6)])
def test_three_body_rows_overflow(omdg_lib, kind, ncell):
    case = converging_silicon(ncell, 12.0, 1.2)
    first, second = 72, 160
    with context(omdg_lib, kind, *case, 0) as ctx:
        capacity = 0
        for _ in range(first):  # the longest row of any list of the first call
            ctx.step(1)
            capacity = max(capacity, longest(ctx))
    out = []
    for cap in (0, capacity):
        with context(omdg_lib, kind, *case, cap) as ctx:
            ctx.step(first)
            k0, p0 = ctx.ledger_history()
            ctx.step(second)  # replayed by the graph of eight steps
            k1, p1 = ctx.ledger_history()
            st = ctx.get_state()
            out.append((st["x"], st["v"], st["f"], st["pot"], np.concatenate([k0, k1]), np.concatenate([p0, p1]),
                        np.diff(ctx.neighbors()[0])))
            wide = ctx.wide_centres()
    assert out[1][6].max() > capacity  # the second call's rows outgrew it
    assert wide > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("sizes", [(4, 6, 5), (5, 17)])
def test_a_replica_rebuilt_alone_overflows(omdg_lib, sizes):
    from objectmd_gb300 import inputs

    parts = [converging_silicon(n, 12.0, 1.2 if k == 1 else 0.0, 71 + k) for k, n in enumerate(sizes)]
    natoms = [len(p[0]) for p in parts]

    def run(capacity, watch):
        with omdg_lib.Context(0) as ctx:
            ctx.set_replicas(natoms, [p[2] for p in parts], [p[3] for p in parts], (1, 1, 1))
            ctx.set_atoms(np.vstack([p[0] for p in parts]), np.vstack([p[1] for p in parts]),
                          masses=[inputs.md_mass("silicon")], znum=[14.0])
            ctx.add_tersoff(TERSOFF)
            if capacity:
                ctx.set_launch("nbr_capacity", capacity)
            ctx.set_neighbor(0.3, 0)
            ctx.set_timestep(0.0005)
            rows = 0
            for _ in range(72 if watch else 1):
                ctx.step(1 if watch else 72)
                rows = max(rows, longest(ctx))
            if not watch:
                ctx.step(160)
            return ctx.get_state()["x"], rows, longest(ctx), ctx.replica_builds(len(parts))

    capacity = run(0, True)[1]
    ample, _, _, builds = run(0, False)
    tight, _, grown, _ = run(capacity, False)
    assert max(builds) > min(builds)  # partial rebuilds took place
    assert grown > capacity
    at = 0
    for n, p in zip(natoms, parts):
        L = np.asarray(p[3]) - np.asarray(p[2])
        d = tight[at:at + n] - ample[at:at + n]
        assert np.abs(d - L * np.round(d / L)).max() <= 1e-5
        at += n


def test_errors_of_discarded_steps_do_not_stop_the_recovery(omdg_lib):
    """Many steps after the overflow in the same call: truncated rows may drive
    atoms anywhere, to non-finite positions too, but those steps are replayed.
    The same call ten times, since what a dropped slot holds is left open."""
    case = converging_silicon(6, 12.0, 1.2)
    with context(omdg_lib, "sw", *case, 0) as ctx:
        ctx.step(2)
        capacity = longest(ctx)
        ctx.step(198)
        ample = ctx.get_state()
    for _ in range(10):
        with context(omdg_lib, "sw", *case, capacity) as ctx:
            ctx.step(2)
            ctx.step(198)
            st = ctx.get_state()
            assert longest(ctx) > capacity
        for k in ("x", "v", "f", "pot"):
            assert np.array_equal(st[k], ample[k]), k


@pytest.mark.parametrize("collide", [True, False])
def test_an_error_before_the_overflow_stands(omdg_lib, collide):
    """Two argon atoms shot at each other pass the table's first knot before the
    call's first rebuild (a skin of 4 A, a rebuild every 200 steps); there the
    rows, all alike in the crystal, overflow, as they do without the shot.  The table's error is reported, not lost in a replay."""
    from objectmd_gb300 import inputs

    table = os.path.join(TABLES, "pair.lj.argon")
    x, v, (lo, hi) = inputs.lj_argon(ncell=8, temp=120.0)
    if collide:
        x = np.vstack([x, [[1.3, 1.3, 1.3], [4.3, 1.3, 1.3]]])
        v = np.vstack([v, [[120.0, 0.0, 0.0], [-120.0, 0.0, 0.0]]])
        keep = np.linalg.norm(x[:-2] - np.array([2.8, 1.3, 1.3]), axis=1) > 4.5
        keep = np.append(keep, [True, True])
        x, v = x[keep], v[keep]

    def context(capacity):
        ctx = omdg_lib.Context(0)
        ctx.set_box(lo, hi)
        ctx.set_atoms(x, v, masses=[inputs.md_mass("argon")], znum=[18.0])
        ctx.add_pair_table(table)
        if capacity:
            ctx.set_launch("nbr_capacity", capacity)
        ctx.set_neighbor(4.0, 200)
        ctx.set_timestep(0.0005)
        return ctx

    with context(0) as ctx:
        ctx.build_neighbors()
        capacity = longest(ctx)
    with context(capacity) as ctx:
        if collide:
            with pytest.raises(omdg_lib.OMDGError) as err:
                ctx.step(600)
            assert err.value.code == omdg_lib.OMDG_ERANGE
        else:
            ctx.step(600)
            assert longest(ctx) > capacity


def test_more_neighbours_than_a_centre_holds_is_an_error(omdg_lib):
    """Silicon driven together until a centre has more than the 24 neighbours
    inside the cutoff that a three-body pass holds (with room in the rows): an
    error, which no growth of the rows would mend."""
    from objectmd_gb300 import inputs

    x, lo, hi = inputs.diamond((6, 6, 6), 4.62)
    d = x - 0.5 * (np.asarray(lo) + np.asarray(hi))
    inner = np.linalg.norm(d, axis=1) < 12.0
    v = np.zeros_like(x)
    v[inner] = -3.0 * d[inner]
    with context(omdg_lib, "sw", x, v, lo, hi, 400) as ctx:
        with pytest.raises(omdg_lib.OMDGError) as err:
            ctx.step(200)
        assert err.value.code == omdg_lib.OMDG_ESTATE
