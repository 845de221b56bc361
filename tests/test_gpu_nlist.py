"""Neighbour-list builds on geometries that stress the FP32 screens: every
build variant (cell-centric, thread-per-atom, 4- and 8-lane groups) against
the FP64 oracle's neighbour set, exactly, and the forces of all variants
bitwise equal (the variants emit every row in the same order).

  lattice_ties  simple cubic with spacing Rv/2: the axial second neighbours
                sit at Rv up to the last FP64 bit, so the FP64 test decides
  far_atoms     a free-surface slab with atoms far above and below the cell
                grid (clamped into the edge cells: large cell-local
                coordinates widen the screening band)
  small_axes    periodic axes holding one and two cells (every cell with
                every image)
"""
import os

import numpy as np
import pytest

from conftest import TABLES, nbr_set

pytestmark = pytest.mark.gpu

EAM_TABLE = os.path.join(TABLES, "eam.aluminum5000")
SKIN = 0.3
MODES = (0, 1, 4, 8)


def cutoff(oc):
    return oc.Table.from_file(EAM_TABLE, "PAIR").max_range() + SKIN


def lattice_ties(rv):
    a = rv / 2.0
    m = 8
    g = np.arange(m, dtype=np.float64) * a
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return x, np.zeros(3), np.full(3, m * a), (1, 1, 1)


def far_atoms(rv):
    from objectmd_gb300 import inputs

    x, _, (lo, hi) = inputs.eam_aluminium(ncell=5, a=4.05, sigma=0.05, temp=300.0, seed_pos=5, seed_vel=6)
    keep = x[:, 2] < 3 * 4.05
    x = x[keep]
    hi = np.array(hi, dtype=np.float64)
    hi[2] = 3 * 4.05
    extra = np.array([[5.0, 6.0, 40.0], [5.0, 6.0, 42.5], [9.0, 1.0, -35.0], [1.0, 1.0, 400.0]])
    return np.concatenate([x, extra]), np.asarray(lo, dtype=np.float64), hi, (1, 1, 0)


def small_axes(rv):
    rng = np.random.default_rng(9)
    L = np.array([1.5 * rv, 2.5 * rv, 4.0 * rv])
    n = int(0.05 * np.prod(L))
    return rng.uniform(0.0, 1.0, (n, 3)) * L, np.zeros(3), L, (1, 1, 1)


def context(omdg, x, lo, hi, periodic, mode):
    from objectmd_gb300 import inputs

    ctx = omdg.Context(0)
    ctx.set_box(lo, hi, tuple(bool(p) for p in periodic))
    ctx.set_atoms(x, np.zeros_like(x), masses=[inputs.md_mass("aluminum")], znum=[13.0])
    ctx.add_eam(EAM_TABLE)
    ctx.set_neighbor(SKIN, 1)
    ctx.set_launch("build_lanes", mode)
    return ctx


@pytest.mark.parametrize("geometry", [lattice_ties, far_atoms, small_axes])
def test_build_variants_match_oracle_and_each_other(omdg_lib, oracle_lib, geometry):
    oc = oracle_lib
    rv = cutoff(oc)
    x, lo, hi, periodic = geometry(rv)
    ref = nbr_set(*oc.neighbors(oc.make_box(lo, hi, periodic), x, rv))
    assert ref
    forces = []
    for mode in MODES:
        with context(omdg_lib, x, lo, hi, periodic, mode) as ctx:
            ctx.compute_forces()
            assert nbr_set(*ctx.neighbors()) == ref, mode
            forces.append(ctx.get_state()["f"])
    for mode, f in zip(MODES[1:], forces[1:]):
        assert np.array_equal(f, forces[0]), mode


# Rows longer than a thread's shared-memory column (64 entries at one thread
# per centre, 32 per run of cells at eight), at the widths where the candidate
# loop's last group is ragged, for one and two atom types.
@pytest.mark.parametrize("n,side,ntypes", [(1500, 3.05, 1), (3001, 3.3, 1), (2003, 2.2, 2), (700, 1.4, 1)])
def test_rows_past_the_shared_columns(omdg_lib, oracle_lib, n, side, ntypes):
    from objectmd_gb300 import inputs

    oc = oracle_lib
    rv = cutoff(oc)
    rng = np.random.default_rng(n)
    L = np.full(3, side * rv)
    x = rng.uniform(0.0, 1.0, (n, 3)) * L
    ref = nbr_set(*oc.neighbors(oc.make_box(np.zeros(3), L, (1, 1, 1)), x, rv, 2048))
    assert len(ref) > 100 * n
    for mode in (1, 8):
        with omdg_lib.Context(0) as ctx:
            ctx.set_box(np.zeros(3), L, (True, True, True))
            ctx.set_atoms(x, types=rng.integers(0, ntypes, n), masses=[inputs.md_mass("aluminum")] * ntypes,
                          znum=[13.0] * ntypes)
            ctx.add_eam(EAM_TABLE)
            ctx.set_neighbor(SKIN, 1)
            ctx.set_launch("build_lanes", mode)
            ctx.build_neighbors()
            assert nbr_set(*ctx.neighbors()) == ref, mode


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 8192, 8193, 16384, 16385, 32768, 32769])
def test_small_sort_edges(omdg_lib, oracle_lib, n):
    """The one-kernel sort at the edges of its blocks and of the atoms a thread
    moves, and the general path one atom past it: the list is the oracle's, and
    after steps that each rebuild (the sort looks for their request) so is the
    list of the new positions, with every atom still under its own id."""
    from objectmd_gb300 import inputs

    oc = oracle_lib
    side = max(3, int(np.ceil((n / 8) ** (1.0 / 3.0))))
    x, v, (lo, hi) = inputs.diamond_silicon(ncell=side, a=5.431, sigma=0.05, temp=600.0, seed_pos=3, seed_vel=4)
    pick = np.random.default_rng(n).permutation(len(x))[:n]  # vacancies, and an order that is not the cells'
    x, v = x[pick], v[pick]
    box = oc.make_box(lo, hi, (1, 1, 1))
    rv = 2.85 + SKIN
    with omdg_lib.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
        ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
        ctx.set_neighbor(SKIN, 1)
        ctx.compute_forces()
        assert nbr_set(*ctx.neighbors()) == nbr_set(*oc.neighbors(box, x, rv))
        ctx.set_timestep(0.001)
        b0 = ctx.stats()["rebuilds"]
        ctx.step(3)
        assert ctx.stats()["rebuilds"] - b0 >= 3
        st = ctx.get_state()
        ctx.compute_forces()
        assert nbr_set(*ctx.neighbors()) == nbr_set(*oc.neighbors(box, st["x"], rv))
    d = st["x"] - x
    d -= (np.asarray(hi) - np.asarray(lo)) * np.round(d / (np.asarray(hi) - np.asarray(lo)))
    assert np.abs(d).max() < 0.5  # three femtoseconds: no atom took another's place


@pytest.mark.parametrize("ncell", [4, 17])
def test_steps_in_one_graph(omdg_lib, ncell):
    """Steps taken one call at a time, and in calls long enough for the graph
    of several steps (with single ones left over), are the same trajectory and
    ledger bit for bit; 512 atoms (the rebuild's kernels look for its request)
    and 39,304 (the conditional node)."""
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=0.05, temp=1500.0, seed_pos=3, seed_vel=4)
    out = []
    for calls in ([1] * 131, [70, 61], [65, 8, 9, 7, 42]):
        with omdg_lib.Context(0) as ctx:
            ctx.set_box(lo, hi)
            ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
            ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
            ctx.set_neighbor(SKIN, 0)
            ctx.set_timestep(0.001)
            ctx.set_thermostat(1200.0, 0.1)
            for k in calls:
                ctx.step(k)
            st = ctx.get_state()
            out.append((st["x"], st["v"], st["f"], ctx.ledger()["energy"], ctx.stats()["rebuilds"]))
    assert out[0][4] > 5
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))


@pytest.mark.parametrize("n", [255, 256, 257, 512, 513, 1024, 1025])
def test_ledger_of_one_block_and_several(omdg_lib, n):
    """The kick's ledger row at the edges of its one-block forms: kinetic and
    potential energy against FP64 sums over the atoms (their own FP32 parts:
    2^-40 relative)."""
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=6, a=5.431, sigma=0.05, temp=900.0, seed_pos=3, seed_vel=4)
    x, v = x[:n], v[:n]
    mass = inputs.md_mass("silicon")
    with omdg_lib.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_atoms(x, v, masses=[mass], znum=[14.0])
        ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
        ctx.set_neighbor(SKIN, 0)
        ctx.set_timestep(0.001)
        ctx.step(2)
        st = ctx.get_state()
        k, p = ctx.ledger_history(2)
    assert abs(k[-1] - 0.5 * mass * (st["v"] ** 2).sum()) <= 2.0 ** -40 * abs(k[-1])
    assert abs(p[-1] - st["pot"].astype(np.float64).sum()) <= 2.0 ** -40 * abs(p[-1])


@pytest.mark.parametrize("kind,ncell,every", [("tersoff", 4, 0), ("tersoff", 17, 0), ("tersoff", 4, 5), ("tersoff", 17, 5),
                                              ("sw", 5, 0), ("eam", 6, 0), ("eam", 22, 4)])
def test_kick_and_drift_in_one_kernel(omdg_lib, kind, ncell, every):
    """Without a thermostat the steps inside one graph join a step's kick and the
    next one's drift: the same trajectory and ledger, bit for bit, as single
    steps, with displacement and periodic rebuilds, in boxes of both forms."""
    from objectmd_gb300 import inputs

    if kind == "eam":
        x, v, (lo, hi) = inputs.eam_aluminium(ncell=ncell, a=4.05, sigma=0.05, temp=900.0, seed_pos=3, seed_vel=4)
    else:
        x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=0.05, temp=1500.0, seed_pos=3, seed_vel=4)
    out = []
    for calls in ([1] * 110, [70, 40], [66, 9, 8, 27]):
        with omdg_lib.Context(0) as ctx:
            ctx.set_box(lo, hi)
            ctx.set_atoms(x, v, masses=[inputs.md_mass("aluminum" if kind == "eam" else "silicon")],
                          znum=[13.0 if kind == "eam" else 14.0])
            if kind == "eam":
                ctx.add_eam(EAM_TABLE)
            elif kind == "sw":
                ctx.add_sw(os.path.join(TABLES, "sw.silicon"))
            else:
                ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
            ctx.set_neighbor(SKIN, every)
            ctx.set_timestep(0.001)
            for k in calls:
                ctx.step(k)
            st = ctx.get_state()
            out.append((st["x"], st["v"], st["f"], st["pot"], ctx.ledger()["energy"], ctx.ledger()["virial"],
                        ctx.stats()["rebuilds"]))
    assert out[0][-1] > 3
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))


@pytest.mark.parametrize("ncell", [4, 17])
def test_the_graph_of_steps_runs(omdg_lib, ncell):
    """Calls of eight steps take the graph of eight once 64 steps were replayed,
    with seven kicks and drifts of each eight in one kernel: seven launches
    fewer.  What a call itself launches comes from calls of two and of four
    steps; the rebuilds are the same in every run."""
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=0.05, temp=1500.0, seed_pos=3, seed_vel=4)
    launches, rebuilds = [], []
    for size in (2, 4, 8):
        with omdg_lib.Context(0) as ctx:
            ctx.set_box(lo, hi)
            ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
            ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
            ctx.set_neighbor(SKIN, 0)
            ctx.set_timestep(0.001)
            for _ in range(64):
                ctx.step(1)
            for _ in range(64 // size):
                ctx.step(size)
            launches.append(ctx.stats()["launches"])
            rebuilds.append(ctx.stats()["rebuilds"])
    assert rebuilds[0] == rebuilds[1] == rebuilds[2]
    per_call = (launches[0] - launches[1]) / 16
    assert launches[1] - launches[2] == 8 * per_call + 7 * 8


@pytest.mark.parametrize("offset", [(0.0, 0.0, 0.0), (3.0e4, -7.0e5, 12.5), (1.0e6, 1.0e6, 1.0e6), (-5.0e8, 0.0, 3.0e3)])
def test_boxes_far_from_the_origin(omdg_lib, oracle_lib, offset):
    """The list is the oracle's wherever the box lies, from one thread and from
    eight lanes a centre, as a box and as two replicas."""
    from objectmd_gb300 import inputs

    oc = oracle_lib
    rv = cutoff(oc)
    x, _, (lo, hi) = inputs.eam_aluminium(ncell=6, a=4.05, sigma=0.1, temp=0.0, seed_pos=31, seed_vel=32)
    offset = np.asarray(offset)
    x, lo, hi = x + offset, np.asarray(lo) + offset, np.asarray(hi) + offset
    ref = nbr_set(*oc.neighbors(oc.make_box(lo, hi, (1, 1, 0)), x, rv))
    for mode in (1, 8):
        with context(omdg_lib, x, lo, hi, (1, 1, 0), mode) as ctx:
            ctx.build_neighbors()
            assert nbr_set(*ctx.neighbors()) == ref
    n = len(x)
    with omdg_lib.Context(0) as ctx:
        far = np.array([2.0e5, 0.0, -4.0e4])
        ctx.set_replicas([n, n], [lo, lo + far], [hi, hi + far], (1, 1, 0))
        ctx.set_atoms(np.vstack([x, x + far]), masses=[inputs.md_mass("silicon")], znum=[14.0])
        ctx.add_tersoff(os.path.join(TABLES, "tersoff.silicon27"))
        ctx.set_neighbor(rv - ctx.max_cut_radius(), 1)
        ctx.build_neighbors()
        rows = nbr_set(*ctx.neighbors())
    assert {q for q in rows if q[0] < n} == ref
    moved = nbr_set(*oc.neighbors(oc.make_box(lo + far, hi + far, (1, 1, 0)), x + far, rv))
    assert {(i - n, j - n, *s) for i, j, *s in rows if i >= n} == moved


def test_a_build_takes_as_long_far_from_the_origin(omdg_lib):
    """256,000 atoms at the origin and 10^6 A away: from the box's corner the
    FP32 screen leaves as few pairs to the FP64 test (from the origin a build
    there took 14 times as long)."""
    import torch

    from objectmd_gb300 import inputs

    x, lo, hi = inputs.fcc((40, 40, 40), 4.05)
    x = inputs.perturb(x, 0.05, 5, lo, hi)
    best = []
    for offset in (0.0, 1.0e6):
        with omdg_lib.Context(0) as ctx:
            ctx.set_box(np.asarray(lo) + offset, np.asarray(hi) + offset)
            ctx.set_atoms(x + offset, masses=[inputs.md_mass("aluminum")], znum=[13.0])
            ctx.add_eam(EAM_TABLE)
            ctx.set_neighbor(SKIN, 0)
            ctx.build_neighbors()
            stream = torch.cuda.ExternalStream(ctx.stream())
            times = []
            for _ in range(10):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                ctx.build_neighbors()
                b.record(stream)
                b.synchronize()
                times.append(a.elapsed_time(b))
            best.append(min(times))
    assert best[1] < 3.0 * best[0], best
