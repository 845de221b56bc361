"""Stillinger-Weber and Tersoff on the GPU.

SW is checked against the reference's own SW with every triplet evaluated
(the sw.cpp:261 guard removed, tests/golden), Tersoff against the FP64 C
oracle (the reference's tersoff.h does not compile).  Tolerance as for EAM:
norm-wise relative force error <= 1e-5, components within
1e-5 * max|f| + 1e-6 eV/A, per-atom energies within 2e-6 eV.
"""
import os

import numpy as np
import pytest

from conftest import TABLES, load_case, nbr_set

pytestmark = pytest.mark.gpu

SW_FILE = os.path.join(TABLES, "sw.silicon")
TERSOFF_FILE = os.path.join(TABLES, "tersoff.silicon27")


def check(f, fref, e=None, eref=None, etol=2e-6):
    rel = np.linalg.norm(f - fref) / np.linalg.norm(fref)
    assert rel <= 1e-5, rel
    assert np.abs(f - fref).max() <= 1e-5 * np.abs(fref).max() + 1e-6
    if e is not None:
        err = np.abs(e - eref)
        assert err.max() <= etol, (err.max(), int(err.argmax()), float(eref[err.argmax()]))


def si_context(omdg, x, v, lo, hi, kind):
    from objectmd_gb300 import inputs

    ctx = omdg.Context(0)
    ctx.set_box(lo, hi)
    ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
    if kind == "sw":
        ctx.add_sw(SW_FILE)
    else:
        ctx.add_tersoff(TERSOFF_FILE)
    ctx.set_neighbor(0.3, 1)
    return ctx


@pytest.mark.parametrize("case", ["sw_si_216", "sw_si_1000"])
def test_sw_matches_reference_every_triplet(omdg_lib, case):
    d = load_case(case)
    with si_context(omdg_lib, d["x0"], d["v0"], d["box_lo"], d["box_hi"], "sw") as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
        mine = nbr_set(*ctx.neighbors())
    check(st["f"], d["f"], st["pot"], d["pot"])
    assert mine == set(map(tuple, d["nbr"].tolist()))


def test_sw_large_vs_oracle(omdg_lib, oracle_lib):
    from objectmd_gb300 import inputs

    oc = oracle_lib
    x, v, (lo, hi) = inputs.diamond_silicon(ncell=8, a=5.431, sigma=0.03, temp=1000.0, seed_pos=41, seed_vel=42)
    box = oc.make_box(lo, hi, (1, 1, 1))
    p = oc.SWParam(eps=2.1683, A=7.049556277, B=0.6022245584, p=4, q=0, sigma=2.0951, a=1.80, lam=21.0, gamma=1.2,
                   icos0=-3.0, usezbl=1, sx0=1.2107, sx1=1.8456, sa0=335.0594, sa1=-492.3905, sa2=244.5280,
                   sa3=-41.2347, z1=14, z2=14)
    fref, eref, _ = oc.sw(box, x, oc.neighbors(box, x, 2.0951 * 1.8 + 0.3), p)
    with si_context(omdg_lib, x, v, lo, hi, "sw") as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
    check(st["f"], fref, st["pot"], eref)


@pytest.mark.parametrize("ncell,sigma,temp", [(3, 0.06, 1000.0), (8, 0.03, 1000.0)])
def test_tersoff_vs_oracle(omdg_lib, oracle_lib, ncell, sigma, temp):
    from objectmd_gb300 import inputs

    oc = oracle_lib
    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=sigma, temp=temp, seed_pos=8, seed_vel=9)
    box = oc.make_box(lo, hi, (1, 1, 1))
    p = oc.TersoffParam(A=3264.7, B=95.373, lambda1=3.2394, lambda2=1.3258, lambda3=1.3258, beta=0.33675, n=22.956,
                        c=4.8381, d=2.0417, h=0.0, R=2.7, D=0.15)
    nb = oc.neighbors(box, x, 2.85 + 0.3)
    fref, eref, _ = oc.tersoff(box, x, nb, p)
    with si_context(omdg_lib, x, v, lo, hi, "tersoff") as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
        assert nbr_set(*ctx.neighbors()) == nbr_set(*nb)
    # bond energies cancel (f_R - b f_A): FP32 exp/pow leave ~1e-6 relative per atom
    check(st["f"], fref, st["pot"], eref, etol=5e-6)


def interstitial_silicon(ncell, seed):
    """Diamond Si with three atoms planted on tetrahedral interstitial sites
    ((1/2, 1/2, 1/2) of a cubic cell, relative to its first site): each has 4 neighbours at sqrt(3)/4 a
    and 6 at a/2, inside both cutoffs, and its 4 nearest hosts gain a fifth."""
    from objectmd_gb300 import inputs

    a = 5.431
    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=a, sigma=0.03, temp=1000.0, seed_pos=seed,
                                            seed_vel=seed + 1)
    cells = np.array([[1, 1, 1], [ncell // 2, 2, ncell - 2], [ncell - 2, ncell // 2, 3]], dtype=np.float64)
    extra = np.array(lo)[None, :] + (cells + 0.5) * a + a / 8  # lattice sites are offset by a/8
    rng = np.random.default_rng(seed + 2)
    x = np.vstack([x, extra + rng.normal(0.0, 0.03, extra.shape)])
    v = np.vstack([v, np.zeros_like(extra)])
    return x, v, lo, hi


@pytest.mark.parametrize("kind", ["sw", "tersoff"])
def test_dense_centres_take_the_wide_kernel(omdg_lib, oracle_lib, kind):
    """Centres with more in-cutoff neighbours than the register path holds go
    to k_sw_wide / k_tersoff_wide; their forces must still match the oracle,
    and the queue count shows that the dense pass ran."""
    oc = oracle_lib
    x, v, lo, hi = interstitial_silicon(6, 61)
    box = oc.make_box(lo, hi, (1, 1, 1))
    if kind == "sw":
        p = oc.SWParam(eps=2.1683, A=7.049556277, B=0.6022245584, p=4, q=0, sigma=2.0951, a=1.80, lam=21.0,
                       gamma=1.2, icos0=-3.0, usezbl=1, sx0=1.2107, sx1=1.8456, sa0=335.0594, sa1=-492.3905,
                       sa2=244.5280, sa3=-41.2347, z1=14, z2=14)
        fref, eref, _ = oc.sw(box, x, oc.neighbors(box, x, 2.0951 * 1.8 + 0.3), p)
        # an interstitial's energy sums ~45 three-body terms of up to ~10 eV in
        # FP32 (measured on a GB300: 5.8e-6 eV); lattice atoms stay below 3e-7
        etol = 2e-5
    else:
        p = oc.TersoffParam(A=3264.7, B=95.373, lambda1=3.2394, lambda2=1.3258, lambda3=1.3258, beta=0.33675,
                            n=22.956, c=4.8381, d=2.0417, h=0.0, R=2.7, D=0.15)
        fref, eref, _ = oc.tersoff(box, x, oc.neighbors(box, x, 2.85 + 0.3), p)
        etol = 5e-6
    with si_context(omdg_lib, x, v, lo, hi, kind) as ctx:
        ctx.compute_forces()
        st = ctx.get_state()
        wide = ctx.wide_centres()
    assert wide >= 3, wide
    check(st["f"], fref, st["pot"], eref, etol=etol)


@pytest.mark.parametrize("kind,ncell,skin", [("sw", 6, 3.0), ("sw", 20, 0.3), ("sw", 20, 3.0), ("tersoff", 6, 3.0),
                                             ("tersoff", 13, 0.3), ("tersoff", 13, 3.0)])
def test_both_forms_over_long_rows(omdg_lib, oracle_lib, kind, ncell, skin):
    """Eight lanes for every centre (1,731 atoms), and a thread a centre with
    eight lanes for the queued ones (17,579 Tersoff and 64,003 SW atoms), over
    rows of one word of hit bits and of three (a skin of 3 A: some 65 and 45
    entries, up to 90)."""
    oc = oracle_lib
    x, v, lo, hi = interstitial_silicon(ncell, 71)
    box = oc.make_box(lo, hi, (1, 1, 1))
    if kind == "sw":
        p = oc.SWParam(eps=2.1683, A=7.049556277, B=0.6022245584, p=4, q=0, sigma=2.0951, a=1.80, lam=21.0,
                       gamma=1.2, icos0=-3.0, usezbl=1, sx0=1.2107, sx1=1.8456, sa0=335.0594, sa1=-492.3905,
                       sa2=244.5280, sa3=-41.2347, z1=14, z2=14)
        fref, eref, _ = oc.sw(box, x, oc.neighbors(box, x, 2.0951 * 1.8 + 0.3), p)
        etol = 2e-5
    else:
        p = oc.TersoffParam(A=3264.7, B=95.373, lambda1=3.2394, lambda2=1.3258, lambda3=1.3258, beta=0.33675,
                            n=22.956, c=4.8381, d=2.0417, h=0.0, R=2.7, D=0.15)
        fref, eref, _ = oc.tersoff(box, x, oc.neighbors(box, x, 2.85 + 0.3), p)
        etol = 5e-6
    with si_context(omdg_lib, x, v, lo, hi, kind) as ctx:
        ctx.set_neighbor(skin, 1)
        ctx.compute_forces()
        st = ctx.get_state()
        wide = ctx.wide_centres()
        ctx.compute_forces()
        again = ctx.get_state()
    assert wide >= 3, wide
    check(st["f"], fref, st["pot"], eref, etol=etol)
    assert np.array_equal(st["f"], again["f"]) and np.array_equal(st["pot"], again["pot"])


def test_tersoff_forms_agree_on_a_repeated_cell(omdg_lib):
    """8,112 atoms (eight lanes a centre) and the same cell three times along z
    (24,336 atoms, a thread a centre).  A relative vector is the FP32 rounding
    of the same difference but for 1e-14, so a component may be off by a unit
    in its last place (2.4e-7 A): with four bonds of at most 50 eV/A^2 a force
    moves by 5e-5 eV/A at most, and an energy, with bond forces of at most 10
    eV/A, by 1e-5 eV."""
    from objectmd_gb300 import inputs

    a, n = 5.431, (13, 13, 6)
    x, lo, hi = inputs.diamond(n, a)
    x = inputs.perturb(x, 0.05, 5, lo, hi, (True, True, True))
    up = np.array([0.0, 0.0, hi[2] - lo[2]])
    out = []
    for y, top in ((x, np.array(hi)), (np.vstack([x, x + up, x + 2 * up]), np.array(hi) + 2 * up)):
        with si_context(omdg_lib, y, np.zeros_like(y), lo, top, "tersoff") as ctx:
            ctx.compute_forces()
            out.append(ctx.get_state())
    for k in range(3):
        part = slice(k * len(x), (k + 1) * len(x))
        assert np.abs(out[1]["f"][part] - out[0]["f"]).max() <= 5e-5
        assert np.abs(out[1]["pot"][part] - out[0]["pot"]).max() <= 1e-5


def test_tersoff_nve_conserves_energy(omdg_lib):
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=4, a=5.431, sigma=0.03, temp=1000.0, seed_pos=4, seed_vel=5)
    with si_context(omdg_lib, x, v, lo, hi, "tersoff") as ctx:
        ctx.set_neighbor(0.3, 0)
        ctx.set_timestep(0.001)
        ctx.set_first_step_mode(False)
        ctx.step(1)
        e0 = ctx.ledger()["energy"]
        ctx.step(500)
        e1 = ctx.ledger()["energy"]
    assert abs(e1 - e0) / len(x) < 2e-4  # eV/atom over 0.5 ps at 1000 K


@pytest.mark.parametrize("kind,bound", [("sw", 3e-4), ("tersoff", 3e-4)])
def test_nve_drift_over_10k_steps(omdg_lib, kind, bound):
    """10^4 NVE steps of 4096 Si atoms at 1000 K, dt 1 fs, displacement-triggered
    rebuilds: the run stays finite (SW pairs at r == rc in FP32 would give
    0 * inf) and the energy drift stays below `bound` eV/atom (measured on a
    GB300: SW 7.5e-5, Tersoff 6.4e-5)."""
    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=8, a=5.431, sigma=0.03, temp=1000.0, seed_pos=4, seed_vel=5)
    with si_context(omdg_lib, x, v, lo, hi, kind) as ctx:
        ctx.set_neighbor(0.3, 0)
        ctx.set_timestep(0.001)
        ctx.set_first_step_mode(False)
        ctx.step(1)
        e0 = ctx.ledger()["energy"]
        ctx.step(10000)
        e1 = ctx.ledger()["energy"]
    assert np.isfinite(e1)
    assert abs(e1 - e0) / len(x) < bound


@pytest.mark.parametrize("ncell", [6, 11])
def test_tersoff_forms_have_the_same_bits(omdg_lib, tmp_path, ncell):
    """The same box through both forms: with a surrogate whose training range
    holds no atom, every centre takes the masked Tersoff pass (a thread a
    centre, the crowded ones queued), where plain Tersoff takes eight lanes for
    every centre of a box this small (1,731 atoms; 10,651 take the threads, and
    the pass is its own check).  The list ranges are made equal: rows and order
    of the sums are the same, and the surrogate's further hits add zeros."""
    x, v, lo, hi = interstitial_silicon(ncell, 71)
    model = str(tmp_path / "none.nn")
    with omdg_lib.Network(0) as net:
        net.set_normalization(np.zeros(32), np.ones(32), np.full(32, 1e9), np.full(32, 2e9))
        net.set_weights(np.zeros(6337))
        net.save(model)
    out = []
    for surrogate in (True, False):
        with si_context(omdg_lib, x, v, lo, hi, "tersoff") if not surrogate else omdg_lib.Context(0) as ctx:
            if surrogate:
                from objectmd_gb300 import inputs

                ctx.set_box(lo, hi)
                ctx.set_atoms(x, v, masses=[inputs.md_mass("silicon")], znum=[14.0])
                ctx.add_nn(model, TERSOFF_FILE)
                reach = ctx.max_cut_radius() + 0.3
            ctx.set_neighbor(reach - ctx.max_cut_radius(), 1)
            ctx.compute_forces()
            if surrogate:
                assert ctx.nn_fallback_atoms() == len(x)
            assert ctx.wide_centres() >= 3
            st = ctx.get_state()
            out.append((st["f"], st["pot"], st["vir"], np.concatenate(ctx.neighbors())))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind,ncell", [("sw", 6), ("tersoff", 6), ("tersoff", 34)])
def test_forces_go_out_beside_the_kick(omdg_lib, kind, ncell):
    """omdg_step_io with forces: the slot gather stays a kernel of its own, so
    that they need not wait for the kick (with velocities too, in a box above
    2,048 atoms a SM): one launch more than a step that only velocities leave.
    Values as get_state gives them."""
    import torch

    from objectmd_gb300 import inputs

    x, v, (lo, hi) = inputs.diamond_silicon(ncell=ncell, a=5.431, sigma=0.03, temp=300.0, seed_pos=4, seed_vel=5)
    n = len(x)
    out = {k: torch.empty((n, 3), dtype=torch.float64).pin_memory().numpy() for k in ("x_out", "v_out", "f_out")}
    launches = {}
    with si_context(omdg_lib, x, v, lo, hi, kind) as ctx:
        ctx.set_neighbor(1.0, 0)
        ctx.set_timestep(0.0001)
        for want in (("v_out",), ("f_out",), ("x_out", "v_out"), ("x_out", "v_out", "f_out")):
            ctx.step_io(1, **{k: out[k] for k in want})
            before = ctx.stats()
            ctx.step_io(1, **{k: out[k] for k in want})
            after = ctx.stats()
            assert after["rebuilds"] == before["rebuilds"]
            launches[want] = after["launches"] - before["launches"]
            st = ctx.get_state()
            for k in want:
                assert np.array_equal(out[k], st[k[0]]), (want, k)
    assert launches[("f_out",)] == launches[("v_out",)] + 1
    # f beside the kick is a launch and a gather more, f with v after it nothing
    apart = n >= 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    assert launches[("x_out", "v_out", "f_out")] == launches[("x_out", "v_out")] + (2 if apart else 0)
