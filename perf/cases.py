"""The work this library is used for, as measurable cases.

Each case is one pass of a program that uses the Python binding: molecular
dynamics that takes a frame every few steps, the reference application's
hand-over of its whole state every step, force evaluations of unrelated
snapshots, the impact ensemble, the heat solver, and the surrogate's training.
Contexts run with the library's default launch shapes, as the drop-in
integrator uses them (it never calls the autotuner).

`exact` restates every path in FP64 torch from the published formulas and the
table files alone.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TABLES = os.path.join(ROOT, "tests", "golden", "tables")
EAM_AL = os.path.join(TABLES, "eam.aluminum5000")
LJ_AR = os.path.join(TABLES, "pair.lj.argon")
AR_SI = os.path.join(TABLES, "pair.ar-si.zbl")
TERSOFF = os.path.join(TABLES, "tersoff.silicon27")
SW = os.path.join(TABLES, "sw.silicon")
NN_MODEL = os.path.join(ROOT, "objectmd_gb300", "models", "nn_tersoff_si.nn")

KB = 8.61734279e-05           # eV/K
AMU = 9.64853397731809e3      # amu per eV ps^2 / A^2
MASS = {"al": 26.98154 / AMU, "si": 28.0855 / AMU, "ar": 39.948 / AMU}
Z = {"al": 13.0, "si": 14.0, "ar": 18.0}
VACUUM = 10.0                 # A above a free surface
SKIN = 0.3                    # A, the library's and the reference's usual list skin

#: potential -> element, lattice constant (A), atoms per cell, Gaussian displacement (A), time step (ps)
SYSTEM = {
    "eam": ("al", 4.05, 4, 0.05, 0.002),
    "lj": ("ar", 5.26, 4, 0.02, 0.001),
    "tersoff": ("si", 5.431, 8, 0.03, 0.001),
    "sw": ("si", 5.431, 8, 0.03, 0.001),
    "nn": ("si", 5.431, 8, 0.03, 0.001),
}

#: per atom: entries of its neighbour row (cutoff + skin), and the floating operations of one force evaluation
ROW = {"eam": 54, "lj": 79, "tersoff": 4, "sw": 16, "nn": 4}
FORCE_FLOPS = {"eam": 42 * 90, "lj": 71 * 45, "tersoff": 1500, "sw": 4 * 60 + 6 * 60, "nn": 28000}


def listed():
    return [
        # the surrogate's training-set generation: 512-atom Tersoff cells held at a temperature by the
        # thermostat, one sample every 50 steps (nn_fit.generate).  The smallest box: launches count.
        dict(name="tersoff_512_sampling", kind="md", pot="tersoff", nx=4, ny=4, nz=4, temp=1500.0, tau=0.1, steps=50),
        # plain Lennard-Jones argon in FP64, the 4000-atom box every MD code starts with
        dict(name="lj_4000_fp64", kind="md", pot="lj", nx=10, ny=10, nz=10, temp=100.0, tau=0.0, steps=100),
        # the drop-in integrator's Integrate(): the application owns the atoms and hands the whole state over
        # every step, in pageable memory
        dict(name="eam_4000_handover", kind="handover", pot="eam", nx=10, ny=10, nz=10, temp=300.0),
        # the drop-in integrator's Iterate(): forces, energies and virials of configurations that are not a
        # trajectory (here a film with free surfaces and ragged sides)
        dict(name="eam_film_snapshots", kind="snapshots", pot="eam", nx=19, ny=17, nz=11, free_z=True, temp=300.0),
        # the configured EAM aluminium box, a frame every 20 steps
        dict(name="eam_256k", kind="md", pot="eam", nx=40, ny=40, nz=40, temp=300.0, tau=0.0, steps=20),
        # the large EAM box
        dict(name="eam_1m", kind="md", pot="eam", nx=64, ny=64, nz=64, temp=300.0, tau=0.0, steps=20),
        # Stillinger-Weber silicon, a ragged box
        dict(name="sw_194k", kind="md", pot="sw", nx=31, ny=27, nz=29, temp=1000.0, tau=0.0, steps=20),
        # the configured Tersoff silicon box
        dict(name="tersoff_512k", kind="md", pot="tersoff", nx=40, ny=40, nz=40, temp=1000.0, tau=0.0, steps=20),
        # the neural surrogate with its Tersoff fallback on the same box
        dict(name="nn_512k", kind="md", pot="nn", nx=40, ny=40, nz=40, temp=1000.0, tau=0.0, steps=10),
        # the configured impact ensemble: 256 uneven slabs, one Ar atom each
        dict(name="impact_256", kind="impact", nrep=256, nmin=1000, nmax=16000, sizes=6, steps=40),
        # the heat solver on a layered sample with a source, as a laser-heating run sets it up
        dict(name="heat_96x80x72", kind="heat", nx=96, ny=80, nz=72, steps=10),
        # the surrogate's fit: eight Adam steps on a batch of 16 configurations of 512 atoms
        dict(name="nn_fit_16x512", kind="fit", nconf=16, ncell=4, epochs=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "md", "handover", "snapshots", "impact", "heat", "fit"])
    if kind == "heat":
        return dict(kind=kind, nx=_log(rng, 16, 120), ny=_log(rng, 16, 90), nz=_log(rng, 8, 80), steps=rng.randint(2, 10))
    if kind == "fit":
        return dict(kind=kind, nconf=_log(rng, 4, 32), ncell=rng.choice([3, 4, 4, 5]), epochs=rng.randint(2, 8))
    if kind == "impact":
        return dict(kind=kind, nrep=_log(rng, 4, 200), nmin=1000, nmax=_log(rng, 2000, 16000), sizes=rng.randrange(1 << 20),
                    steps=rng.randint(10, 40))
    pot = "eam" if kind != "md" else rng.choice(["eam", "eam", "lj", "tersoff", "sw", "nn"])
    most = {"eam": 52, "lj": 16, "tersoff": 38, "sw": 34, "nn": 36}[pot] if kind == "md" else 24
    side = _log(rng, 5, most)  # the box's mean side, over its logarithm; the three sides differ by up to a half
    n = [max(4, int(round(side * rng.uniform(0.75, 1.25)))) for _ in range(3)]
    case = dict(kind=kind, pot=pot, nx=min(n[0], most), ny=min(n[1], most), nz=min(n[2], most))
    case["temp"] = float(rng.randint(40, 120) if pot == "lj" else rng.randint(100, 900) if pot == "eam" else rng.randint(300, 1600))
    if kind == "md":
        case["tau"] = rng.choice([0.0, 0.0, 0.1])
        case["steps"] = rng.randint(5, 20)
    if kind == "snapshots":
        case["free_z"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs

def _crystal(case, seed):
    """Positions, velocities, box of a perturbed crystal at the case's temperature."""
    elem, a, _, sigma, _ = SYSTEM[case["pot"]]
    from objectmd_gb300 import inputs

    n = (case["nx"], case["ny"], case["nz"])
    free = case.get("free_z", False)
    x, lo, hi = (inputs.fcc if SYSTEM[case["pot"]][2] == 4 else inputs.diamond)(n, a)
    x = inputs.perturb(x, sigma, 2 * seed + 1, lo, hi, (True, True, not free))
    v = inputs.maxwell_boltzmann(len(x), case["temp"], MASS[elem], 2 * seed + 2)
    if free:
        lo, hi = np.array([0.0, 0.0, -VACUUM]), np.array([hi[0], hi[1], hi[2] + VACUUM])
    return x, v, lo, hi, (True, True, not free)


def _context(case, x, v, lo, hi, periodic):
    from objectmd_gb300 import omdg

    elem, _, _, _, dt = SYSTEM[case["pot"]]
    ctx = omdg.Context(0)
    ctx.set_box(lo, hi, periodic)
    ctx.set_atoms(x, v, masses=[MASS[elem]], znum=[Z[elem]])
    if case["pot"] == "eam":
        ctx.add_eam(EAM_AL)
    elif case["pot"] == "lj":
        ctx.add_pair_table(LJ_AR, fp64=True)
    elif case["pot"] == "tersoff":
        ctx.add_tersoff(TERSOFF)
    elif case["pot"] == "sw":
        ctx.add_sw(SW)
    else:
        ctx.add_nn(NN_MODEL, TERSOFF)
    ctx.set_neighbor(SKIN, 0)
    ctx.set_timestep(dt)
    ctx.set_first_step_mode(True)
    if case.get("tau", 0.0) > 0.0:
        ctx.set_thermostat(case["temp"], case["tau"])
    return ctx


def _pinned(n):
    return torch.zeros((n, 3), dtype=torch.float64).pin_memory()


class _Frame:
    """The pinned buffers a trajectory writer takes its frames in."""

    def __init__(self, n, L):
        self.h = [_pinned(n) for _ in range(3)]
        self.np = [t.numpy() for t in self.h]
        self.L = torch.as_tensor(L, dtype=torch.float64, device="cuda")  # 0 on free axes

    def take(self, narrow):
        """The frame on the GPU, positions folded into the box.  Forces that
        are summed in single precision, and the velocities they give, are kept
        as such."""
        x, v, f = (t.cuda() for t in self.h)
        out = {"x": _fold(x, self.L), "v": v, "f": f}
        if narrow:
            out["v"], out["f"] = v.float(), f.float()
        return out


def _fold(x, L):
    return x - L * torch.floor(torch.nan_to_num(x / L, nan=0.0, posinf=0.0, neginf=0.0))


def _energies(ctx, steps, narrow):
    k, p = ctx.ledger_history(steps)
    e = np.stack([k, p], axis=1)
    return e.astype(np.float32) if narrow else e


class State:
    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        own = getattr(self, "own", None)
        if own is not None:
            own.close()


def _impact_inputs(case, seed):
    """Si diamond slabs of uneven size (fixed by the case), periodic in x and y with a free surface, each aimed at by
    one Ar atom of 10-500 eV within 30 degrees of the normal, as inputs.impact_ensemble makes them."""
    from objectmd_gb300 import inputs

    sizes, rng, a, height = np.random.default_rng(case["sizes"]), np.random.default_rng(seed), 5.431, 5.0
    xs, vs, ts, los, his = [], [], [], [], []
    for _ in range(case["nrep"]):
        want = math.exp(sizes.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        nx = max(2, int(round((want / 8.0) ** (1.0 / 3.0))))
        x, _, hi = inputs.lattice(inputs.DIAMOND_BASIS, (nx, nx, max(2, int(round(want / (8.0 * nx * nx))))), a, 0.125)
        x = x + rng.normal(0.0, 0.03, size=x.shape)
        x[:, :2] = np.mod(x[:, :2], hi[:2])
        top = float(x[:, 2].max())
        p, pv = inputs.projectile(rng.uniform(0.0, 1.0, 2) * hi[:2], top, height, rng.uniform(0.0, 30.0),
                                  rng.uniform(0.0, 360.0), math.exp(rng.uniform(math.log(10.0), math.log(500.0))), MASS["ar"])
        p[:2] = np.mod(p[:2], hi[:2])
        xs += [x, p[None]]
        vs += [inputs.maxwell_boltzmann(len(x), 300.0, MASS["si"], int(rng.integers(1 << 31))), pv[None]]
        ts += [np.zeros(len(x), dtype=np.int32), np.ones(1, dtype=np.int32)]
        los.append([0.0, 0.0, -0.5 * a])
        his.append([hi[0], hi[1], top + height + VACUUM])
    return {"natoms": np.array([len(t) + 1 for t in ts[::2]]), "x": np.concatenate(xs), "v": np.concatenate(vs),
            "types": np.concatenate(ts), "lo": np.array(los), "hi": np.array(his), "masses": [MASS["si"], MASS["ar"]],
            "znum": [Z["si"], Z["ar"]]}


def _heat_setup(case, seed):
    """A film (symbol b) on a substrate (symbol a), hot blocks, and a source
    near the surface."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    film = max(1, n[2] // 4)
    blocks = []
    for _ in range(6):
        lo = [int(rng.integers(0, max(1, q // 2))) for q in n]
        hi = [min(q - 1, p + int(rng.integers(1, max(2, q // 3)))) for p, q in zip(lo, n)]
        blocks.append((lo, hi, float(np.round(rng.uniform(400.0, 3000.0), 3))))
    c = [q // 2 for q in n]
    src = ([max(0, c[0] - 4), max(0, c[1] - 4), n[2] - film], [min(n[0] - 1, c[0] + 4), min(n[1] - 1, c[1] + 4), n[2] - 1],
           float(np.round(rng.uniform(1.0, 20.0), 3)))
    con = [float(np.round(rng.uniform(0.3, 0.6), 3)), float(np.round(rng.uniform(0.8, 2.0), 3))]
    cap = [float(np.round(rng.uniform(1.0, 1.5), 3)), float(np.round(rng.uniform(2.0, 3.0), 3))]
    return dict(n=n, film=film, blocks=blocks, src=src, con=con, cap=cap, dt=0.05, h=1.0)


def _block(b):
    return "@ %d,%d,%d,%d,%d,%d=%r" % (b[0][0], b[0][1], b[0][2], b[1][0], b[1][1], b[1][2], b[2])


FIT_W = dict(wE=1.0, wF=1.0, lr=1e-3, lr_final=1e-5)


def _fit_descriptors():
    """nn_fit's descriptor set: Tersoff's own switch, 16 radial centres, the default angular terms."""
    rs = np.linspace(1.9, 2.85, 16)
    h = rs[1] - rs[0]
    ang = [(z, l, e) for e in (0.0, 0.3) for z in (1, 2, 4, 8) for l in (1.0, -1.0)]
    return (2.85, 2.55), (rs, np.full(16, 1.0 / (2.0 * h * h)), np.array([a[0] for a in ang], dtype=np.int32),
                          np.array([a[1] for a in ang]), np.array([a[2] for a in ang]))


def _fit_data(case, seed):
    """Configurations at spread temperatures' displacements, labelled with Tersoff energies and forces."""
    from objectmd_gb300 import inputs

    xs, es, fs = [], [], []
    rng = np.random.default_rng(seed)
    for k in range(case["nconf"]):
        x, lo, hi = inputs.diamond(case["ncell"], 5.431)
        x = inputs.perturb(x, float(rng.uniform(0.04, 0.16)), 1000 * seed + k, lo, hi)
        e, f = _autograd(lambda d, i, j, n: _tersoff(d, i, j, n), torch.as_tensor(x, device="cuda"), hi, 2.85)
        xs.append(x)
        es.append(e.cpu().numpy())
        fs.append(f.cpu().numpy())
    n = len(xs[0])
    w = np.concatenate([rng.normal(0.0, 1.0 / math.sqrt(32), 64 * 32), np.zeros(64),
                        rng.normal(0.0, 1.0 / 8.0, 64 * 64), np.zeros(64), rng.normal(0.0, 0.0125, 64),
                        [float(np.mean(es))]]).astype(np.float32)
    return n, np.concatenate(xs), np.tile(hi, (case["nconf"], 1)), np.concatenate(es), np.concatenate(fs), w


def prepare(case, seed):
    kind = case["kind"]
    if kind == "md":
        x, v, lo, hi, per = _crystal(case, seed)
        ctx = _context(case, x, v, lo, hi, per)
        return State(kind=kind, own=ctx, steps=case["steps"], frame=_Frame(len(x), np.asarray(hi) - lo),
                     narrow=case["pot"] != "lj")
    if kind == "handover":
        x, v, lo, hi, per = _crystal(case, seed)
        ctx = _context(case, x, v, lo, hi, per)
        n = len(x)
        return State(kind=kind, own=ctx, x=np.array(x), v=np.array(v), f=np.zeros((n, 3)), pot=np.zeros(n),
                     vir=np.zeros(n), L=torch.as_tensor(np.asarray(hi) - lo, device="cuda"))
    if kind == "snapshots":
        x, v, lo, hi, per = _crystal(case, 2 * seed)
        x2 = _crystal(case, 2 * seed + 1)[0]
        ctx = _context(case, x, v, lo, hi, per)
        n = len(x)
        return State(kind=kind, own=ctx, snaps=[(np.array(x), np.array(v)), (np.array(x2), np.array(v))],
                     out=[(np.zeros((n, 3)), np.zeros(n), np.zeros(n)) for _ in range(2)])
    if kind == "impact":
        from objectmd_gb300 import omdg

        e = _impact_inputs(case, seed)
        ctx = omdg.Context(0)
        ctx.set_replicas(e["natoms"], e["lo"], e["hi"], (1, 1, 0))
        ctx.set_atoms(e["x"], e["v"], types=e["types"], masses=e["masses"], znum=e["znum"])
        ctx.add_tersoff(TERSOFF)
        ctx.add_pair_table(AR_SI, 1, 0)
        ctx.set_neighbor(SKIN, 0)
        ctx.set_timestep(0.0005)
        ctx.set_first_step_mode(True)
        L = np.repeat(e["hi"] - e["lo"], e["natoms"], axis=0)
        L[:, 2] = 0.0
        return State(kind=kind, own=ctx, steps=case["steps"], frame=_Frame(len(e["x"]), L), narrow=True)
    if kind == "heat":
        from objectmd_gb300 import omdg

        s = _heat_setup(case, seed)
        nx, ny, nz = s["n"]
        g = omdg.FDTD(nx, ny, nz, "a pppppp b pppppp", "a" * (nx * ny * (nz - s["film"])) + "b" * (nx * ny * s["film"]))
        g.set_spacestep(s["h"])
        g.set_timestep(s["dt"])
        g.set_cell("* 300 " + " ".join(_block(b) for b in s["blocks"]))
        g.set_conductivity("a %r b %r" % tuple(s["con"]))
        g.set_capacity("a %r b %r" % tuple(s["cap"]))
        g.set_source(_block(s["src"]))
        return State(kind=kind, own=g, steps=case["steps"])
    from objectmd_gb300 import omdg

    n, x, box, e, f, w = _fit_data(case, seed)
    net = omdg.Network(0)
    cutoff, desc = _fit_descriptors()
    net.set_cutoff(*cutoff)
    net.set_descriptors(*desc)
    net.set_dataset(np.full(case["nconf"], n), x, box, e.reshape(case["nconf"], n).sum(1), f)
    net.normalize_from_dataset()
    net.set_atom_energies(e)
    net.set_weights(w)
    return State(kind=kind, own=net, nconf=case["nconf"], epochs=case["epochs"])


def run(state):
    s = state
    if s.kind in ("md", "impact"):
        x, v, f = s.frame.np
        s.own.step_io(s.steps, x_out=x, v_out=v, f_out=f)
        out = s.frame.take(s.narrow)
        out["energies"] = _energies(s.own, s.steps, s.narrow)
        return out
    if s.kind == "handover":
        s.own.step_io(1, s.x, s.v, s.x, s.v, s.f)
        s.own.get_state_into(pot=s.pot, vir=s.vir)
        return {"x": _fold(torch.from_numpy(s.x).cuda(), s.L), "v": s.v.astype(np.float32), "f": s.f.astype(np.float32),
                "pot": s.pot.astype(np.float32), "vir": s.vir.astype(np.float32)}
    if s.kind == "snapshots":
        for (x, v), (f, pot, vir) in zip(s.snaps, s.out):
            s.own.set_state(x, v)
            s.own.compute_forces()
            s.own.get_state_into(f=f, pot=pot, vir=vir)
        return [tuple(a.astype(np.float32) for a in o) for o in s.out]
    if s.kind == "heat":
        s.own.step(s.steps)
        return s.own.vector()
    hist = s.own.train(s.epochs, s.nconf, FIT_W["lr"], FIT_W["wE"], FIT_W["wF"], 7, FIT_W["lr_final"])
    return {"loss": hist.astype(np.float32), "weights": s.own.weights()}


# ------------------------------------------------------------------ work

def _atoms(case):
    return case["nx"] * case["ny"] * case["nz"] * SYSTEM[case["pot"]][2]


def work(case):
    kind = case["kind"]
    if kind == "md":
        n, pot, steps = _atoms(case), case["pot"], case["steps"]
        wide = 8 if pot == "lj" else 4  # force word
        # a step: velocity Verlet reads x, v, f and writes x, v (108 B with FP32 forces), the force passes read a
        # position and a neighbour row per atom (EAM twice) and write force and energy
        step = 96 + 3 * wide + (2 if pot == "eam" else 1) * (24 + 4 * ROW[pot]) + 4 * wide
        return {"bytes": n * (steps * step + 48 + 3 * wide), "flops": n * steps * FORCE_FLOPS[pot]}
    if kind == "handover":
        return {"bytes": _atoms(case) * (48 + 48 + 24 + 16 + 2 * (24 + 4 * 54) + 16), "flops": _atoms(case) * FORCE_FLOPS["eam"]}
    if kind == "snapshots":
        return {"bytes": 2 * _atoms(case) * (48 + 24 + 16 + 3 * (24 + 4 * 54) + 16), "flops": 2 * _atoms(case) * FORCE_FLOPS["eam"]}
    if kind == "impact":
        # the mean of the log-uniform slab sizes
        n = case["nrep"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        return {"bytes": n * (case["steps"] * (108 + 24 + 16 + 16) + 72), "flops": n * case["steps"] * 1500}
    if kind == "heat":
        n = case["nx"] * case["ny"] * case["nz"]
        # temperature read and written; conductivity, capacity and source are a few values per symbol or block
        return {"bytes": n * (16 * case["steps"] + 8), "flops": n * case["steps"] * 26}
    n = case["nconf"] * 8 * case["ncell"] ** 3
    # per Adam step and atom: normalised descriptors, 4-5 neighbour Jacobian blocks of 32 x 3 floats, labels
    return {"bytes": case["epochs"] * n * (128 + 4.5 * 384 + 16), "flops": case["epochs"] * n * (6 * 2 * 6272 + 4.5 * 4 * 192)}


# ------------------------------------------------------------------ the same in FP64 torch

class _Table:
    """A table section with the cubic spline of the reference's TableReader
    (second differences S from a tridiagonal system with corner entries 5)."""

    def __init__(self, path, name=""):
        par, tag = [], "#$" + name
        with open(path) as fh:
            for line in fh:
                t = line.split()
                if t and t[0] == tag:
                    if t[1:2] == ["--"]:
                        break
                    par += t[1:]
            n = int(par[par.index("NumberOfData") + 1])
            y = []
            while len(y) < n:
                y += [float(q) for q in next(fh).split()]
        self.dr = float(par[par.index("Spacing") + 1])
        self.off = float(par[par.index("Offset") + 1]) if "Offset" in par else 0.0
        self.rmult = "RMULT" in par
        self.n, y = n, np.array(y[:n])
        d = y[2:] - 2.0 * y[1:-1] + y[:-2]
        b = np.full(n - 2, 4.0)
        b[0] = b[-1] = 5.0
        for k in range(1, n - 2):
            m = 1.0 / b[k - 1]
            b[k] -= m
            d[k] -= m * d[k - 1]
        S = np.zeros(n)
        S[n - 2] = d[-1] / b[-1]
        for k in range(n - 4, -1, -1):
            S[k + 1] = (d[k] - S[k + 2]) / b[k]
        S[n - 1], S[0] = S[n - 2], S[1]
        co = np.zeros((n, 4))
        co[:-1, 3] = (S[1:] - S[:-1]) / self.dr ** 3
        co[:-1, 2] = 3.0 * S[:-1] / self.dr ** 2
        co[:-1, 1] = (y[1:] - y[:-1] - 2.0 * S[:-1] - S[1:]) / self.dr
        co[:, 0] = y
        self.co = torch.as_tensor(co, device="cuda")
        self.top = self.off + (n - 1) * self.dr

    def __call__(self, r):
        u = r - self.off
        k = torch.clamp((u / self.dr).long(), 0, self.n - 2)
        dx = u - k.double() * self.dr
        c = self.co[k]
        val = c[:, 0] + dx * (c[:, 1] + dx * (c[:, 2] + dx * c[:, 3]))
        der = c[:, 1] + dx * (2.0 * c[:, 2] + 3.0 * dx * c[:, 3])
        if self.rmult:
            val = val / r
            der = (der - val) / r
        return val, der


_tables = {}


def _table(path, name=""):
    if (path, name) not in _tables:
        _tables[path, name] = _Table(path, name)
    return _tables[path, name]


def _edges(x, L, rc):
    """Every directed pair within rc: i, j and x_j - x_i of the nearest image (L 0 on free axes)."""
    n = len(x)
    L = torch.as_tensor(L, dtype=torch.float64, device="cuda")
    near = lambda d: d - L * torch.round(torch.nan_to_num(d / L, nan=0.0, posinf=0.0, neginf=0.0))  # noqa: E731
    x = _fold(x, L)
    lo = torch.where(L > 0, torch.zeros_like(L), x.min(0).values)
    ext = torch.where(L > 0, L, x.max(0).values - lo + 1e-9)
    nc = [max(1, int(e / rc)) for e in ext.tolist()]
    if n <= 6000 or any(c < 3 and q > 0 for c, q in zip(nc, L.tolist())):
        out = []
        step = max(1, 40_000_000 // n)
        for a in range(0, n, step):
            d = near(x[None] - x[a:a + step, None])
            i, j = torch.nonzero((d * d).sum(2) < rc * rc, as_tuple=True)
            keep = i + a != j
            i, j = i[keep], j[keep]
            out.append((i + a, j, d[i, j]))
        return tuple(torch.cat(q) for q in zip(*out))
    ncell = torch.tensor(nc, device="cuda")
    c = torch.minimum(((x - lo) / ext * ncell).long().clamp(min=0), ncell - 1)
    cid = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    order = torch.argsort(cid)
    cnt = torch.bincount(cid, minlength=nc[0] * nc[1] * nc[2])
    start = torch.cumsum(cnt, 0) - cnt
    rank = torch.arange(n, device="cuda") - start[cid[order]]
    tab = torch.full((len(cnt) + 1, int(cnt.max())), -1, dtype=torch.long, device="cuda")
    tab[cid[order], rank] = order
    ii = torch.arange(n, device="cuda")
    out = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                q = c + torch.tensor([dx, dy, dz], device="cuda")
                bad = torch.zeros(n, dtype=torch.bool, device="cuda")
                for k in range(3):
                    if L[k] > 0:
                        q[:, k] %= nc[k]
                    else:
                        bad |= (q[:, k] < 0) | (q[:, k] >= nc[k])
                k = torch.where(bad, len(cnt), (q[:, 2] * nc[1] + q[:, 1]) * nc[0] + q[:, 0])
                cand = tab[k]
                a, b = torch.nonzero(cand >= 0, as_tuple=True)
                j = cand[a, b]
                i = ii[a]
                d = near(x[j] - x[i])
                keep = ((d * d).sum(1) < rc * rc) & (i != j)
                out.append((i[keep], j[keep], d[keep]))
    return tuple(torch.cat(q) for q in zip(*out))


def _sum_at(i, v, n):
    return torch.zeros((n,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, i, v)


def _eam(x, L):
    phi, den, emb = (_table(EAM_AL, q) for q in ("PAIR", "EDENS", "EMBED"))
    n = len(x)
    i, j, d = _edges(x, L, max(phi.top, den.top))
    r = d.norm(dim=1)
    p, dp = phi(r)
    ok = r <= phi.top
    p, dp = p * ok, dp * ok
    g, dg = den(r)
    ok = r <= den.top
    F, dF = emb(_sum_at(i, g * ok, n))
    fr = -((dF[i] + dF[j]) * (dg * ok) + dp) / r
    return F + 0.5 * _sum_at(i, p, n), -_sum_at(i, d * fr[:, None], n), _sum_at(i, fr * r * r, n)


def _pair(x, L, path):
    phi = _table(path)
    n = len(x)
    i, j, d = _edges(x, L, phi.top)
    r = d.norm(dim=1)
    p, dp = phi(r)
    return 0.5 * _sum_at(i, p, n), _sum_at(i, d * (dp / r)[:, None], n)


def _autograd(energy, x, L, rc):
    """Per-atom energies and forces of energy(d, i, j, n) -> per-atom energies."""
    i, j, d = _edges(x, L, rc)
    d.requires_grad_(True)
    e = energy(d, i, j, len(x))
    g, = torch.autograd.grad(e.sum(), d)
    return e.detach(), _sum_at(i, g, len(x)) - _sum_at(j, g, len(x))


def _rows(d, i, n, far):
    """The edges as one row of vectors per centre, padded with a vector of length `far`; the padding's mask."""
    order = torch.argsort(i, stable=True)
    cnt = torch.bincount(i, minlength=n)
    start = torch.cumsum(cnt, 0) - cnt
    rank = torch.arange(len(i), device="cuda") - start[i[order]]
    k = max(2, int(cnt.max()))
    rows = torch.zeros((n, k, 3), dtype=torch.float64, device="cuda")
    rows[..., 0] = far
    real = torch.zeros((n, k), dtype=torch.bool, device="cuda")
    real[i[order], rank] = True
    return rows.index_put((i[order], rank), d[order]), real


def _params(path):
    out = {}
    with open(path) as fh:
        for line in fh:
            t = line.split("#")[0].split()
            if len(t) > 1:
                out[t[0].split(".")[-1]] = t[1]
    return {k: float(v) for k, v in out.items() if v not in ("yes", "no", "true", "false")}


def _switch(r, lo, hi):
    """1 below lo, a cosine down to 0 at hi."""
    return 0.5 * (1.0 + torch.cos(math.pi * (r.clamp(lo, hi) - lo) / (hi - lo)))


def _tersoff(d, i, j, n):
    """Tersoff, PRB 37, 6991 (1988): 1/2 sum_j fc (fR - b fA) per centre."""
    q = _params(TERSOFF)
    lo, hi = q["R"] - q["D"], q["R"] + q["D"]
    rows, real = _rows(d, i, n, 2.0 * hi)
    r = rows.norm(dim=2)
    fc = _switch(r, lo, hi) * real
    u = rows / r[..., None]
    cs = torch.einsum("nac,nbc->nab", u, u)
    g = 1.0 + (q["c"] / q["d"]) ** 2 - q["c"] ** 2 / (q["d"] ** 2 + (q["h"] - cs) ** 2)
    both = real[:, :, None] & real[:, None, :] & ~torch.eye(r.shape[1], dtype=torch.bool, device="cuda")
    dr = torch.where(both, r[:, :, None] - r[:, None, :], 0.0)
    zeta = torch.where(both, fc[:, None, :] * g * torch.exp(q["lambda_3"] ** 3 * dr ** 3), 0.0).sum(2)
    b = (1.0 + (q["beta"] * zeta) ** q["n"]) ** (-0.5 / q["n"])
    v = fc * (q["A"] * torch.exp(-q["lambda_1"] * r) - b * q["B"] * torch.exp(-q["lambda_2"] * r))
    return 0.5 * torch.where(real, v, 0.0).sum(1)


def _sw(d, i, j, n):
    """Stillinger-Weber, PRB 31, 5262 (1985), beyond the spline core (1.8456 A)."""
    q = _params(SW)
    s, rc = q["sigma"], q["sigma"] * q["a"]
    rows, real = _rows(d, i, n, 2.0 * rc)
    r = rows.norm(dim=2)
    gap = torch.where(real, r - rc, -1.0)
    two = q["A"] * q["epsilon"] * (q["B"] * (s / r) ** q["p"] - (s / r) ** q["q"]) * torch.exp(s / gap)
    w = torch.where(real, torch.exp(s * q["gamma"] / gap), 0.0)
    u = rows / r[..., None]
    a, b = torch.triu_indices(r.shape[1], r.shape[1], 1, device="cuda")
    cs = (u[:, a] * u[:, b]).sum(2)
    three = q["lambda"] * q["epsilon"] * w[:, a] * w[:, b] * (cs - 1.0 / q["invers_cos0"]) ** 2
    return 0.5 * torch.where(real, two, 0.0).sum(1) + three.sum(1)


def _descriptors(rows, real, rc, rin, rs, eta_r, zeta, lam, eta_a):
    r = rows.norm(dim=2)
    fc = _switch(r, rin, rc) * real
    t = lambda v: torch.as_tensor(np.asarray(v, dtype=np.float64), device="cuda")  # noqa: E731
    rad = (torch.exp(-t(eta_r) * (r[..., None] - t(rs)) ** 2) * fc[..., None]).sum(1)
    a, b = torch.triu_indices(r.shape[1], r.shape[1], 1, device="cuda")
    cs = ((rows[:, a] * rows[:, b]).sum(2) / (r[:, a] * r[:, b])) * (real[:, a] & real[:, b])
    ff, s2 = fc[:, a] * fc[:, b], r[:, a] ** 2 + r[:, b] ** 2
    ang = []
    for z, l, e in zip(zeta, lam, eta_a):
        ang.append((2.0 ** (1.0 - z) * (1.0 + l * cs) ** int(z) * torch.exp(-e * s2) * ff).sum(1))
    return torch.cat([rad, torch.stack(ang, 1)], 1)


def _network(g, w):
    """w: 64x32, 64, 64x64, 64, 64, 1 back to back."""
    w1, b1, w2, b2, w3, b3 = torch.split(w, [2048, 64, 4096, 64, 64, 1])
    a = torch.tanh(g @ w1.view(64, 32).T + b1)
    return torch.tanh(a @ w2.view(64, 64).T + b2) @ w3 + b3


def _surrogate(d, i, j, n):
    """The model file's network; centres whose descriptors leave the training range take Tersoff's energy."""
    m = {}
    with open(NN_MODEL) as fh:
        for line in fh:
            t = line.split()
            if t and t[0] != "params":
                m[t[0]] = np.array([float(q) for q in t[1:]])
            if t and t[0] == "w":
                m["w"] = np.array([float(q) for q in t[1:]] + [float(q) for q in fh.read().split()])[:6337]
    rows, real = _rows(d, i, n, 2.0 * m["rc"][0])
    G = _descriptors(rows, real, m["rc"][0], m["rin"][0], m["rs"], m["eta_r"], m["zeta"], m["lambda"], m["eta_a"])
    t = lambda k: torch.as_tensor(m[k], device="cuda")  # noqa: E731
    inside = ((G >= t("gmin")) & (G <= t("gmax"))).all(1)
    e = _network((G - t("mu")) / t("sigma"), t("w"))
    return torch.where(inside, e, _tersoff(d, i, j, n))


def _forces(pot, x, L):
    if pot == "eam":
        e, f, _ = _eam(x, L)
        return e, f
    if pot == "lj":
        return _pair(x, L, LJ_AR)
    if pot == "tersoff":
        return _autograd(_tersoff, x, L, 2.85)
    if pot == "sw":
        return _autograd(_sw, x, L, 1.8 * 2.0951)
    return _autograd(_surrogate, x, L, 2.8499999)


def _verlet(force, x, v, m, dt, steps, temp=0.0, tau=0.0):
    """Velocity Verlet as the reference starts it: the first half-kick has no
    force (its first step follows a force evaluation that it discards).  With
    tau, Berendsen's factor from each step's kinetic energy but the first's."""
    f, lam, rows = torch.zeros_like(x), 1.0, []
    for k in range(steps):
        v = v * lam + 0.5 * dt * f / m
        x = x + dt * v
        e, f = force(x)
        v = v + 0.5 * dt * f / m
        kin, lam = 0.5 * float((m * v * v).sum()), 1.0
        if tau > 0.0 and k > 0:
            lam = math.sqrt(1.0 + dt / tau * (temp / ((2.0 / 3.0) / KB * kin / len(x)) - 1.0))
        rows.append((kin, float(e.sum())))
    return x, v * lam, f, torch.tensor(rows, dtype=torch.float64)


def _impact_force(e):
    """Tersoff between the Si atoms and the Ar-Si table, slab by slab."""
    ends = np.concatenate([[0], np.cumsum(e["natoms"])])
    L = e["hi"] - e["lo"]
    zbl = _table(AR_SI)

    def force(x):
        en, fo = [], []
        for r in range(len(e["natoms"])):
            y = x[ends[r]:ends[r + 1]]
            box = torch.as_tensor([L[r, 0], L[r, 1], 0.0], dtype=torch.float64, device="cuda")
            si = len(y) - 1  # the Ar atom comes last
            es, fs = _autograd(_tersoff, y[:si], box, 2.85)
            d = y[:si] - y[si]
            d = d - box * torch.round(torch.nan_to_num(d / box, nan=0.0, posinf=0.0, neginf=0.0))
            rr = d.norm(dim=1)
            p, dp = zbl(rr.clamp(max=zbl.top - 1e-9))
            p, dp = p * (rr < zbl.top), dp * (rr < zbl.top)
            pull = -d * (dp / rr)[:, None]
            en.append(torch.cat([es + 0.5 * p, 0.5 * p.sum()[None]]))
            fo.append(torch.cat([fs + pull, -pull.sum(0)[None]]))
        return torch.cat(en), torch.cat(fo)

    return force


def _exact_heat(case, seed):
    s = _heat_setup(case, seed)
    nx, ny, nz = s["n"]
    T = torch.full((nz, ny, nx), 300.0, dtype=torch.float64, device="cuda")
    S = torch.zeros_like(T)
    box = lambda a, lo, hi, v: a[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].fill_(v)  # noqa: E731
    for b in s["blocks"]:
        box(T, *b)
    box(S, *s["src"])
    con, cap = torch.full_like(T, s["con"][0]), torch.full_like(T, s["cap"][0])
    con[nz - s["film"]:], cap[nz - s["film"]:] = s["con"][1], s["cap"][1]
    for _ in range(case["steps"]):
        acc = torch.zeros_like(T)
        for axis in range(3):
            for way in (-1, 1):
                cn = torch.roll(con, way, axis)
                acc += con * cn / (con + cn) * (torch.roll(T, way, axis) - T)
        T = T + (2.0 * acc / s["h"] ** 2 + S) * s["dt"] / cap
    return T.reshape(-1).cpu()


def _exact_fit(case, seed):
    n, x, box, e_ref, f_ref, w = _fit_data(case, seed)
    (rc, rin), desc = _fit_descriptors()
    ii, jj, dd = [], [], []
    for c in range(case["nconf"]):
        i, j, d = _edges(torch.as_tensor(x[c * n:(c + 1) * n], device="cuda"), box[c], rc)
        ii.append(i + c * n)
        jj.append(j + c * n)
        dd.append(d)
    i, j, d = torch.cat(ii), torch.cat(jj), torch.cat(dd).requires_grad_(True)
    G = _descriptors(*_rows(d, i, len(x), 2.0 * rc), rc, rin, *desc)
    mu = G.detach().mean(0)
    sg = (G.detach() ** 2).mean(0).sub(mu * mu).clamp(min=0).sqrt()
    sg = torch.where(sg > 1e-6 * mu.abs(), sg, 1.0)
    g = (G - mu) / sg
    w = torch.as_tensor(w.astype(np.float64), device="cuda").requires_grad_(True)
    e_ref, f_ref = (torch.as_tensor(q, device="cuda") for q in (e_ref, f_ref))
    m1 = m2 = 0.0
    losses = []
    for k in range(case["epochs"]):
        e = _network(g, w)
        q, = torch.autograd.grad(e.sum(), d, create_graph=True)
        f = torch.zeros_like(f_ref).index_add(0, i, q).index_add(0, j, -q)
        loss = FIT_W["wE"] * ((e - e_ref) ** 2).mean() + FIT_W["wF"] * ((f - f_ref) ** 2).mean()
        gw, = torch.autograd.grad(loss, w, retain_graph=True)
        lr = FIT_W["lr_final"] + 0.5 * (FIT_W["lr"] - FIT_W["lr_final"]) * (1.0 + math.cos(math.pi * k / max(1, case["epochs"] - 1)))
        if case["epochs"] == 1:
            lr = FIT_W["lr"]
        m1, m2 = 0.9 * m1 + 0.1 * gw, 0.999 * m2 + 0.001 * gw * gw
        step = lr * math.sqrt(1.0 - 0.999 ** (k + 1)) / (1.0 - 0.9 ** (k + 1))
        with torch.no_grad():
            w -= step * m1 / (m2.sqrt() + 1e-8)
        losses.append(float(loss.detach()))
    return {"loss": np.array(losses), "weights": w.detach().cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "heat":
        return _exact_heat(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    gpu = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")  # noqa: E731
    if kind == "impact":
        if case["nrep"] * case["steps"] > 2000:
            return None  # slab by slab it takes a minute
        e = _impact_inputs(case, seed)
        m = gpu(np.where(e["types"] == 0, e["masses"][0], e["masses"][1])[:, None])
        x, v, f, rows = _verlet(_impact_force(e), gpu(e["x"]), gpu(e["v"]), m, 0.0005, case["steps"])
        L = np.repeat(e["hi"] - e["lo"], e["natoms"], axis=0)
        L[:, 2] = 0.0
        return {"x": _fold(x, gpu(L)), "v": v, "f": f, "energies": rows}
    if kind == "snapshots":
        out = []
        for k in range(2):
            x, _, lo, hi, per = _crystal(case, 2 * seed + k)
            e, f, w = _eam(gpu(x), (np.asarray(hi) - lo) * np.asarray(per))
            out.append((f, e, w))
        return out
    x, v, lo, hi, per = _crystal(case, seed)
    L = np.asarray(hi) - lo
    elem, _, _, _, dt = SYSTEM[case["pot"]]
    steps = case.get("steps", 1)
    x, v, f, rows = _verlet(lambda y: _forces(case["pot"], y, L), gpu(x), gpu(v), MASS[elem], dt, steps,
                            case["temp"], case.get("tau", 0.0))
    out = {"x": _fold(x, gpu(L)), "v": v, "f": f}
    if kind == "md":
        out["energies"] = rows
    else:
        out["pot"], _, out["vir"] = _eam(x, L)
    return out
