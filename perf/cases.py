"""Performance cases of the Monte Carlo path, from one short call to 3.2 million beads.

Every case goes through an entry point that a program of this package calls:

* ``call``     ``mc_sim`` on one ``Chromatin`` chain in one ``UniformDensityField``, the
               reference's own call: everything is built, run and read back each time.
* ``mc``       chains resident on the device (one or many, FP32 or FP64 positions, with or
               without spherical confinement or SSTWLC twist): MC steps, or rounds of MC
               steps and replica exchange, and the chains read back.
* ``sample``   MC steps with the energy terms of every replica added to the running sums
               after each (the reweighting estimates).
* ``energies`` chains uploaded from host arrays, densities rebuilt, FP64 energies read.
* ``gradient`` dE/dr of every bead and the energy terms, read back.
* ``autograd`` ``replica_energy`` on CUDA tensors, forward and backward.
* ``steric``   the clash energy of one chain and its change for one moved segment.

Chains are worm-like walks of 16.5 nm bonds (lp = 53 nm) rounded to binary32, with Markov mark
tracks and partly filled binding sites.  Controllers start at the amplitudes they settle at
(segments of up to 150 beads, ~13 rotated tangents), so that passes cost what the moves of a
long run cost.
"""
import math
from pathlib import Path

import numpy as np
import torch

import chromo_gb300
from chromo_gb300 import _native as nat
from chromo_gb300.autograd import replica_energy
from chromo_gb300.device import binding_params, field_params, move_ctl
from chromo_gb300.synthetic import confined_walks

SPACING, LP, VOXEL, BEAD_RAD = 16.5, 53.0, 40.0, 5.0
R_INT, SITES, E_MOD, E_NOMOD = 3.0, 2, -0.01, 1.52
EPS = (-4.0, -3.0, -2.0)            # self-interaction of binder b (kT)
CROSS_01 = 1.0                      # cross talk of binders 0 and 1, stored on binder 0
VF_LIMIT = 0.5
BEAD_VOL = 4.0 / 3.0 * math.pi * BEAD_RAD ** 3
V_INT = 4.0 / 3.0 * math.pi * R_INT ** 3
LT = 100.0                          # twist persistence length (nm)
EXCLUDED = 2 * BEAD_RAD             # steric excluded distance
CYCLE = {"crank_shaft": 30, "end_pivot": 1, "slide": 60, "tangent_rotation": 60,
         "change_binding_state": 10}


def listed():
    return [
        # the smallest call: one MC step of the reference's mc_sim on a short chain
        dict(name="call_1k", kind="call", beads=1000, steps=1) | _dims(30, 30, 30),
        # one plain chain, FP32 positions, one binder (60^3 grid)
        _mc("chain_10k", 1, 10000, 10000, (60, 60, 60), 1, 10),
        # one short chain in the reference's arithmetic, one attempt of each move per step
        _mc("chain_1k_fp64", 1, 1000, 1000, (30, 30, 30), 1, 60, fp64=True, one_each=True),
        # many uneven chains on a chi ladder, two rounds of MC steps and exchange
        _mc("batch_256", 256, 2000, 20000, (40, 40, 40), 2, 10, rounds=2, rungs=16),
        # a few very long chains
        _mc("large_32", 32, 100000, 100000, (100, 100, 100), 2, 5),
        # confined chains with accessible volumes at the surface
        _mc("sphere_128", 128, 3000, 3000, (40, 40, 40), 2, 10, radius=700.0),
        # SSTWLC chains (twist energy in every move)
        _mc("twist_64", 64, 2000, 2000, (24, 24, 24), 1, 10, twist=True),
        # reweighting samples: one MC step and one sample of the terms, four times
        dict(name="sample_64", kind="sample", replicas=64, lo=5000, hi=5000, nb=2, steps=1,
             samples=4) | _dims(40, 40, 40),
        # a batch of host chains: upload, density, energies (what a push and a check cost)
        dict(name="energies_256", kind="energies", replicas=256, lo=2000, hi=20000, nb=2,
             fp64=False, radius=0.0) | _dims(40, 40, 40),
        # derivatives of the energy on host arrays
        dict(name="gradient_64", kind="gradient", replicas=64, lo=5000, hi=5000, nb=2,
             fp64=False) | _dims(40, 40, 40),
        # the same on CUDA tensors through autograd, forward and backward
        dict(name="autograd_64", kind="autograd", replicas=64, lo=5000, hi=5000, nb=2,
             tangents=True) | _dims(40, 40, 40),
        # clash energy of a dense chain, and of a moved segment
        dict(name="steric_10k", kind="steric", beads=10000, radius=250.0, segment=100),
    ]


def _dims(nx, ny, nz):
    return dict(nx=nx, ny=ny, nz=nz)


def _mc(name, replicas, lo, hi, dims, nb, steps, *, rounds=0, rungs=0, fp64=False, one_each=False,
        radius=0.0, twist=False):
    return dict(name=name, kind="mc", replicas=replicas, lo=lo, hi=hi, nb=nb, steps=steps, rounds=rounds,
                rungs=rungs, fp64=fp64, one_each=one_each, radius=radius, twist=twist) | _dims(*dims)


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "mc", "mc", "mc", "mc", "sample", "energies", "gradient", "autograd", "steric"])
    dims = _dims(*(rng.randint(20, 44) for _ in range(3)))
    nb = rng.randint(1, 3)
    if kind == "call":
        return dict(kind="call", beads=log(200, 3000), steps=rng.randint(1, 8)) | dims
    if kind == "steric":
        beads = log(500, 12000)
        return dict(kind="steric", beads=beads, radius=12.0 * beads ** (1 / 3), segment=rng.randint(1, 150))
    lo = log(700, 8000)
    hi = min(20000, int(lo * rng.uniform(1.0, 4.0)))
    replicas = max(1, min(log(1, 256), 1_200_000 // hi))
    if kind == "mc":
        mode = rng.choice(["plain", "plain", "exchange", "fp64", "sphere", "twist"])
        rungs = rng.choice([2, 4, 8]) if mode == "exchange" else 0
        if rungs:
            replicas = max(rungs, replicas // rungs * rungs)
        if mode == "fp64":
            replicas = min(replicas, 64)
        if mode == "sphere":
            lo, hi = min(lo, 3000), min(hi, 4000)
            hi = max(lo, hi)
        radius = 0.45 * VOXEL * min(dims["nx"], dims["ny"], dims["nz"]) if mode == "sphere" else 0.0
        c = _mc("", replicas, lo, hi, tuple(dims.values()), nb, rng.randint(2, 12),
                rounds=rng.randint(1, 3) if rungs else 0, rungs=rungs, fp64=mode == "fp64",
                one_each=rng.random() < 0.2, radius=radius, twist=mode == "twist")
        del c["name"]
        return c
    c = dict(kind=kind, replicas=replicas, lo=lo, hi=hi, nb=nb) | dims
    if kind == "sample":
        c |= dict(replicas=min(replicas, 96), steps=rng.randint(1, 3), samples=rng.randint(1, 4))
    if kind == "energies":
        c |= dict(fp64=rng.random() < 0.3, radius=0.0)
    if kind == "gradient":
        c |= dict(fp64=rng.random() < 0.3)
    if kind == "autograd":
        c |= dict(tangents=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------- inputs

def _f32(a):
    return a.astype(np.float32).astype(np.float64)


def _frames(rng, t):
    """A unit t2 perpendicular to each unit t3."""
    t2 = np.cross(t, rng.standard_normal(t.shape))
    return t2 / np.linalg.norm(t2, axis=1)[:, None]


def _walk(rng, n):
    """A worm-like walk: tangents of an AR(1) Gaussian process (correlation exp(-spacing / lp)
    per bond), bonds along them with a little noise."""
    y = rng.standard_normal((n + 64, 3))
    a = math.exp(-SPACING / LP)
    for k in (1, 2, 4, 8, 16, 32):
        y[k:] = y[k:] + a ** k * y[:-k]
    t = y[64:] / np.linalg.norm(y[64:], axis=1)[:, None]
    step = 0.95 * SPACING * t[:-1] + 1.5 * rng.standard_normal((n - 1, 3))
    r = np.zeros((n, 3))
    r[1:] = np.cumsum(step, axis=0)
    return r, t


def _marks(rng, n, run=50):
    jump = (rng.random(n) < 1.0 / run) * rng.integers(1, 3, size=n)
    return (int(rng.integers(0, 3)) + np.cumsum(jump)) % 3


def _chains(case, seed):
    """Per replica: r, t3, t2, states, marks."""
    rng = np.random.default_rng([seed, 7])
    lo, hi, nb = case["lo"], case["hi"], case["nb"]
    R = case["replicas"]
    # the lengths belong to the case: log-uniform, the same for every seed
    u = np.random.default_rng([R, lo, hi]).random(R)
    lengths = np.clip(np.round(lo * (hi / lo) ** u).astype(np.int64), lo, hi)
    inside = None
    if case.get("radius", 0.0) > 0:
        inside = confined_walks(rng, R, int(lengths.max()), SPACING, 0.97 * case["radius"])
    out = []
    for k in range(R):
        n = int(lengths[k])
        if inside is None:
            r, t3 = _walk(rng, n)
        else:
            r = inside[k, :n]
            t3 = np.gradient(r, axis=0)
            t3 = t3 / np.linalg.norm(t3, axis=1)[:, None]
        marks = np.stack([_marks(rng, n) for _ in range(nb)], axis=1)
        bound = np.where(marks > 0, 0.45, 0.15)
        states = (rng.random((n, nb)) < bound).astype(np.int64) + (rng.random((n, nb)) < bound)
        out.append(dict(r=_f32(r), t3=_f32(t3), t2=_f32(_frames(rng, t3)), states=states, marks=marks))
    mu = rng.uniform(-1.0, 0.0, size=(R, nb))
    rungs = case.get("rungs") or 1
    chi = np.tile(np.linspace(0.5, 2.0, rungs), R // rungs) if rungs > 1 else np.full(R, 1.0)
    return out, mu, chi


_TABLE = []


def _bonds(n):
    """eps_bend, gamma, eps_par, eps_perp, eta of n bonds of the chain, from the dssWLC table."""
    if not _TABLE:
        _TABLE.append(np.loadtxt(Path(chromo_gb300.__file__).parent / "data" / "dssWLCparams"))
    t, d = _TABLE[0], SPACING / LP
    c = [np.interp(d, t[:, 0], t[:, k]) for k in range(1, 6)]
    one = [c[0] / d, c[1] * d * LP, c[2] / (d * LP ** 2), c[3] / (d * LP ** 2), c[4] / LP]
    return np.tile(np.array(one), (n, 1))


def _prefactors(nb, vol):
    pref = [0.5 * EPS[b] * V_INT * vol for b in range(nb)]
    intra = [EPS[b] * (1 - V_INT / vol) for b in range(nb)]
    x = np.zeros((nb, nb))
    if nb > 1:
        x[0, 1] = CROSS_01 * V_INT * vol
    return pref, intra, x


def _controls(n, one_each):
    """The five moves under SimpleControl, at the amplitudes they settle at."""
    seg = {"crank_shaft": (min(30, n), min(150, n)), "end_pivot": (min(50, n / 4), min(150, n // 2)),
           "slide": (min(10, n), min(150, n)), "tangent_rotation": (1, n), "change_binding_state": (1, 1)}
    amp = {"crank_shaft": (0.1 * np.pi, 0.25 * np.pi), "end_pivot": (0.2 * np.pi, 0.25 * np.pi),
           "slide": (0.2 * SPACING, 0.3 * SPACING), "tangent_rotation": (0.05 * np.pi, 0.2 * np.pi),
           "change_binding_state": (0.0, 0.0)}
    return [move_ctl(m, amp_move=0.5 * (amp[m][0] + amp[m][1]),
                     amp_bead=min(13, n) if m == "tangent_rotation" else int(seg[m][1]),
                     num_per_cycle=1 if one_each else CYCLE[m], simple=True, bead_bounds=seg[m],
                     move_bounds=amp[m], acc_rate=0.5) for m in nat.MOVE_NAMES]


_VOLUMES = {}


def _volumes(case):
    """Accessible volumes of the confining sphere (one table per grid, as a program keeps)."""
    from chromo_gb300.fields import spherical_accessible_volumes
    key = (case["nx"], case["ny"], case["nz"], case["radius"])
    if key not in _VOLUMES:
        _VOLUMES[key] = spherical_accessible_volumes(*key[:3], VOXEL, VOXEL, VOXEL, key[3], VOXEL ** 3)
    return _VOLUMES[key]


def _resident(case, seed):
    """The chains resident on the device, and the same chains on the host."""
    chains, mu, chi = _chains(case, seed)
    nb, dims = case["nb"], (case["nx"], case["ny"], case["nz"])
    radius = case.get("radius", 0.0)
    n_beads = [len(c["r"]) for c in chains]
    sim = nat.Sim(n_beads, [dims] * len(chains), nb, pos_fp64=case.get("fp64", False), max_segment=152,
                  max_tangent=max(n_beads), nonuniform_access=radius > 0)
    pref, intra, x = _prefactors(nb, VOXEL ** 3)
    for k, c in enumerate(chains):
        n = n_beads[k]
        sim.set_chain(k, bonds=_bonds(n - 1), **c)
        if case.get("twist"):
            sim.set_twist(k, np.full(n - 1, LT / SPACING), np.full(n - 1, SPACING * (2 * np.pi / 10.5) / 0.332))
        sim.set_field(k, field_params(field_kind=2, nxyz=dims, widths=tuple(VOXEL * d for d in dims),
                                      n_binders=nb, chi=float(chi[k]), vf_limit=VF_LIMIT, bead_vol=BEAD_VOL,
                                      pref=pref, intra=intra, xpref=x, confine_kind=1 if radius > 0 else 0,
                                      confine_length=radius),
                      access_vol=_volumes(case) if radius > 0 else None)
        sim.set_binding(k, binding_params(sites=[SITES] * nb, e_mod=[E_MOD] * nb, e_nomod=[E_NOMOD] * nb,
                                          mu=list(mu[k])))
        sim.set_controllers(k, _controls(n, case.get("one_each", False)))
    sim.deposit(-1)
    return sim, chains


class _Buffers:
    """One host array for r, t3, t2 and states of all chains, and each chain's part of it."""

    def __init__(self, n_beads, nb):
        total = int(sum(n_beads))
        self.whole = [np.zeros((total, 3)) for _ in range(3)] + [np.zeros((total, nb), dtype=np.int64)]
        at = np.concatenate([[0], np.cumsum(n_beads)])
        self.parts = [tuple(a[at[k]:at[k + 1]] for a in self.whole) for k in range(len(n_beads))]


def _call_objects(case, seed):
    from chromo_gb300 import binders, mc
    from chromo_gb300.fields import UniformDensityField
    from chromo_gb300.mc.mc_controller import SimpleControl, all_moves
    from chromo_gb300.polymers import Chromatin
    c = _chains(dict(lo=case["beads"], hi=case["beads"], replicas=1, nb=1), seed)[0][0]
    poly = Chromatin("Chr", c["r"], bead_length=np.full(case["beads"] - 1, SPACING), t3=c["t3"], t2=c["t2"],
                     states=c["states"], binder_names=np.array(["HP1"]), chemical_mods=c["marks"],
                     chemical_mod_names=np.array(["H3K9me3"]))
    readers = binders.make_binder_collection(["HP1"])
    dims = (case["nx"], case["ny"], case["nz"])
    field = UniformDensityField([poly], readers, *(v for d in dims for v in (VOXEL * d, d)))
    bead, move = mc.get_amplitude_bounds([poly])
    return dict(poly=poly, readers=readers, field=field,
                controls=all_moves("", bead.bounds, move.bounds, SimpleControl))


class _Batch:
    """Resident chains as ``replica_energy`` takes them."""

    def __init__(self, sim):
        self.sim = sim


def prepare(case, seed):
    kind = case["kind"]
    if kind == "call":
        return dict(case=case, seed=seed) | _call_objects(case, seed)
    if kind == "steric":
        n, m = case["beads"], case["segment"]
        r, trial, ind0 = _steric_inputs(case, seed)
        sim = nat.Sim([n], [(1, 1, 1)], 1)
        sim.set_chain(0, r=r, t3=np.tile([0.0, 0.0, 1.0], (n, 1)), t2=np.tile([1.0, 0.0, 0.0], (n, 1)),
                      states=np.zeros((n, 1), np.int64), marks=np.zeros((n, 1), np.int64), bonds=_bonds(n - 1))
        return dict(case=case, sim=sim, trial=trial, ind0=ind0, indf=ind0 + m)
    sim, chains = _resident(case, seed)
    state = dict(case=case, seed=seed, sim=sim)
    if kind in ("mc", "sample"):
        state["buffers"] = _Buffers(sim.n_beads, case["nb"])
    if kind == "energies":
        state["chains"] = [{k: c[k] for k in ("r", "t3", "t2", "states")} for c in chains]
    if kind == "autograd":
        dev = torch.device("cuda")
        state["batch"] = _Batch(sim)
        state["r"] = torch.from_numpy(np.concatenate([c["r"] for c in chains])).to(dev).requires_grad_()
        state["t3"] = torch.from_numpy(np.concatenate([c["t3"] for c in chains])).to(dev)
        state["t3"].requires_grad_(case["tangents"])
        state["weight"] = torch.linspace(0.5, 1.5, sim.R, dtype=torch.float64, device=dev)
    return state


def _steric_inputs(case, seed):
    rng = np.random.default_rng([seed, 13])
    n, m = case["beads"], case["segment"]
    r = _f32(confined_walks(rng, 1, n, SPACING, case["radius"])[0])
    ind0 = int(rng.integers(0, n - m + 1))
    return r, r[ind0:ind0 + m] + rng.normal(0.0, 3.0, (m, 3)), ind0


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        from chromo_gb300.mc import mc_sim
        poly, field = state["poly"], state["field"]
        mc_sim([poly], state["readers"], case["steps"], state["controls"], field, 1.0, state["seed"])
        return dict(r=poly.r, t3=poly.t3, t2=poly.t2, states=poly.states, density=field.density_fixed_point,
                    amplitudes=[c.move.amp_move for c in state["controls"]],
                    accepted=[c.move.num_success for c in state["controls"]])
    sim = state["sim"]
    if kind == "mc":
        if case["rounds"]:
            sim.run_batched(case["rounds"], case["steps"], case["rungs"], state["seed"])
        else:
            sim.run(case["steps"], state["seed"])
        sim.sync()
        sim.get_chains(state["buffers"].parts)
        r, t3, t2, states = state["buffers"].whole
        out = dict(r=r, t3=t3, t2=t2, states=states)
        if case["rounds"]:
            out["chi"] = sim.chi()
        return out
    if kind == "sample":
        for k in range(case["samples"]):
            sim.run(case["steps"], state["seed"] + k)
            sim.sample_terms()
        sim.sync()
        sum_t, sum_tt, count = sim.samples()
        sim.get_chains(state["buffers"].parts)
        r, t3, t2, states = state["buffers"].whole
        return dict(sum_t=sum_t, sum_tt=sum_tt, count=count, r=r, t3=t3, t2=t2, states=states)
    if kind == "energies":
        sim.set_chains(state["chains"])
        sim.deposit(-1)
        return sim.energies()
    if kind == "gradient":
        g, terms = sim.gradient()
        return dict(dEdr=g, terms=terms)
    if kind == "autograd":
        r, t3 = state["r"], state["t3"]
        r.grad = t3.grad = None
        E = replica_energy(r, state["batch"], t3)
        (E * state["weight"]).sum().backward()
        out = dict(E=E.detach(), r=r.grad)
        if case["tangents"]:
            out["t3"] = t3.grad
        return out
    return dict(energy=sim.steric_energy(0, EXCLUDED),
                change=sim.steric_delta(0, state["ind0"], state["indf"], state["trial"], EXCLUDED))


# ---------------------------------------------------------------- work

def _moves_work(case, moves_per_step, one_each):
    """Bytes and operations of the attempted moves: the moved beads' vectors and states, two
    neighbours and bonds, the touched voxels' columns, and the write-back of the accepted ones
    (mean segment and voxel counts of settled amplitudes)."""
    nb, k = case.get("nb", 1), 8 if case.get("fp64") else 4
    v = 3 * k
    per = {}
    for m, (beads, voxels, acc, vecs) in {"crank_shaft": (28.5, 49.0, 0.73, 3), "end_pivot": (29.5, 62.0, 0.77, 3),
                                          "slide": (28.5, 47.5, 0.53, 1), "tangent_rotation": (7.0, 0.0, 0.5, 2),
                                          "change_binding_state": (1.0, 5.3, 0.67, 0)}.items():
        read = beads * (vecs * v + nb) + voxels * (1 + nb) * 8 + 4 * v + 10 * k
        if m == "tangent_rotation":
            read = beads * (6 * v + 10 * k)
        flops = beads * 250 + voxels * (20 + 10 * nb)
        per[m] = (read + acc * (beads * vecs * v + voxels * (1 + nb) * 8), flops)
    count = {m: 1 if one_each else CYCLE[m] for m in CYCLE}
    return tuple(moves_per_step * sum(count[m] * per[m][i] for m in CYCLE) for i in (0, 1))


def _mean_length(case):
    lo, hi = case["lo"], case["hi"]
    return float(lo) if hi <= lo else (hi - lo) / math.log(hi / lo)


def work(case):
    kind = case["kind"]
    if kind == "steric":
        n, m = case["beads"], case["segment"]
        return dict(bytes=2 * 12.0 * n + 24 * m, flops=10.0 * (n * (n - 1) / 2 + 2 * m * n))
    vox = case["nx"] * case["ny"] * case["nz"]
    if kind == "call":
        b, f = _moves_work(case, case["steps"], False)
        return dict(bytes=b + 2 * case["beads"] * 88 + vox * 16, flops=f)
    R, nb = case["replicas"], case["nb"]
    beads = R * _mean_length(case)
    state, grid = beads * (72 + 8 * nb), R * vox * 8.0 * (1 + nb)
    if kind == "mc":
        b, f = _moves_work(case, R * case["steps"] * max(1, case["rounds"]), case["one_each"])
        return dict(bytes=b + state, flops=f)
    if kind == "sample":
        b, f = _moves_work(case, R * case["steps"] * case["samples"], False)
        return dict(bytes=b + state + case["samples"] * (grid + 4 * beads), flops=f + case["samples"] * R * vox * 12.0)
    # energies and derivatives: chains and bonds read once, the grid written and read once
    elastic, field = 60.0, 8 * 12.0
    if kind == "energies":
        return dict(bytes=state + beads * (24 + 48) + 2 * grid, flops=beads * (elastic + field) + R * vox * 12.0)
    if kind == "gradient":
        return dict(bytes=beads * (24 + 40 + 8 * nb + 12) + grid, flops=beads * (2 * elastic + 2 * field))
    return dict(bytes=beads * (2 * 24 + 40 + 8 * nb + 24 + (24 if case["tangents"] else 0)) + 2 * grid,
                flops=beads * (4 * elastic + 3 * field))


# ---------------------------------------------------------------- 64-bit values

def _bind_table():
    """-ln of the single-site binding partition function for (marked, bound) tails."""
    f = np.zeros((3, 3))
    for nm in range(3):
        for s in range(3):
            z = sum(math.comb(nm, i) * math.comb(SITES - nm, s - i) * math.exp(-(i * E_MOD + (s - i) * E_NOMOD))
                    for i in range(s + 1) if s - i <= SITES - nm)
            f[nm, s] = -math.log(z)
    return f


def _elastic(r, t3, bonds):
    dr, a0, a1 = r[1:] - r[:-1], t3[:-1], t3[1:]
    eb, g, ep, epp, eta = bonds
    par = (a0 * dr).sum(1)
    dp = dr - a0 * par[:, None]
    bend = a1 - a0 - eta * dp
    return (0.5 * eb * (bend * bend).sum(1) + 0.5 * ep * (par - g) ** 2 + 0.5 * epp * (dp * dp).sum(1)).sum()


def _density(r, states, dims):
    """[1 + nb, voxels]: trilinear bead weight, and weight x state, per voxel."""
    n = torch.tensor(dims, dtype=torch.float64, device=r.device)
    width = VOXEL * n
    t = torch.remainder(r + 0.5 * width, width) / VOXEL - 0.5
    low = torch.floor(t.detach())
    frac = t - low
    low = torch.where(low < 0, n - 1, low).long()
    high = torch.where(low + 1 == n.long(), torch.zeros_like(low), low + 1)
    cols = [torch.ones(len(r), dtype=torch.float64, device=r.device)] + [s.double() for s in states.T]
    out = torch.zeros((len(cols), dims[0] * dims[1] * dims[2]), dtype=torch.float64, device=r.device)
    for c in range(8):
        bit = [(c >> j) & 1 for j in range(3)]
        w = 1.0
        at = 0
        for j, stride in zip(range(3), (1, dims[0], dims[0] * dims[1])):
            w = w * (frac[:, j] if bit[j] else 1 - frac[:, j])
            at = at + stride * (high if bit[j] else low)[:, j]
        out = out.index_add(1, at, torch.stack([w * k for k in cols]))
    return out


def _terms(c, chi, mu, dims, dev, grad=False):
    """(r, t3, elastic, binding, field, S, grid sums) of one chain in 64 bits."""
    r = torch.from_numpy(c["r"]).to(dev).requires_grad_(grad)
    t3 = torch.from_numpy(c["t3"]).to(dev).requires_grad_(grad)
    s, m = torch.from_numpy(c["states"]).to(dev), torch.from_numpy(c["marks"]).to(dev)
    nb, V = s.shape[1], VOXEL ** 3
    table = torch.from_numpy(_bind_table()).to(dev)
    el = _elastic(r, t3, tuple(float(x) for x in _bonds(1)[0]))
    bi = sum((table[m[:, b], s[:, b]] - mu[b] * s[:, b]).sum() for b in range(nb))
    pref, intra, x = _prefactors(nb, V)
    w = _density(r, s, dims)
    rho, vf = w[1:] / V, w[0] / V * BEAD_VOL
    over = vf > VF_LIMIT
    S = (torch.where(over, torch.zeros_like(vf), (V / BEAD_VOL) * vf * vf)).sum()
    fe = chi * S + (1e99 * vf[over]).sum()
    for b in range(nb):
        fe = fe + pref[b] * (rho[b] ** 2).sum() + intra[b] * (s[:, b] == 2).sum()
        for e in range(nb):
            if x[b, e]:
                fe = fe + x[b, e] * (rho[b] * rho[e]).sum()
    return r, t3, el, bi, fe, S, rho, w[0] / V, s


def exact(case, seed):
    kind = case["kind"]
    if kind in ("call", "mc", "sample"):
        return None  # a Markov chain's state: which moves are taken is decided, not computed
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "steric":
        return _steric_exact(case, seed, dev)
    chains, mu, chi = _chains(case, seed)
    dims = (case["nx"], case["ny"], case["nz"])
    if kind == "energies":
        rows = []
        for k, c in enumerate(chains):
            _, _, el, bi, fe, S, *_ = _terms(c, float(chi[k]), mu[k], dims, dev)
            rows.append([float(el), float(bi), float(fe), 0.0, float(S)])
        return np.array(rows)
    energies, grads, grads_t, terms = [], [], [], []
    weight = torch.linspace(0.5, 1.5, len(chains), dtype=torch.float64).tolist() if kind == "autograd" else None
    for k, c in enumerate(chains):
        r, t3, el, bi, fe, S, rho, dens, s = _terms(c, float(chi[k]), mu[k], dims, dev, grad=True)
        E = el + bi + fe
        (E * weight[k] if weight else E).backward()
        energies.append(E.detach())
        grads.append(r.grad)
        grads_t.append(t3.grad)
        nb = case["nb"]
        row = torch.zeros(14, dtype=torch.float64, device=dev)
        row[0], row[13] = S.detach(), (dens ** 2).sum().detach()
        for b in range(nb):
            row[1 + b] = (rho[b] ** 2).sum().detach()
            row[7 + b], row[10 + b] = (s[:, b] == 2).sum(), s[:, b].sum()
        for i, (b, e) in enumerate(((0, 1), (0, 2), (1, 2))):
            if e < nb:
                row[4 + i] = (rho[b] * rho[e]).sum().detach()
        terms.append(row)
    if kind == "gradient":
        return dict(dEdr=torch.cat(grads), terms=torch.stack(terms))
    out = dict(E=torch.stack(energies), r=torch.cat(grads))
    if case["tangents"]:
        out["t3"] = torch.cat(grads_t)
    return out


def _steric_exact(case, seed, dev):
    r, trial, ind0 = _steric_inputs(case, seed)
    m = case["segment"]
    after = r.copy()
    after[ind0:ind0 + m] = trial

    def energy(a, b, keep):
        """Sum over rows of a against b of the clash energy where keep(i, j)."""
        total = torch.zeros((), dtype=torch.float64, device=dev)
        for i0 in range(0, len(a), 512):
            x = a[i0:i0 + 512]
            d2 = sum((x[:, None, j] - b[None, :, j]) ** 2 for j in range(3))
            i = torch.arange(i0, i0 + len(x), device=dev)[:, None]
            use = keep(i, torch.arange(len(b), device=dev)[None, :]) & (d2 < EXCLUDED ** 2)
            f6 = (EXCLUDED ** 2 / d2[use]) ** 3
            total += (f6 * f6 - 2 * f6 + 1).sum()
        return total

    def moved(x):
        """Pairs with at least one bead of the segment, counted once."""
        x = torch.from_numpy(x).to(dev)
        seg = x[ind0:ind0 + m]
        return energy(seg, x, lambda i, j: (j < ind0) | (j >= ind0 + m) | (j > i + ind0))

    x = torch.from_numpy(r).to(dev)
    return dict(energy=float(energy(x, x, lambda i, j: j > i)), change=float(moved(after) - moved(r)))
