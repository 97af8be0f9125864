"""Work that programs built on this engine have it do, as cases to be timed.

Five kinds of replica-exchange blocks, full energies of poses and snapshots,
the energy adjoint, the reference's own GPU energy call, and the two
post-processing tools. Sizes are those of the benchmark workloads
(remcdockingsimulator_b200/synth.py), of the reference's two-chain structures
and of the tests; `draw` gives others from the same ranges.

Systems are made here rather than by synth.py, whose random insertion takes
half a minute for 64 systems: chains are compact lattice walks with 3.8 A
bonds under a random rotation, chains and crowders sit on jittered lattice
sites without overlap, at the same densities.
"""
import ctypes
import math

import numpy as np
import torch

from remcdockingsimulator_b200 import post
from remcdockingsimulator_b200.engine import Engine, make_params
from remcdockingsimulator_b200.model import (AminoAcidTable, Molecule, System, geometric_ladder,
                                             reference_step_ladder)
from remcdockingsimulator_b200.reference_abi import abi, pack_reference_layout

BOND = 3.8


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one replica-exchange block (Metropolis steps, then one exchange
        # round) and the state read back, as a driver loop does. Threads and
        # CTAs per replica are the autotuner's choices for these workloads.
        # - the smallest docking problem: two chains (76 + 24 residues), 20
        #   temperatures; every step moves a chain
        dict(name="run_two_chains", kind="run", systems=1, chains="76,24", crowders=0, radius=12.0,
             box=100.0, replicas=20, steps=1000, model="wall", threads=128, cluster=1),
        # - the same pair among 400 crowders, 32 temperatures
        dict(name="run_crowded", kind="run", systems=1, chains="76,24", crowders=400, radius=12.0,
             box=200.0, replicas=32, steps=1000, model="wall", threads=128, cluster=1),
        # - a batch of 64 unlike systems, 16 temperatures each: the throughput
        #   workload (2-8 chains of 20-300 residues, 0-1000 crowders)
        dict(name="run_batch", kind="run", systems=64, chains="", crowders=1000, radius=12.0,
             box=0.0, replicas=16, steps=1000, model="wall", threads=128, cluster=1),
        # - one large assembly: 60 chains of 150 residues, 2000 crowders, 32
        #   temperatures, four CTAs per replica
        dict(name="run_assembly", kind="run", systems=1, chains="150*60", crowders=2000,
             radius=10.0, box=400.0, replicas=32, steps=300, model="wall", threads=256, cluster=4),
        # - the reference's own settings, which the command-line driver takes
        #   by default: (6/r)^6 crowders with a 15 A cutoff that also rotate,
        #   its step-size ladder, odd chain lengths
        dict(name="run_reference_model", kind="run", systems=1, chains="129,57,201", crowders=233,
             radius=6.0, box=150.0, replicas=20, steps=1000, model="reference", threads=128,
             cluster=1),
        # new poses of a docked pair scored: upload, full energy (the
        # trajectory tool's use; small, so calls and launches count)
        dict(name="score_poses", kind="score", chains="76,24", crowders=0, radius=12.0, box=118.4,
             replicas=100, model="reference"),
        # the full energy of many crowded snapshots already on the device
        dict(name="energy_snapshots", kind="energy", chains="76,24", crowders=400, radius=12.0,
             box=200.0, replicas=4096, model="wall"),
        # dE/dlambda of every replica between two sampling chunks (the
        # driver's --sensitivity)
        dict(name="sensitivity", kind="sensitivity", chains="76,24", crowders=400, radius=12.0,
             box=200.0, replicas=32, model="wall"),
        # forces, torques and parameter derivatives of snapshots, for a fit
        dict(name="adjoint_snapshots", kind="adjoint", chains="76,24", crowders=400, radius=12.0,
             box=200.0, replicas=512, model="wall"),
        # the reference program's energy call on one replica in its own device
        # layout, on a stream, for a structure of some 1300 beads
        dict(name="reference_call", kind="refcall", chains="150,150,287,120", crowders=600,
             radius=6.0, box=180.0, model="reference"),
        # bound poses of two chains rebuilt and compared with the loaded pair
        dict(name="pdbgen_poses", kind="pdbgen", chains="76,24", crowders=0, radius=12.0,
             box=118.4, frames=1000),
        # a trajectory of four equal chains compared with a reference
        # structure, in both molecule orders
        dict(name="trajectory_drms", kind="drms", chains="150*4", crowders=0, radius=12.0,
             box=150.0, frames=500),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shorter(case, flops=4e10):
    """The case with fewer steps where chains alone make every step costly."""
    w = work(case)["flops"]
    return dict(case, steps=max(10, int(case["steps"] * flops / w))) if w > flops else case


def draw(rng):
    kind = rng.choice(["run", "run", "run", "batch", "score", "energy", "sensitivity", "adjoint",
                       "refcall", "pdbgen", "drms"])
    model = rng.choice(["wall", "reference"])
    radius = 12.0 if model == "wall" else 6.0
    chains = ",".join(str(rng.randint(20, 300)) for _ in range(rng.randint(2, 8)))
    if kind == "run":
        crowders = rng.choice([0, _log_int(rng, 20, 1000)])
        case = dict(kind="run", systems=1, chains=chains, crowders=crowders, radius=radius,
                    box=_box(chains, crowders, radius, rng.uniform(0.1, 0.25)),
                    replicas=rng.randint(8, 40), steps=_log_int(rng, 60, 1000), model=model,
                    threads=rng.choice([128, 256]), cluster=rng.choice([1, 1, 2]))
        return _shorter(case)
    if kind == "batch":
        case = dict(kind="run", systems=rng.randint(4, 24), chains="", crowders=1000, radius=radius,
                    box=0.0, replicas=rng.randint(5, 20), steps=_log_int(rng, 60, 500), model=model,
                    threads=rng.choice([128, 256]), cluster=1)
        return _shorter(case)
    if kind == "pdbgen":
        return dict(kind="pdbgen", chains=chains, crowders=0, radius=radius,
                    box=_box(chains, 0, radius, 0.1), frames=_log_int(rng, 20, 1500))
    if kind == "drms":
        chains = "%d*%d" % (rng.randint(20, 200), rng.randint(2, 5))
        return dict(kind="drms", chains=chains, crowders=0, radius=radius,
                    box=_box(chains, 0, radius, 0.1), frames=_log_int(rng, 20, 500))
    crowders = rng.choice([0, _log_int(rng, 20, 800)])
    case = dict(kind=kind, chains=chains, crowders=crowders, radius=radius,
                box=_box(chains, crowders, radius, rng.uniform(0.1, 0.25)),
                model="reference" if kind == "refcall" else model)
    if kind != "refcall":
        most = {"score": 200, "energy": 1000, "sensitivity": 64, "adjoint": 128}[kind]
        case["replicas"] = _log_int(rng, 4, most)
    return case


# ------------------------------------------------------------------ inputs
def _lengths(chains):
    out = []
    for part in chains.split(","):
        n, _, times = part.partition("*")
        out += [int(n)] * int(times or 1)
    return out


def _extent(n):
    """Radius of the sphere around a compact lattice walk of n beads."""
    return 0.5 * math.sqrt(3.0) * BOND * (math.ceil(n ** (1.0 / 3.0)) + 1)


def _box(chains, crowders, radius, phi):
    """Box edge for the packing fraction phi, never too small for the chains."""
    n = _lengths(chains)
    vol = crowders * 4.0 / 3.0 * math.pi * radius ** 3 + sum(n) * 4.0 / 3.0 * math.pi * 27.0
    big = 2.0 * max(_extent(k) for k in n) + 2.0
    room = len(n) * big ** 3 + 1.8 * crowders * (2.0 * radius + 1.0) ** 3
    return round(max((vol / phi) ** (1.0 / 3.0), room ** (1.0 / 3.0),
                     math.ceil(len(n) ** (1.0 / 3.0)) * big, 80.0), 1)


def _rotation(g):
    q = g.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])


def _walk(n, g):
    """A compact walk of n beads: up and down the rows of a cubic lattice."""
    a = max(1, math.ceil(n ** (1.0 / 3.0)))
    k = np.arange(a ** 3)
    z, y, x = k // (a * a), (k // a) % a, k % a
    y = np.where(z % 2, a - 1 - y, y)
    x = np.where((k // a) % 2, a - 1 - x, x)
    p = np.stack([x, y, z], axis=1)[:n] * BOND
    p = (p - p.mean(axis=0)) @ _rotation(g).T
    return p.astype(np.float32)


def _sites(g, n, box, size, taken, clear):
    """n points of a jittered lattice, `size` apart or more, none within
    `clear` of a point in `taken` (minimum image)."""
    k = max(1, int(box // size))
    while True:
        step = box / k
        s = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
        s = (s + 0.5) * step + g.uniform(-0.5, 0.5, size=s.shape) * max(step - size, 0.0) * 0.95
        if len(taken):
            dev = "cuda" if torch.cuda.is_available() else "cpu"
            a, b = (torch.from_numpy(v.astype(np.float32)).to(dev) for v in (s, taken))
            near = torch.full((len(s),), math.inf, device=dev)
            for c in range(0, len(taken), 2048):
                d = a[:, None, :] - b[None, c:c + 2048, :]
                d -= box * torch.round(d / box)
                near = torch.minimum(near, d.square_().sum(-1).amin(1))
            s = s[(near >= clear * clear).cpu().numpy()]
        if len(s) >= n:
            return s[g.permutation(len(s))[:n]]
        k += 1
        if k * size > 1.3 * box:
            raise ValueError("box too small for %d sites" % n)


def _system(g, table, lengths, crowders, radius, box, model):
    big = 2.0 * max(_extent(n) for n in lengths) + 2.0
    centres = _sites(g, len(lengths), box, big, np.zeros((0, 3)), 0.0)
    mols = []
    for n, c in zip(lengths, centres):
        m = Molecule.from_beads(g.integers(0, 20, size=n), _walk(n, g))
        m.set_position(c.astype(np.float32))
        mols.append(m)
    if crowders:
        beads = np.concatenate([m.pos for m in mols]).astype(np.float64)
        at = _sites(g, crowders, box, 2.0 * radius, beads, radius + 3.0).astype(np.float32)
        zero = np.zeros(1, np.int32)
        for c in np.mod(at, np.float32(box)):
            mols.append(Molecule(zero, c[None, :].copy(), np.zeros((1, 3), np.float32), c.copy(),
                                 np.array([1.0, 0.0, 0.0, 0.0]), True))
    return System(mols, float(np.float32(box)), table, crowder_radius=radius,
                  translate_only_crowders=model == "wall")


def _table(g):
    """Contacts U[-1.2, 0.2] kT, symmetric, as the raw table of lambda = 0.16."""
    t = AminoAcidTable.synthetic(vdw=6.0)
    eps = g.uniform(-1.2, 0.2, size=(20, 20))
    t.pairs = ((np.triu(eps) + np.triu(eps, 1).T) / 0.16 - 2.27).astype(np.float32)
    return t


def _params(model):
    if model == "wall":
        return make_params(lambda_=0.16, crowder_mode=1, crowder_cutoff=0.0)
    return make_params()


def _systems(case, seed):
    g = np.random.default_rng(seed)
    table = _table(g)
    if case.get("chains"):
        lengths = [_lengths(case["chains"])] * case.get("systems", 1)
        return [_system(g, table, n, case["crowders"], case["radius"], case["box"], case["model"]
                        if "model" in case else "wall") for n in lengths], g
    # a batch of unlike systems; the sizes belong to the case, the rest to the seed
    sizes = np.random.default_rng(case["systems"] * 7919 + case["replicas"] + 2)
    out = []
    for _ in range(case["systems"]):
        n = [int(sizes.integers(20, 301)) for _ in range(int(sizes.integers(2, 9)))]
        crowders = int(sizes.integers(0, case["crowders"] + 1))
        box = _box(",".join(map(str, n)), crowders, case["radius"], float(sizes.uniform(0.1, 0.25)))
        out.append(_system(g, table, n, crowders, case["radius"], box, case["model"]))
    return out, g


def _batch_sizes(case):
    """(beads of each chain, crowders) of every system, without building it."""
    if case.get("chains"):
        return [(_lengths(case["chains"]), case["crowders"])] * case.get("systems", 1)
    sizes = np.random.default_rng(case["systems"] * 7919 + case["replicas"] + 2)
    out = []
    for _ in range(case["systems"]):
        n = [int(sizes.integers(20, 301)) for _ in range(int(sizes.integers(2, 9)))]
        crowders = int(sizes.integers(0, case["crowders"] + 1))
        sizes.uniform(0.1, 0.25)
        out.append((n, crowders))
    return out


def _moved(system, frames, g):
    """States of `frames` poses of a system: every chain turned and shifted
    within its surroundings, every crowder shifted a little."""
    pos0, rel0, cen0, _ = system.state()
    n_mol, box = system.n_mol, system.box
    chains = [m for m in system.molecules if not m.crowder]
    shift = np.where(np.array([m.crowder for m in system.molecules])[:, None], 0.6, 2.0)
    cen = np.mod(cen0[None] + g.uniform(-1, 1, size=(frames, n_mol, 3)) * shift, box)
    cen = np.minimum(cen.astype(np.float32), np.nextafter(np.float32(box), np.float32(0)))
    quat = np.zeros((frames, n_mol, 4))
    quat[:, :, 0] = 1.0
    rel = np.broadcast_to(rel0, (frames,) + rel0.shape).copy()
    axis = g.normal(size=(frames, len(chains), 3)) * 0.15
    q = np.concatenate([np.ones((frames, len(chains), 1)), axis], axis=2)
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    quat[:, :len(chains)] = q
    b = 0
    for k, m in enumerate(chains):
        w, x, y, z = (q[:, k, i, None] for i in range(4))
        u = q[:, k, None, 1:]
        v = m.rel[None].astype(np.float64)
        t = 2.0 * np.cross(u, v)
        rel[:, b:b + m.n] = v + w[:, :, None] * t + np.cross(u, t)
        b += m.n
    mol = np.repeat(np.arange(n_mol), [m.n for m in system.molecules])
    pos = (rel + cen[:, mol]).astype(np.float32)
    return (pos.reshape(-1, 3), np.ascontiguousarray(rel.reshape(-1, 3), np.float32),
            cen.reshape(-1, 3), quat.reshape(-1, 4))


def _pinned(a):
    a = np.ascontiguousarray(a)
    t = torch.from_numpy(a)
    return (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)).numpy()


def prepare(case, seed):
    kind = case["kind"]
    systems, g = _systems(case, seed)
    s = systems[0]
    if kind == "run":
        R = case["replicas"]
        eng = Engine(systems, R, _params(case["model"]))
        if case["model"] == "wall":
            t, r = np.full(R, 0.5, np.float32), np.full(R, 0.2)
        else:
            t, r = reference_step_ladder(R)
        n = len(systems)
        eng.set_replica_params([geometric_ladder(290.0, 450.0, R)] * n, np.tile(t, n), np.tile(r, n))
        # the molecules' centres in shared memory too, where they fit beside the beads
        eng.set_schedule(case["threads"], s.n_beads < 8000)
        if case["cluster"] > 1:
            eng.set_cluster(case["cluster"])
        eng.energy_full()
        nb, nm = sum(x.n_beads for x in systems) * R, sum(x.n_mol for x in systems) * R
        out = [torch.empty(k, dtype=d, pin_memory=True).numpy()
               for k, d in (((nb, 3), torch.float32), ((nb, 3), torch.float32),
                            ((nm, 3), torch.float32), ((nm, 4), torch.float64))]
        return dict(kind=kind, engine=eng, out=out, steps=case["steps"], seed=1000 + seed, block=0)
    if kind == "refcall":
        pos, meta = pack_reference_layout(s, 32)
        L = abi()
        table = torch.empty(400, dtype=torch.float32, device="cuda")
        pairs = np.ascontiguousarray(s.table.pairs, np.float32)
        L.copyLJPotentialDataToDevice(ctypes.c_void_p(table.data_ptr()), pairs.ctypes.data)
        L.CUDA_setBoxDimension(s.box)
        grid = pos.shape[0] // 32
        return dict(kind=kind, pos=torch.from_numpy(pos).cuda(), meta=torch.from_numpy(meta).cuda(),
                    table=table, grid=grid, out=torch.zeros(grid * grid, device="cuda"), box=s.box)
    if kind in ("pdbgen", "drms"):
        F = case["frames"]
        pos, _, cen, quat = _moved(s, F, g)
        ms = np.concatenate([[0], np.cumsum([m.n for m in s.molecules])]).astype(np.int32)
        ref = np.concatenate([m.pos for m in s.molecules]).astype(np.float32)
        return dict(kind=kind, molecules=s.molecules, box=s.box, ms=ms, ref=ref,
                    quat=quat.reshape(F, -1, 4), centre=cen.reshape(F, -1, 3),
                    frames=pos.reshape(F, -1, 3))
    R = case["replicas"]
    eng = Engine([s], R, _params(case["model"]))
    poses = [_pinned(a) for a in _moved(s, R, g)]
    if kind != "score":
        eng.upload_state(*poses)
        eng.sync()
    return dict(kind=kind, engine=eng, poses=poses)


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "run":
        eng, k, n = state["engine"], state["block"], state["steps"]
        eng.run(1, n, state["seed"], k * n, k)
        state["block"] = k + 1
        pos, rel, centre, quat = eng.download_state(out=state["out"])
        return dict(pos=pos, rel=rel, centre=centre, quat=quat, energy=eng.energies(),
                    temperature=eng.temperature_map(), moves=eng.counters())
    if kind == "refcall":
        L, p = abi(), ctypes.c_void_p
        L.CUDA_setBoxDimension(state["box"])
        L.CUDA_EonDevice_async(p(state["pos"].data_ptr()), p(state["meta"].data_ptr()), None, None,
                               None, p(state["table"].data_ptr()), p(state["out"].data_ptr()),
                               state["grid"], 32, state["pos"].shape[0], 0,
                               p(torch.cuda.current_stream().cuda_stream))
        return state["out"]
    if kind == "pdbgen":
        mols = state["molecules"]
        pos, centre = post.rebuild(mols, [1] * len(mols), state["box"], state["quat"],
                                   state["centre"])
        return (pos, centre) + post.drms(pos, state["ref"], state["ms"])
    if kind == "drms":
        return post.drms(state["frames"], state["ref"], state["ms"], reverse=True)
    if kind == "score":
        state["engine"].upload_state(*state["poses"])
        return state["engine"].energy_full()
    if kind == "energy":
        return state["engine"].energy_full()
    if kind == "sensitivity":
        return state["engine"].dE_dlambda()
    return state["engine"].adjoint()


# ------------------------------------------------------------------ work
RESIDUE_FLOP, CROWDER_FLOP = 41, 26  # per pair energy, a fused multiply-add as two


def work(case):
    kind = case["kind"]
    if kind == "run":
        flops = nbytes = 0.0
        for n, crowders in _batch_sizes(case):
            beads, mols = sum(n) + crowders, len(n) + crowders
            per = 0.0  # one step: the moved molecule's pairs, before and after
            for k in n:
                per += k * ((sum(n) - k) * RESIDUE_FLOP + crowders * CROWDER_FLOP)
            moves = 1.0 if case["model"] == "wall" else 0.5  # a turned crowder stays where it is
            per += moves * crowders * (beads - 1) * CROWDER_FLOP
            flops += case["replicas"] * case["steps"] * 2.0 * per / mols
            nbytes += case["replicas"] * 2.0 * (24.0 * beads + 44.0 * mols)
        return dict(bytes=nbytes, flops=flops)
    n, crowders = _lengths(case["chains"]), case["crowders"]
    beads, mols = sum(n) + crowders, len(n) + crowders
    rr = (sum(n) ** 2 - sum(k * k for k in n)) / 2.0
    cr = sum(n) * crowders + crowders * (crowders - 1) / 2.0
    energy = rr * RESIDUE_FLOP + cr * CROWDER_FLOP
    if kind == "refcall":
        return dict(bytes=32.0 * beads, flops=energy)
    if kind == "pdbgen":
        return dict(bytes=case["frames"] * (24.0 * beads + 56.0 * mols),
                    flops=case["frames"] * (10.0 * rr + 30.0 * beads))
    if kind == "drms":
        return dict(bytes=case["frames"] * 12.0 * beads, flops=case["frames"] * 20.0 * rr)
    R = case["replicas"]
    if kind == "score":
        return dict(bytes=R * (24.0 * beads + 44.0 * mols), flops=R * energy)
    if kind == "energy":
        return dict(bytes=R * 12.0 * beads, flops=R * energy)
    if kind == "sensitivity":
        return dict(bytes=R * 12.0 * beads, flops=R * rr * RESIDUE_FLOP)
    return dict(bytes=R * (36.0 * beads + 48.0 * mols + 3216.0), flops=R * 2.0 * energy)


# ------------------------------------------------------------------ 64 bits
def _energies(system, pos, p, derivatives=False, rel=None):
    """Energy of every frame of pos [frames, beads, 3] in 64 bits, and with
    `derivatives` the forces, the molecules' forces and torques, and the
    derivatives by lambda, the Debye length and the contact energies."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f8 = dict(dtype=torch.float64, device=dev)
    types, mol, charge = [], [], []
    for k, m in enumerate(system.molecules):
        types += [20] * m.n if m.crowder else list(m.types)
        mol += [k] * m.n
    types, mol = torch.tensor(np.array(types), device=dev), torch.tensor(mol, device=dev)
    t = system.table
    vdw = torch.tensor(list(map(float, t.vdw)) + [2.0 * system.crowder_radius], **f8)
    charge = torch.tensor(list(map(float, t.charge)) + [0.0], **f8)
    raw = torch.zeros(21, 21, **f8)
    raw[:20, :20] = torch.tensor(t.pairs.astype(np.float64).reshape(20, 20), **f8)
    i, j = torch.triu_indices(len(mol), len(mol), 1, device=dev)
    keep = mol[i] != mol[j]
    i, j = i[keep], j[keep]
    ti, tj = types[i], types[j]
    wall = (ti == 20) | (tj == 20)
    lj_cf = float(p.lj_cf) * float(p.kbt_cf)
    sigma = 0.5 * (vdw[ti] + vdw[tj])
    slope = raw[ti, tj] - float(p.e0)
    eps = float(p.lambda_) * slope
    qq = charge[ti] * charge[tj] * float(p.dh_const) * float(p.kbt_cf)
    xi, L = float(p.debye_length), float(system.box)
    cut = float(p.crowder_cutoff) if p.crowder_cutoff > 0 else math.inf
    power = 12 if p.crowder_mode else 6
    reach = sigma if p.crowder_mode else torch.full_like(sigma, 6.0)
    strength = lj_cf * (float(p.crowder_eps) if p.crowder_mode else 1.0)
    a, b = torch.minimum(ti, tj), torch.maximum(ti, tj)
    out = {k: [] for k in ("energy", "forces", "mol_force_torque", "dE_dlambda", "dE_dxi", "dE_deps")}
    for f in range(len(pos)):
        x = torch.as_tensor(pos[f]).to(**f8)
        d = x[i] - x[j]
        d = d - L * torch.round(d / L)
        r = d.square().sum(-1).sqrt()
        s6 = (sigma / r) ** 6
        flip = (eps > 0) & (r < sigma * 2.0 ** (1.0 / 6.0))
        shape = torch.where(flip, 2.0 - 4.0 * s6 * (1.0 - s6), 4.0 * s6 * (1.0 - s6)) * lj_cf
        dh = qq * torch.exp(-r / xi) / r
        e_wall = torch.where(r < cut, strength * (reach / r) ** power, torch.zeros_like(r))
        out["energy"].append(torch.where(wall, e_wall, eps * shape + dh).sum())
        if not derivatives:
            continue
        steep = 24.0 * lj_cf * s6 * (1.0 - 2.0 * s6) / r * torch.where(flip, -1.0, 1.0)
        push = torch.where(wall, power * e_wall / r, eps * steep + dh * (1.0 / xi + 1.0 / r))
        v = d * (push / r)[:, None]
        F = torch.zeros_like(x).index_add_(0, i, v).index_add_(0, j, -v)
        ft = torch.zeros(system.n_mol, 6, **f8)
        ft.index_add_(0, mol, torch.cat([F, torch.cross(torch.as_tensor(rel[f]).to(**f8), F, dim=1)], 1))
        zero = torch.zeros_like(r)
        deps = torch.zeros(441, **f8).index_add_(0, a * 21 + b, torch.where(wall, zero, shape))
        deps = deps.view(21, 21)[:20, :20]
        out["forces"].append(F)
        out["mol_force_torque"].append(ft)
        out["dE_dlambda"].append(torch.where(wall, zero, shape * slope).sum())
        out["dE_dxi"].append(torch.where(wall, zero, dh * r / xi ** 2).sum())
        out["dE_deps"].append(deps + deps.T - torch.diag(torch.diag(deps)))
    got = {k: torch.stack(v).cpu().numpy() for k, v in out.items() if v}
    if derivatives:
        got["forces"] = got["forces"].reshape(-1, 3)
        got["mol_force_torque"] = got["mol_force_torque"].reshape(-1, 6)
    return got


def _distances(x, starts, ref, swap):
    """Sum over the bead pairs of different molecules of |d - d_ref|, 64 bits."""
    total, pairs = torch.zeros(len(x), dtype=x.dtype, device=x.device), 0
    for I in range(len(starts) - 1):
        for J in range(I + 1, len(starts) - 1):
            a, b = slice(starts[I], starts[I + 1]), slice(starts[J], starts[J + 1])
            d = torch.cdist(x[:, a], x[:, b], compute_mode="donot_use_mm_for_euclid_dist")
            A, B = (b, a) if swap else (a, b)
            e = torch.cdist(ref[A], ref[B], compute_mode="donot_use_mm_for_euclid_dist")
            total += (d - e).abs().sum((1, 2))
            pairs += e.numel()
    return total / pairs


def _drms(frames, ref, starts, reverse):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(frames).to(device=dev, dtype=torch.float64)
    ref = torch.as_tensor(ref).to(device=dev, dtype=torch.float64)
    starts = [int(v) for v in starts]
    d = _distances(x, starts, ref, False)
    if reverse:
        d = torch.minimum(d, _distances(x, starts, ref, True))
    return (d.cpu().numpy(), None, None, None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        return None  # a trajectory: its value is the engine's own random walk
    systems, g = _systems(case, seed)
    s = systems[0]
    if kind == "refcall":
        e = np.zeros((-(-s.n_beads // 32)) ** 2)
        p = _params("reference")
        e[0] = _energies(s, [s.state()[0]], p)["energy"][0] / float(p.kbt_cf)
        return torch.from_numpy(e)
    if kind in ("pdbgen", "drms"):
        F = case["frames"]
        pos, _, cen, quat = _moved(s, F, g)
        starts = np.concatenate([[0], np.cumsum([m.n for m in s.molecules])])
        ref = np.concatenate([m.pos for m in s.molecules]).astype(np.float32)
        if kind == "drms":
            return _drms(pos.reshape(F, -1, 3), ref, starts, True)
        box, c = s.box, cen.reshape(F, -1, 3).astype(np.float64)
        c0 = s.molecules[0].centre.astype(np.float64)
        first = c[:, :1] - box * np.round((c[:, :1] - c0) / box)
        c = np.concatenate([first, c[:, 1:] - box * np.round((c[:, 1:] - first) / box)], axis=1)
        q = quat.reshape(F, -1, 4)
        q = q / np.linalg.norm(q, axis=2, keepdims=True)
        x = []
        for k, m in enumerate(s.molecules):
            u, v = q[:, k, None, 1:], m.rel[None].astype(np.float64)
            t = 2.0 * np.cross(u, v)
            x.append(v + q[:, k, None, :1] * t + np.cross(u, t) + c[:, k, None])
        x = np.concatenate(x, axis=1)
        return (x, c) + _drms(x, ref, starts, False)
    pos, rel, _, _ = _moved(s, case["replicas"], g)
    R = case["replicas"]
    got = _energies(s, pos.reshape(R, -1, 3), _params(case["model"]), kind in ("sensitivity", "adjoint"),
                    rel.reshape(R, -1, 3))
    if kind in ("score", "energy"):
        return got["energy"]
    if kind == "sensitivity":
        return got["dE_dlambda"]
    return got
