"""The work a user of so3lr_b200 has it do, as measurable cases: single molecules and periodic cells through the ASE-style calculator,
molecular dynamics in three ensembles from 192 to a million atoms, batches of independent molecules, the evaluation of a dataset of
padded batches, and the jax-md style loop (both neighbor lists updated and forces differentiated every step).

A case is a dict of plain values.  `prepare` makes what a user's program holds before the call, `run` is one pass."""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from so3lr_b200 import So3lr, So3lrCalculator, So3lrPotential, System, to_jax_md
from so3lr_b200 import md
from so3lr_b200 import workloads as W
from so3lr_b200.api import get_kgrid_mesh_shape
from so3lr_b200.batch import ShardedBatch

DENSITY = 333333 / 215.0 ** 3            # water molecules per cubic Angstrom of the million-atom box
KT = 300.0 * W.KB_EV
DT = 0.5                                 # fs
SKIN = 1.0                               # Angstrom, lists rebuilt when an atom moved further than half of it
LR_CUTOFF = 12.0
FRAMES = 8                               # position sets a calculator case cycles through


def listed():
    return [
        # geometry optimisation or sampling of one organic molecule: the smallest call, host positions in, host results out
        {"name": "ase_molecule_22", "kind": "ase", "atoms": 22},
        # single-point energy, forces and stress of independent frames of a periodic cell (no skin: lists are new every call)
        {"name": "ase_water_1536", "kind": "ase_cell", "molecules": 512},
        # thermostatted dynamics of the smallest periodic box, where a step is bound by launches
        {"name": "nvt_water_192", "kind": "md", "system": "water", "molecules": 64, "ensemble": "nvt", "kspace": "none", "steps": 10},
        # ordinary production dynamics of a solvent box
        {"name": "nvt_water_24k", "kind": "md", "system": "water", "molecules": 8000, "ensemble": "nvt", "kspace": "none", "steps": 4},
        # the same with the reciprocal-space Coulomb sum on a mesh, at a size beyond the L2
        {"name": "nvt_water_98k_pme", "kind": "md", "system": "water", "molecules": 32768, "ensemble": "nvt", "kspace": "pme", "steps": 2},
        # a solvated biopolymer with salt under a barostat: six elements, virial in every evaluation
        {"name": "npt_polymer_99k", "kind": "md", "system": "polymer", "edge": 100.0, "ensemble": "npt", "kspace": "none", "steps": 2},
        # the largest box on one GPU
        {"name": "nve_water_1m", "kind": "md", "system": "water", "molecules": 333333, "ensemble": "nve", "kspace": "none", "steps": 2},
        # screening of many small molecules at once: energy, forces, charges, Hirshfeld ratios and dipoles, host to host
        {"name": "molecules_512", "kind": "batch", "molecules": 512},
        # evaluation of a dataset: every batch holds other molecules, padded to one shape, some of them charged
        {"name": "dataset_6x32", "kind": "dataset", "batches": 6, "batch_size": 32, "charged": True},
        # the jax-md loop of the command line: lists updated every step without a skin, forces by differentiation
        {"name": "jaxmd_water_1536", "kind": "jaxmd", "molecules": 512},
        {"name": "jaxmd_water_24k", "kind": "jaxmd", "molecules": 8000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "ase", "ase_cell", "batch", "dataset", "jaxmd"])
    if kind == "md":
        ensemble = rng.choice(["nve", "nvt", "npt"])
        if ensemble == "npt" and rng.random() < 0.5:
            return {"kind": kind, "system": "polymer", "edge": round(rng.uniform(40.0, 100.0), 2), "ensemble": ensemble,
                    "kspace": rng.choice(["none", "none", "pme"]), "steps": 2}
        n = _log_int(rng, 64, 333333 if ensemble == "nve" else 100000)
        return {"kind": kind, "system": "water", "molecules": n, "ensemble": ensemble, "kspace": rng.choice(["none", "none", "pme"]),
                "steps": 10 if n < 1000 else 4 if n < 16000 else 2}
    if kind == "ase":
        return {"kind": kind, "atoms": _log_int(rng, 8, 150)}
    if kind == "ase_cell":
        return {"kind": kind, "molecules": _log_int(rng, 64, 8000)}
    if kind == "batch":
        return {"kind": kind, "molecules": _log_int(rng, 16, 2048)}
    if kind == "dataset":
        return {"kind": kind, "batches": 6, "batch_size": _log_int(rng, 4, 64), "charged": rng.random() < 0.5}
    return {"kind": kind, "molecules": _log_int(rng, 64, 8000)}


# ---- structures -------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _polymer(edge):
    return W.solvated_polymer(box=edge, n_polymer_atoms=int(round(5000 * (edge / 100.0) ** 3)))


@functools.lru_cache(maxsize=64)
def _molecule(atoms, variant):
    return W.molecule(np.random.default_rng(100 * atoms + variant), atoms)


def _molecule_set(rng, count, pick):
    """`count` molecules of 10 to 40 atoms that `pick` chooses from a library of structures, each a conformer (0.03 A) drawn from `rng`."""
    Zs, Rs, start = [], [], [0]
    for _ in range(count):
        Z, R = _molecule(int(pick.integers(10, 41)), int(pick.integers(0, 2)))
        Zs.append(Z)
        Rs.append(R + rng.normal(scale=0.03, size=R.shape))
        start.append(start[-1] + len(Z))
    return np.concatenate(Zs), np.concatenate(Rs), np.array(start, dtype=np.int32)


def _water(molecules, seed):
    return W.water_box(molecules, (molecules / DENSITY) ** (1.0 / 3.0), seed)


def _masses(Z):
    table = np.zeros(max(W.MASS) + 1, dtype=np.float32)
    for z, m in W.MASS.items():
        table[z] = m
    return table[Z]


def _velocities(Z, seed):
    rng = np.random.default_rng(seed)
    m = _masses(Z).astype(np.float64)
    v = rng.normal(size=(len(Z), 3)) * np.sqrt(KT * md.ACC_UNIT / m)[:, None]
    return v - (v * m[:, None]).sum(0) / m.sum()


class _Atoms:
    """The part of an ase.Atoms record that a calculator reads."""

    def __init__(self, Z, R, cell=None):
        self._Z, self._R, self._cell = Z, R, cell
        self.info = {}

    def get_positions(self):
        return self._R

    def get_atomic_numbers(self):
        return self._Z

    def get_cell(self):
        return self._cell if self._cell is not None else np.zeros((3, 3))

    def get_pbc(self):
        return np.array([self._cell is not None] * 3)


def _dataset_batch(rng, batch_size, charged):
    """One batch as a data loader hands it over: host arrays, both lists, padded to the shape that the largest batch has."""
    Z, R, gs = _molecule_set(rng, batch_size, rng)
    n, cap = len(Z), 40 * batch_size + 1
    seg = np.repeat(np.arange(batch_size), np.diff(gs))
    i = np.repeat(np.arange(n), np.diff(gs)[seg])
    j = np.concatenate([np.tile(np.arange(a, b), b - a) for a, b in zip(gs[:-1], gs[1:])])
    keep = i != j
    i, j = i[keep], j[keep]
    near = ((R[i] - R[j]) ** 2).sum(1) < 4.5 ** 2
    pad = lambda a, m, v: np.concatenate([a, np.full(m - len(a), v)])
    pairs = 40 * 39 * batch_size
    charge = np.zeros(batch_size + 1)
    if charged:
        charge[:-1] = rng.choice([0.0, 1.0, -1.0], size=batch_size, p=[0.875, 0.0625, 0.0625])
    return dict(positions=np.concatenate([R, np.zeros((cap - n, 3))]).astype(np.float32), atomic_numbers=pad(Z, cap, 1).astype(np.int32),
                idx_i=pad(i[near], pairs, cap).astype(np.int32), idx_j=pad(j[near], pairs, cap).astype(np.int32),
                idx_i_lr=pad(i, pairs, cap).astype(np.int32), idx_j_lr=pad(j, pairs, cap).astype(np.int32), cell=None,
                total_charge=charge.astype(np.float32), num_unpaired_electrons=np.zeros(batch_size + 1, np.float32),
                batch_segments=pad(seg, cap, batch_size).astype(np.int32), node_mask=np.arange(cap) < n,
                graph_mask=np.arange(batch_size + 1) < batch_size)


# ---- what a program holds before the call ------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "ase":
        Z, R = _molecule(case["atoms"], 0)
        frames = [_Atoms(Z, R + rng.normal(scale=0.03, size=R.shape)) for _ in range(FRAMES)]
        return {"run": _run_ase, "calc": So3lrCalculator(), "frames": frames, "next": 0}
    if kind == "ase_cell":
        Z, R, cell = _water(case["molecules"], seed)
        frames = [_Atoms(Z, R + rng.normal(scale=0.02, size=R.shape), cell) for _ in range(FRAMES)]
        return {"run": _run_ase, "calc": So3lrCalculator(calculate_stress=True), "frames": frames, "next": 0}
    if kind == "md":
        return _prepare_md(case, seed, rng)
    if kind == "batch":
        Z, R, gs = _molecule_set(rng, case["molecules"], np.random.default_rng(case["molecules"]))
        frames = [(R + rng.normal(scale=0.02, size=R.shape)).astype(np.float32) for _ in range(FRAMES)]
        return {"run": _run_batch, "batch": ShardedBatch(Z, gs, 1, 0, lr_cutoff=1000.0), "frames": frames, "next": 0}
    if kind == "dataset":
        batches = [_dataset_batch(rng, case["batch_size"], case["charged"]) for _ in range(case["batches"])]
        return {"run": _run_dataset, "fn": So3lr(lr_cutoff=1000.0), "batches": batches}
    if kind == "jaxmd":
        Z, R, cell = _water(case["molecules"], seed)
        box = np.diag(cell).copy()
        neighbor_fn, neighbor_fn_lr, energy_fn = to_jax_md(So3lrPotential(lr_cutoff=LR_CUTOFF), None, box, species=Z)
        dev = torch.device("cuda", 0)
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float32), device=dev)
        frac, V, m = t(R / box), t(_velocities(Z, seed + 1)), t(_masses(Z))
        return {"run": _run_jaxmd, "energy_fn": energy_fn, "R": frac, "V": V, "kick": (DT * md.ACC_UNIT / m)[:, None], "drift": t(DT / box),
                "box": box, "nbrs": neighbor_fn.allocate(frac, box=box), "nbrs_lr": neighbor_fn_lr.allocate(frac, box=box)}
    raise ValueError(kind)


def _prepare_md(case, seed, rng):
    if case["system"] == "polymer":
        Z, R, cell = _polymer(case["edge"])
        R = R + rng.normal(scale=0.02, size=R.shape)
    else:
        Z, R, cell = _water(case["molecules"], seed)
    system = System(Z, cell, cutoff_lr=LR_CUTOFF, damping=2.0, skin=SKIN)
    system.defer_skin_test(True, 0.05)
    if case["kspace"] == "pme":
        system.set_kspace(get_kgrid_mesh_shape(cell, 1.0), 2.4, "pme")
    V, m = _velocities(Z, seed + 1), _masses(Z)
    if case["ensemble"] == "nve":
        init, apply = md.nve(system, DT)
        state = init(R, m, velocity=V)
    elif case["ensemble"] == "nvt":
        init, apply = md.nvt_nose_hoover(system, DT, KT)
        state = init(R, m, velocity=V)
    else:
        init, apply = md.npt_nose_hoover(system, DT, 1.0 * md.BAR, KT)
        state = init(R, cell, m, velocity=V)
    return {"run": _run_md, "apply": apply, "state": state, "steps": case["steps"], "system": system}


# ---- one pass ----------------------------------------------------------------------------------------------------------------
def run(state):
    return state["run"](state)


def _frame(s):
    f = s["frames"][s["next"]]
    s["next"] = (s["next"] + 1) % len(s["frames"])
    return f


def _run_ase(s):
    atoms = _frame(s)
    s["calc"].get_forces(atoms)
    out = dict(s["calc"].results)
    if atoms.get_pbc().any():
        out.pop("dipole")         # of a periodic cell: depends on where the cell is cut, and cancels to a few parts in a thousand
    return out


def _run_batch(s):
    return s["batch"].compute_host(_frame(s))


def _run_md(s):
    st = s["state"] = s["apply"](s["state"], s["steps"])
    out = {"position": st.position, "velocity": st.velocity, "force": st.force, "energy": st.energy}
    if st.chain is not None:
        out["chain"] = st.chain
    if st.box is not None:
        out["box"] = st.box
    return out


def _run_dataset(s):
    return [s["fn"](b) for b in s["batches"]]


def _run_jaxmd(s):
    """One leapfrog step as a caller's integrator makes it around the two list updates and the differentiated energy."""
    s["nbrs"] = s["nbrs"].update(s["R"], box=s["box"])
    s["nbrs_lr"] = s["nbrs_lr"].update(s["R"], box=s["box"])
    R = s["R"].clone().requires_grad_(True)
    E = s["energy_fn"](R, neighbor=s["nbrs"].idx, neighbor_lr=s["nbrs_lr"].idx, box=s["box"])
    (g,) = torch.autograd.grad(E, R)
    s["V"] = s["V"] - s["kick"] * g
    s["R"] = s["R"] + s["drift"] * s["V"]
    return {"energy": E.detach(), "forces": -g, "position": s["R"], "velocity": s["V"],
            "overflow": bool(s["nbrs"].did_buffer_overflow or s["nbrs_lr"].did_buffer_overflow)}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------
def work(case):
    """Operations of the network and the pair terms in their cheapest known exact form (radial filters as functions of the distance,
    spherical filters as the small networks they are), inputs read and results written once, weights read once."""
    kind = case["kind"]
    evals, io = 1, 60
    if kind == "ase":
        n, per_edge_list, pairs = case["atoms"], 14.0, case["atoms"] / 2.0
    elif kind in ("batch", "dataset"):
        n = 25 * case["molecules"] if kind == "batch" else 25 * case["batch_size"] * case["batches"]
        per_edge_list, pairs, io = 18.0, 28.0, 60 if kind == "batch" else 60 + 46 * 16
    else:
        n = int(round(3 * DENSITY * case["edge"] ** 3)) if case.get("system") == "polymer" else 3 * case["molecules"]
        per_edge_list, pairs = 38.6, 363.0
        evals = case.get("steps", 1)
        if kind == "jaxmd":
            io = 60 + int((38.6 + 363.0) * 8)
    edge_flops = 2 * (1024 + 8448 + 1024) * 3           # forward + reverse, per directed entry and layer
    atom_flops = 2 * 3 * (3 * 70700 + 45000)
    flops = evals * n * (3 * per_edge_list * edge_flops + atom_flops + 150 * pairs)
    return {"bytes": float(n * io + 4 * 530238), "flops": float(flops)}


def tolerance(case):
    """Four times what the path differs by from a float64 evaluation on the same inputs (2-norm / largest): single molecules 5e-6 / 1e-5,
    periodic cells 1.1e-6 / 5e-6 (stress 3e-6 / 4e-6), batches 2e-6 / 1e-5, forces behind float32 fractional coordinates 7e-6 / 3e-5.  Ten
    steps of dynamics: velocities and forces 1.1e-5 / 7e-5; in large boxes single atoms differ more (5e-4 between two runs of the
    same code), because a position near 200 A is rounded to 1.5e-5 A in every step."""
    kind = case["kind"]
    if kind == "md":
        return {"rel": 5e-5, "max": 2e-3}
    if kind == "jaxmd":
        return {"rel": 3e-5, "max": 1.5e-4}
    return {"rel": 2e-5, "max": 1e-4}
