"""Sizes at which a rule of a launch changes what a kernel does: tiles handed out by the queue (csrc/attention_tc.cu), rows shared by several
warps and the queue of the pairs inside the cutoff (csrc/pair_kernels.cu), both lists' row kernels side by side (csrc/nlist.cu).

The kernels behind them evaluate the same FP32 formulas in another order of summation: tolerances of the variant tests, 2e-6 relative
and 5e-5 eV/A.  The common reference is `by_hand`: lists from a float64 search over all pairs, evaluated through the caller-supplied-list
entry point, whose pair kernel never shares a row between warps and whose lists no kernel of csrc/nlist.cu has touched."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DENSITY = 333333 / 215.0 ** 3
CHILD = r"""
import os, sys, numpy as np, torch
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import test_gpu_launch_shapes as T
from so3lr_b200 import workloads as W
from so3lr_b200.engine import System
sms = torch.cuda.get_device_properties(0).multi_processor_count
# 128 pairs a tile, 20.03 pairs an atom: 7 tiles per CTA, on either side of 8, where the queue begins, and odd counts beyond
for k, tiles in enumerate((7.0, 7.9, 8.1, 8.45, 10.3)):
    n = int(tiles * sms * 128 / 20.03 / 3)
    Z, R, cell = W.water_box(n, (n / (333333 / 215.0 ** 3)) ** (1 / 3), 50 + k)
    s = System(Z, cell, cutoff_lr=6.0, damping=2.0)
    Rd = torch.tensor(np.asarray(R, dtype=np.float32), device="cuda")
    first, o = s.compute(Rd)["forces"].clone(), s.compute(Rd)          # the queue serves every launch of an evaluation, and the next one
    if "SO3LR_B200_ATTENTION" not in os.environ:
        assert (T.tiles_per_block(s.valid_edges() // 2) >= 8) == (tiles > 8), (tiles, s.valid_edges())
    assert (first - o["forces"]).abs().max().item() <= 5e-5
    np.savez(f"{sys.argv[2]}.{k}.npz", E=o["energy"].double().cpu().numpy().sum(), F=o["forces"].cpu().numpy(), pairs=s.valid_edges())
"""


def tiles_per_block(pairs):
    """Tiles that every CTA has at least (entries_per_warp, TileWalk); from 8 on they come from the queue."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rounds = -(-pairs // (128 * sms))
    per_tile = 16 * -(-pairs // (16 * rounds * sms))
    return -(-pairs // per_tile) // sms


def pairs_by_hand(R, cell, radius, ordered):
    """Sorted entries (i, j, d = R_j - R_i of the nearest image) of a float64 search over all pairs."""
    R64, n = R.double(), len(R)
    c = None if cell is None else torch.tensor(np.asarray(cell, dtype=np.float32), dtype=torch.float64, device=R.device)
    found = []
    for a in range(0, n, 512):
        d = R64[None] - R64[a:a + 512, None]
        if c is not None:
            d -= torch.round(d @ torch.linalg.inv(c)) @ c
        near = (d ** 2).sum(-1) < radius ** 2
        k = torch.arange(a, min(a + 512, n), device=R.device)[:, None], torch.arange(n, device=R.device)[None]
        near &= k[1] > k[0] if ordered else k[1] != k[0]
        i, j = torch.nonzero(near, as_tuple=True)
        found.append((i + a, j, d[i, j]))
    return [torch.cat(x) for x in zip(*found)]


def by_hand(Z, R, cell, cutoff, drop=None):
    """Energy, forces, charges, virial through caller-supplied lists; `drop`: leaves out this short-range entry."""
    from so3lr_b200.engine import System
    i, j, d = pairs_by_hand(R, cell, 4.5, False)
    if drop is not None:
        keep = torch.arange(len(i), device=i.device) != drop(i, j, d)
        i, j, d = i[keep], j[keep], d[keep]
    il, jl, dl = pairs_by_hand(R, cell, cutoff, True)
    s = System(Z, cell, cutoff_lr=cutoff, damping=2.0)
    for _ in range(2):
        o = s.graph_eval(i, j, d, il, jl, dl)
    F, W = torch.zeros(len(Z), 3, dtype=torch.float64, device=R.device), torch.zeros(3, 3, dtype=torch.float64, device=R.device)
    for a, b, x, g in ((i, j, d, o["g_edges"].double()), (il, jl, dl, o["g_edges_lr"].double())):
        F.index_add_(0, a, g)
        F.index_add_(0, b, -g)
        W += x.T @ g
    return [x.double().cpu().numpy() for x in (o["e_atom"].double().sum(), F, o["partial_charges"], 0.5 * (W + W.T))] + [s]


def same(got, want):
    """Virial: sums over all pairs that cancel to a fraction of their terms, 2e-4 of the largest component."""
    (E0, F0, q0, W0), (E1, F1, q1, W1) = got, want
    assert abs(E0.sum() - E1.sum()) <= 2e-6 * abs(E1.sum())
    assert np.abs(F0 - F1).max() <= 5e-5 and np.abs(q0 - q1).max() <= 1e-5
    assert np.abs(W0 - W1).max() <= 2e-4 * np.abs(W1).max()


def evaluate(s, R):
    o = s.compute(R)
    return [o[k].double().cpu().numpy() for k in ("energy", "forces", "partial_charges", "virial")]


def test_tiles_from_the_queue(tmp_path):
    def run(name, env):
        e = {k: v for k, v in os.environ.items() if k != "SO3LR_B200_ATTENTION"}
        subprocess.run([sys.executable, "-c", CHILD, ROOT, str(tmp_path / name)], check=True, timeout=600, env={**e, **env})
        return [np.load(tmp_path / f"{name}.{k}.npz") for k in range(5)]
    for a, b in zip(run("default", {}), run("mma", {"SO3LR_B200_ATTENTION": "mma"})):
        assert abs(float(a["E"]) - float(b["E"])) <= 2e-6 * abs(float(b["E"])), int(a["pairs"])
        assert np.abs(a["F"] - b["F"]).max() <= 5e-5, (int(a["pairs"]), np.abs(a["F"] - b["F"]).max())


def _box(n, seed):
    from so3lr_b200 import workloads as W
    Z, R, cell = W.water_box(n, (n / DENSITY) ** (1 / 3), seed)
    return Z, torch.tensor(np.asarray(R, dtype=np.float32), device="cuda"), cell


@pytest.mark.parametrize("tiles,unpaired", [(7.6, False), (8.3, False), (9.4, False), (4.4, True)])
def test_tiles_of_caller_supplied_lists(tiles, unpaired):
    """On either side of the queue's line, with the virial.  `unpaired`: one entry at the cutoff, where it weighs nothing, without its partner: the
    forward kernel walks every entry, twice as many tiles, the tiled reverse kernel returns at its gate."""
    from so3lr_b200.engine import System
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    Z, R, cell = _box(int(tiles * sms * 128 / 20.03 / 3), 120)
    s = System(Z, cell, cutoff_lr=6.0, damping=2.0)
    s.enable_virial(True)
    evaluate(s, R)
    want = evaluate(s, R)
    *got, g = by_hand(Z, R, cell, 6.0, (lambda i, j, d: (d ** 2).sum(-1).argmax()) if unpaired else None)
    pairs = s.valid_edges() // 2
    assert g.valid_edges() // 2 == pairs or unpaired
    assert (tiles_per_block(2 * pairs - 1 if unpaired else pairs) >= 8) == (tiles > 8 or unpaired)
    same(got, want)


@pytest.mark.parametrize("molecules", [1, 9, 64, 130, 270, 512, 790, 1600])
def test_rows_shared_by_warps_and_queued_pairs(molecules):
    """Several warps a row down to one, against one warp a row over lists from elsewhere.  Lists with a skin queue the pairs inside the cutoff,
    lists without do not."""
    from so3lr_b200.engine import System
    cutoff = min(12.0, 0.49 * (molecules / DENSITY) ** (1 / 3)) if molecules < 64 else 12.0
    Z, R, cell = _box(molecules, 70 + molecules)
    if molecules < 64:
        cell, cutoff = None, 12.0
    *want, _ = by_hand(Z, R, cell, cutoff)
    for skin in (0.0, 1.0):
        s = System(Z, cell, cutoff_lr=cutoff, damping=2.0, skin=skin)
        s.enable_virial(True)
        same(evaluate(s, R), want)


@pytest.mark.parametrize("molecules,form,cutoff", [(3, "free", 9.0), (64, "box", 9.0), (300, "free", 9.0), (512, "box", 9.0), (2048, "box", 9.0),
                                                   (11000, "box", 9.0), (1200, "box", 12.0), (2048, "box", 12.0), (2048, "sheared", 12.0),
                                                   (4100, "long", 12.0)])
def test_lists_built_for_an_evaluation(molecules, form, cutoff):
    """Both lists of an evaluation, whose row kernels may overlap: the numbers of entries against each list exported alone, exactly, and what was
    written into them by evaluating it, against the lists of a search over all pairs; in two positions of the cells."""
    from so3lr_b200.engine import System
    Z, R, cell = _box(molecules if form != "long" else molecules // 4, 90)
    if form == "free":
        cell = None
    elif form == "sheared":      # the same lattice from other vectors
        cell = np.array([[1.0, 0, 0], [1.0, 1.0, 0], [0, 0, 1.0]]) @ np.asarray(cell, dtype=np.float64)
    elif form == "long":         # four boxes in a row
        step = torch.tensor([float(cell[0][0]), 0.0, 0.0], device="cuda")
        Z, R = np.tile(Z, 4), torch.cat([R + k * step for k in range(4)])
        cell = np.asarray(cell, dtype=np.float64) * np.array([[4.0], [1.0], [1.0]])
    s = System(Z, cell, cutoff_lr=cutoff, damping=2.0)
    s.enable_virial(True)
    alone = System(Z, cell, cutoff_lr=cutoff, damping=2.0)
    for shift in (0.0, 3.37):
        got = evaluate(s, R + shift)
        both = s.stats()
        for which, key in ((0, "edges"), (1, "pairs")):
            _, count, overflow = alone.neighbor_list(R + shift, which, both[key] + 8)
            assert count == both[key] and not overflow, (which, count, both[key])
        *want, _ = by_hand(Z, R + shift, cell, cutoff)
        same(got, want)


def test_chain_of_four():
    """The lengths that the chain kernel keeps in registers: this one is not among those of the other tests."""
    from test_gpu_md import test_chain_kernel_matches_oracle as check
    check(4, 2, 3)
