"""Sizes at which a rule of a launch changes what a kernel does: tiles handed out by the queue (csrc/attention_tc.cu), rows shared by several
warps and the queue of the pairs inside the cutoff (csrc/pair_kernels.cu), both lists' row kernels side by side (csrc/nlist.cu).

The kernels behind them evaluate the same FP32 formulas in another order of summation: tolerances of the variant tests, 2e-6 relative
and 5e-5 eV/A; lists are compared exactly."""
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
import sys, numpy as np, torch
sys.path.insert(0, sys.argv[1])
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
    assert (first - o["forces"]).abs().max().item() <= 5e-5
    np.savez(f"{sys.argv[2]}.{k}.npz", E=o["energy"].double().cpu().numpy().sum(), F=o["forces"].cpu().numpy(), pairs=s.valid_edges())
"""


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


@pytest.mark.parametrize("molecules", [1, 9, 64, 130, 270, 512, 790, 1600])
def test_rows_shared_by_warps_and_queued_pairs(molecules):
    """Several warps a row down to one.  Lists with a skin queue the pairs inside the cutoff, lists without do not."""
    from so3lr_b200.engine import System
    cutoff = min(12.0, 0.49 * (molecules / DENSITY) ** (1 / 3)) if molecules < 64 else 12.0
    Z, R, cell = _box(molecules, 70 + molecules)
    if molecules < 64:
        cell, cutoff = None, 12.0
    got = []
    for skin in (0.0, 1.0):
        s = System(Z, cell, cutoff_lr=cutoff, damping=2.0, skin=skin)
        s.enable_virial(True)
        o = s.compute(R)
        got.append([o[k].double().cpu().numpy() for k in ("energy", "forces", "partial_charges", "virial")])
    (E0, F0, q0, W0), (E1, F1, q1, W1) = got
    assert abs(E0.sum() - E1.sum()) <= 2e-6 * abs(E0.sum())
    assert np.abs(F0 - F1).max() <= 5e-5 and np.abs(q0 - q1).max() <= 1e-5
    assert np.abs(W0 - W1).max() <= 2e-4 * np.abs(W0).max()


@pytest.mark.parametrize("molecules,form,cutoff", [(3, "free", 9.0), (64, "box", 9.0), (300, "free", 9.0), (512, "box", 9.0), (2048, "box", 9.0),
                                                   (11000, "box", 9.0), (1200, "box", 12.0), (2048, "box", 12.0), (2048, "sheared", 12.0),
                                                   (4100, "long", 12.0)])
def test_lists_built_for_an_evaluation(molecules, form, cutoff):
    """Both lists of an evaluation, whose row kernels may overlap, against each of them exported alone: the numbers of entries exactly, in two
    positions of the cells."""
    from so3lr_b200.engine import System
    Z, R, cell = _box(molecules, 90)
    if form == "free":
        cell = None
    elif form == "sheared":      # a skewed cell of the same volume: another packing, whose overlaps do not matter to a list
        cell = np.asarray(cell, dtype=np.float64) + np.array([[0, 0, 0], [0.3, 0, 0], [-0.2, 0.25, 0]]) * float(cell[0][0])
    elif form == "long":
        cell = np.asarray(cell, dtype=np.float64) * np.array([[2.0], [1.0], [0.8]])
        R = R * torch.tensor([2.0, 1.0, 0.8], device="cuda")
    s = System(Z, cell, cutoff_lr=cutoff, damping=2.0)
    alone = System(Z, cell, cutoff_lr=cutoff, damping=2.0)
    for shift in (0.0, 3.37):
        s.compute(R + shift)
        both = s.stats()
        for which, key in ((0, "edges"), (1, "pairs")):
            _, count, overflow = alone.neighbor_list(R + shift, which, both[key] + 8)
            assert count == both[key] and not overflow, (which, count, both[key])


def test_chain_of_four():
    """The lengths that the chain kernel keeps in registers: this one is not among those of the other tests."""
    from test_gpu_md import test_chain_kernel_matches_oracle as check
    check(4, 2, 3)
