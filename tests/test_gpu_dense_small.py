"""The per-atom blocks of short lists (csrc/atom_kernels_small.cu) against the tensor-core blocks (SO3LR_B200_DENSE=tc, read once per process)
at list lengths around every change of the tile size, through energies, charges and forces of separate water clusters.

Both evaluate the same FP32 formulas in another order of summation: tolerances of the variant tests, 2e-6 relative and 5e-5 eV/A."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import sys, numpy as np, torch
sys.path.insert(0, sys.argv[1])
from so3lr_b200 import workloads as W
from so3lr_b200.engine import System
sms = torch.cuda.get_device_properties(0).multi_processor_count
Z, R, _ = W.water_box(3000, (3000 * 29.9) ** (1 / 3), 3)
o = np.argsort(np.repeat(R[::3, 2], 3), kind="stable")      # whole molecules along z: a prefix is a connected slab
Z, R = Z[o], np.asarray(R[o], dtype=np.float32)
out = {}
sizes = [1, 2, 3, 5, 31] + [k * sms + d for k in (2, 4, 6, 8, 10, 12, 16) for d in (0, 1)]
for n in sizes:
    s = System(Z[:n], None, cutoff_lr=8.0, damping=2.0)
    r = s.compute(torch.tensor(R[:n], device="cuda"))
    out[f"E{n}"] = r["energy"].double().cpu().numpy().sum()
    out[f"F{n}"] = r["forces"].cpu().numpy()
    out[f"q{n}"] = r["partial_charges"].cpu().numpy()
    out[f"h{n}"] = r["hirshfeld_ratios"].cpu().numpy()
np.savez(sys.argv[2], sizes=np.array(sizes), **out)
"""


def test_short_lists_agree_with_the_tensor_core_blocks(tmp_path):
    def run(name, env):
        out = str(tmp_path / f"{name}.npz")
        e = {k: v for k, v in os.environ.items() if k != "SO3LR_B200_DENSE"}
        subprocess.run([sys.executable, "-c", CHILD, ROOT, out], check=True, timeout=600, env={**e, **env})
        return np.load(out)
    a, b = run("default", {}), run("tc", {"SO3LR_B200_DENSE": "tc"})
    for n in a["sizes"]:
        assert abs(a[f"E{n}"] - b[f"E{n}"]) <= 2e-6 * abs(b[f"E{n}"]), n
        assert np.isfinite(a[f"F{n}"]).all()
        assert np.abs(a[f"F{n}"] - b[f"F{n}"]).max() <= 5e-5, (n, np.abs(a[f"F{n}"] - b[f"F{n}"]).max())
        assert np.abs(a[f"q{n}"] - b[f"q{n}"]).max() <= 1e-5 and np.abs(a[f"h{n}"] - b[f"h{n}"]).max() <= 1e-5, n
