"""Evaluation contexts that receive the blocks of released ones (csrc/devmem.cu): contexts of other sizes, created and released on
several threads, do not disturb the results of a context that reuses their memory."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _energies(Z, R, gs, skin=0.0):
    from so3lr_b200.engine import System
    s = System(Z, None, cutoff_lr=12.0, damping=2.0, lr_format="sparse", graph_start=gs, skin=skin)
    out = s.compute(torch.tensor(R, dtype=torch.float32, device="cuda"))
    return out["energy"].cpu().numpy(), out["forces"].cpu().numpy(), out["partial_charges"].cpu().numpy()


def test_reused_blocks_give_the_same_results():
    from so3lr_b200 import workloads as W
    sets = [W.molecule_batch(m, seed=m) for m in (1, 2, 3, 7, 8, 9)]
    ref = [_energies(Z, R, gs) for Z, R, gs in sets]
    errors = []

    def work(order):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in order:
                    e, f, q = _energies(*sets[k])
                    # the same kernels on the same inputs: only the order of the atomic additions differs
                    np.testing.assert_allclose(e, ref[k][0], rtol=2e-6)
                    np.testing.assert_allclose(f, ref[k][1], atol=5e-5)
                    np.testing.assert_allclose(q, ref[k][2], atol=2e-6)
        except BaseException as err:       # noqa: BLE001 - reported by the main thread
            errors.append(err)

    rng = np.random.default_rng(0)
    threads = [threading.Thread(target=work, args=(rng.integers(0, len(sets), 12),)) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors[0]


@pytest.mark.parametrize("charges", [[1.0, 0.0, 0.0], [0.0, 0.0, -1.0], [2.0, 0.0, 1.0], [1.0, -1.0, 1.0]])
@pytest.mark.parametrize("kind", ["total_charge", "num_unpaired"])
def test_charged_graphs_without_atoms(charges, kind):
    """Three graphs of which the first and the last have no atoms: they have no embedding rows, and a charge of theirs changes nothing."""
    from so3lr_b200 import workloads as W
    from so3lr_b200.engine import System
    Z, R = W.molecule(np.random.default_rng(3), 70)
    R = torch.tensor(R, dtype=torch.float32, device="cuda")
    gs = [0, 0, len(Z), len(Z)]
    make = lambda c: System(Z, None, cutoff_lr=12.0, damping=2.0, lr_format="sparse", graph_start=gs, **{kind: c}).compute(R)
    got, ref = make(charges), make([0.0, charges[1], 0.0])
    assert abs(float(got["energy"][1] - ref["energy"][1])) <= 2e-6 * abs(float(ref["energy"][1]))
    assert float((got["forces"] - ref["forces"]).abs().max()) <= 5e-5
    assert float(got["energy"][0]) == float(got["energy"][2]) == 0.0
