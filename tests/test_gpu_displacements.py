"""Displacements of caller-supplied lists and their transpose (csrc/displacements.cu) against the same gathers in float64 torch.

Tolerances: a displacement is one subtraction and one lattice translation of numbers up to max|R| + 2 |cell|, so it is off by a few
units in the last place of that; a transposed sum of m float32 terms by at most m ulp of the largest partial sum."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,entries,grouped,cell", [(1, 0, True, None), (2, 1, True, "cube"), (7, 31, True, None), (40, 33, False, "skew"),
                                                    (97, 256, True, "skew"), (513, 70001, True, "cube"), (300, 40000, False, None)])
def test_displacements_and_transpose(n, entries, grouped, cell, dtype):
    from so3lr_b200.engine import displacements, displacements_vjp, lists_unsorted
    rng = np.random.default_rng(n + entries)
    h = {None: None, "cube": np.eye(3) * 11.0, "skew": np.array([[11.0, 0.0, 0.0], [2.0, 9.0, 0.0], [-1.5, 3.0, 12.0]])}[cell]
    R = torch.tensor(rng.normal(size=(n, 3)) * 8.0, dtype=dtype, device="cuda")
    i, j = rng.integers(0, n + 1, entries), rng.integers(0, n + 1, entries)      # index n = padding
    if grouped:
        i = np.sort(i)
    ti, tj = (torch.tensor(a, dtype=torch.int32, device="cuda") for a in (i, j))
    ct = None if h is None else torch.tensor(h, dtype=dtype, device="cuda")
    d = displacements(R, ct, ti, tj, dtype)
    R64 = R.double().cpu().numpy()
    ci, cj = np.minimum(i, n - 1), np.minimum(j, n - 1)
    ref = R64[cj] - R64[ci]
    if h is not None:
        s = ref @ np.linalg.inv(h)
        keep = np.abs(np.abs(s - np.round(s)) - 0.5).min(1, initial=1.0) > 1e-5      # no tie of the minimum image
        ref = ref - np.round(s) @ h
    else:
        keep = np.ones(entries, bool)
    eps = torch.finfo(dtype).eps
    scale = float(R.abs().max()) * 2 + (0 if h is None else 6 * np.abs(h).max())
    np.testing.assert_allclose(d.double().cpu().numpy()[keep], ref[keep], atol=4 * eps * scale)
    assert float(d[torch.tensor((ci == cj), device="cuda")].abs().sum()) == 0.0
    g = rng.normal(size=(entries, 3)) * (rng.random((entries, 1)) < 0.7)              # zeros are skipped
    tg = torch.tensor(g, dtype=dtype, device="cuda")
    g64 = tg.double().cpu().numpy()
    out = displacements_vjp(n, dtype, R.device, [(ti, tj, tg), (tj, ti, tg * 0.5)], sign=-2.0)
    want = np.zeros((n, 3))
    for a, sg in ((cj, -2.0), (ci, 2.0)):
        np.add.at(want, a, sg * g64 - 0.5 * sg * g64)
    terms = 4 * max(1, np.bincount(np.concatenate([ci, cj]), minlength=n).max())
    np.testing.assert_allclose(out.double().cpu().numpy(), want, atol=terms * eps * 2.0 * max(1.0, np.abs(g).max(initial=0.0)) * np.sqrt(terms))
    assert lists_unsorted(ti, tj) == (bool((np.diff(i) < 0).any()), bool((np.diff(j) < 0).any()))


def test_negative_indices_count_from_the_end():
    """As in the gathers of torch (and of JAX): -1 is the last atom.  Below -n there is no atom: clamped to the first."""
    from so3lr_b200.engine import displacements, displacements_vjp
    R = torch.randn(6, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    i, j = (torch.tensor(a, dtype=torch.int32, device="cuda") for a in ([0, 1, 2, -1, -6, 3, 6], [-1, -2, -6, 4, 5, -99, -3]))
    ci, cj = (torch.tensor(a, device="cuda") for a in ([0, 1, 2, 5, 0, 3, 5], [5, 4, 0, 4, 5, 0, 3]))
    assert torch.equal(displacements(R, None, i, j), R[cj] - R[ci])
    g = torch.randn(7, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    want = torch.zeros(6, 3, device="cuda").index_add(0, cj, g).index_add(0, ci, -g)
    assert torch.allclose(displacements_vjp(6, torch.float32, R.device, [(i, j, g)]), want, atol=2e-6)      # at most 4 terms of size 3
