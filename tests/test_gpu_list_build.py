"""Neighbor lists of the cell builder (csrc/nlist.cu) against a float64 search over all pairs: boxes of 1, 3, 4 and more cells per axis,
orthorhombic (cells beyond the radius are left out) and skew, atoms far outside the box, counts around a warp's width.  Pairs
within 1e-4 A of the radius may fall on either side."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,edge,skew,spread", [(2, 14.0, 0.0, 0), (33, 13.0, 0.0, 0), (600, 16.6, 0.0, 0), (600, 16.6, 0.0, 3), (700, 23.0, 0.0, 0),
                                                (700, 23.0, 3.0, 2), (1500, (14.1, 31.0, 20.5), 0.0, 2), (2600, 38.0, 0.0, 1), (2600, 38.0, 5.0, 0)])
@pytest.mark.parametrize("ordered", [False, True])
def test_rows_are_exact(n, edge, skew, spread, ordered):
    from so3lr_b200.engine import System
    rng = np.random.default_rng(n)
    L = np.broadcast_to(np.asarray(edge, float), 3)
    cell = np.diag(L).astype(np.float32).astype(np.float64)
    cell[1, 0], cell[2, 1] = skew, -skew
    f = rng.random((n, 3))
    f[: n // 4] = np.round(f[: n // 4] * 4) / 4 + rng.normal(scale=1e-6, size=(n // 4, 3))      # on the borders of cells
    R = ((f + rng.integers(-spread, spread + 1, (n, 3))) @ cell).astype(np.float32)
    s = System(np.full(n, 8), cell, cutoff_lr=6.0, damping=2.0, lr_format="ordered_sparse" if ordered else "sparse")
    Rt = torch.tensor(R, device="cuda")
    for which, rc in ((0, 4.5), (1, 6.0)):
        _, count, _ = s.neighbor_list(Rt, which, 1)
        idx, count, over = s.neighbor_list(Rt, which, max(int(count), 1))
        i, j = idx[:, : int(count)].cpu().numpy().astype(np.int64)
        d = R[None].astype(np.float64) - R[:, None]
        d -= np.round(d @ np.linalg.inv(cell)) @ cell
        r = np.sqrt((d ** 2).sum(-1))
        np.fill_diagonal(r, 1e9)
        if which == 1 and ordered:
            r[np.tril_indices(n)] = 1e9
        got = np.zeros((n, n), dtype=np.int64)
        np.add.at(got, (i, j), 1)
        assert got.max(initial=0) <= 1 and (np.diff(i) >= 0).all()
        sure, never = r < rc - 1e-4, r > rc + 1e-4
        assert got[sure].all() and not got[never].any()


@pytest.mark.parametrize("n", [1, 2, 31, 255, 257, 1024, 1025])
def test_free_space_lists_of_an_evaluation(n):
    """Below and above the size up to which all atoms of a free-space structure are candidates: the list sizes of an evaluation equal those
    of a search over all pairs, and an infinite position is refused."""
    from so3lr_b200.engine import System
    rng = np.random.default_rng(n)
    g = np.stack(np.meshgrid(*[np.arange(11)] * 3), -1).reshape(-1, 3)[:n] * 1.9
    R = (g + rng.normal(scale=0.1, size=g.shape)).astype(np.float32)
    s = System(np.full(n, 8), None, cutoff_lr=6.0, damping=2.0)
    Rt = torch.tensor(R, device="cuda")
    o = s.compute(Rt)
    torch.cuda.synchronize()
    r = np.linalg.norm(R[None].astype(np.float64) - R[:, None], axis=-1)
    np.fill_diagonal(r, 1e9)
    st = s.stats()
    near = lambda rc: ((r < rc - 1e-4).sum(), (r < rc + 1e-4).sum())
    lo, hi = near(4.5)
    assert lo <= st["edges"] <= hi
    lo, hi = near(6.0)
    assert lo <= 2 * st["pairs"] <= hi or lo <= st["pairs"] <= hi
    assert torch.isfinite(o["forces"]).all()
    for bad in (float("inf"), -float("inf")):
        Rb = Rt.clone()
        Rb[n - 1, 2] = bad
        with pytest.raises(Exception):
            s.compute(Rb)
    o2 = s.compute(Rt)
    assert float((o2["forces"] - o["forces"]).abs().max()) <= 1e-4 * max(1.0, float(o["forces"].abs().max()))


@pytest.mark.parametrize("n,atoms", [(n, a) for n in (1, 2, 31, 1024) for a in ("all", "one")] + [(1025, "all")])
@pytest.mark.parametrize("skin", [0.0, 1.0])
def test_positions_that_are_no_numbers_are_refused(n, atoms, skin):
    """A structure that has blown up has no neighbours and no forces: it must not come back as a converged one.  Above 1,024 atoms the
    bounding box decides, which looks for a finite extent: NaN along a whole axis."""
    from so3lr_b200.engine import System
    R = (np.arange(3 * n).reshape(n, 3) * 0.37 % 19.0).astype(np.float32)
    Rb = R.copy()
    Rb[slice(None) if atoms == "all" else n // 2, :] = np.nan
    s = System(np.full(n, 8), None, cutoff_lr=6.0, damping=2.0, skin=skin)
    with pytest.raises(Exception):
        s.compute_host(Rb)
    assert np.isfinite(s.compute_host(R + np.arange(n)[:, None].astype(np.float32))["energy"]).all()
