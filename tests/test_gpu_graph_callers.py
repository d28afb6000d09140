"""What the graph-level callers (So3lr, the jax-md adapter) refuse, accept and differentiate around the displacement kernels
(csrc/displacements.cu)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _water(n=64):
    from so3lr_b200 import workloads as W
    Z, R, cell = W.water_box(n, (n * 29.9) ** (1 / 3), 3)
    return Z, np.asarray(R, np.float32), np.asarray(cell, np.float32)


def _inputs(Z, R, cell):
    from oracle import so3lr_oracle as O
    i, j = O.neighbor_list(R.astype(np.float64), cell.astype(np.float64), 4.5, ordered=False)
    il, jl = O.neighbor_list(R.astype(np.float64), cell.astype(np.float64), 6.0, ordered=False)
    return dict(positions=R, atomic_numbers=Z, idx_i=i, idx_j=j, idx_i_lr=il, idx_j_lr=jl, cell=cell)


_SINGULAR = {"zero_edge": np.diag([10.0, 10.0, 0.0]), "two_equal_vectors": np.array([[10.0, 0, 0], [10.0, 0, 0], [0, 0, 10.0]]),
             "in_a_plane": np.array([[1.0, 2, 3], [4, 5, 6], [7, 8, 9]]), "not_finite": np.diag([10.0, 10.0, np.inf])}


@pytest.mark.parametrize("name", list(_SINGULAR))
@pytest.mark.parametrize("where", ["cpu", "cuda"])
def test_singular_cells_are_refused(name, where):
    """Every entry's displacement would be NaN and drop out: the energy of isolated atoms without an error."""
    from so3lr_b200 import So3lr, So3lrPotential, to_jax_md
    Z, R, cell = _water()
    inputs = _inputs(Z, R, cell)
    bad = torch.tensor(_SINGULAR[name], dtype=torch.float32, device=where)
    fn = So3lr(lr_cutoff=6.0)
    with pytest.raises(torch.linalg.LinAlgError):
        fn({**inputs, "cell": bad})
    assert np.isfinite(float(fn(inputs)["energy"]))
    _, _, energy_fn = to_jax_md(So3lrPotential(lr_cutoff=6.0), None, None, species=Z, fractional_coordinates=False)
    nb = [torch.tensor(np.stack([inputs[a], inputs[b]]), device="cuda") for a, b in (("idx_i", "idx_j"), ("idx_i_lr", "idx_j_lr"))]
    Rt = torch.tensor(R, device="cuda")
    boxes = [bad.T] if name != "zero_edge" else [bad, torch.diagonal(bad)]
    for box in boxes:
        with pytest.raises(torch.linalg.LinAlgError):
            energy_fn(Rt, *nb, box=box)
    assert np.isfinite(float(energy_fn(Rt, *nb, box=torch.diagonal(torch.tensor(cell, device=where)))))


@pytest.mark.parametrize("shape", [(3,), (1,), (2, 3), (9,)])
def test_cells_that_are_no_matrix_are_refused(shape):
    from so3lr_b200 import So3lr
    Z, R, cell = _water()
    with pytest.raises((ValueError, RuntimeError)):
        So3lr(lr_cutoff=6.0)({**_inputs(Z, R, cell), "cell": np.full(shape, 12.0, np.float32)})


@pytest.mark.parametrize("key", ["idx_i", "idx_j", "idx_i_lr", "idx_j_lr"])
@pytest.mark.parametrize("order", ["sorted", "shuffled"])
def test_lists_of_unequal_length_are_refused(key, order):
    """The kernels take one length per list; a shorter partner array would be read past its end."""
    from so3lr_b200 import Graph, So3lr, So3lrPotential
    Z, R, cell = _water()
    inputs = _inputs(Z, R, cell)
    if order == "shuffled":
        for a, b in (("idx_i", "idx_j"), ("idx_i_lr", "idx_j_lr")):
            p = np.random.default_rng(0).permutation(len(inputs[a]))
            inputs[a], inputs[b] = inputs[a][p], inputs[b][p]
    short = {**inputs, key: inputs[key][:-3]}
    with pytest.raises((ValueError, RuntimeError)):
        So3lr(lr_cutoff=6.0)(short)
    t = {k: torch.tensor(short[k], device="cuda") for k in ("idx_i", "idx_j", "idx_i_lr", "idx_j_lr")}
    d, dl = (torch.ones(len(inputs[k]), 3, device="cuda") for k in ("idx_i", "idx_i_lr"))
    g = Graph(None, d, torch.tensor(Z), t["idx_i"], t["idx_j"], None, None, None, dl, t["idx_i_lr"], t["idx_j_lr"], None)
    with pytest.raises((ValueError, RuntimeError)):
        So3lrPotential(lr_cutoff=6.0)(g)


def test_arrays_the_kernels_cannot_read_are_refused():
    from so3lr_b200.engine import displacements, displacements_vjp, lists_unsorted
    R = torch.zeros(5, 3, device="cuda")
    i = torch.arange(4, dtype=torch.int32, device="cuda")
    g = torch.zeros(4, 3, device="cuda")
    for a in (i[:3], i.long(), i.cpu(), i.reshape(2, 2)):
        for pair in ((i, a), (a, i)):
            with pytest.raises(ValueError):
                displacements(R, None, *pair)
            with pytest.raises(ValueError):
                displacements_vjp(5, torch.float32, R.device, [(*pair, g)])
    for bad in (R.half(), R.cpu(), R.reshape(-1), torch.zeros(5, 4, device="cuda")):
        with pytest.raises(ValueError):
            displacements(bad, None, i, i)
    for bad in (g[:3], g.half(), g.double(), g.cpu(), g.reshape(-1)):
        with pytest.raises(ValueError):
            displacements_vjp(5, torch.float32, R.device, [(i, i, bad)])
    with pytest.raises(ValueError):
        displacements(R, torch.ones(3, device="cuda"), i, i)
    with pytest.raises(ValueError):
        lists_unsorted(i, i.long())
    # strided arrays are taken as what they show
    R2, i2, g2 = torch.randn(5, 6, device="cuda")[:, ::2], torch.arange(8, dtype=torch.int32, device="cuda")[::2] % 5, torch.randn(3, 4, device="cuda").T
    ref = R2[i2.long()] - R2[i.long()]
    assert torch.equal(displacements(R2, None, i, i2), ref)
    want = torch.zeros(5, 3, device="cuda").index_add(0, i2.long(), g2).index_add(0, i.long(), -g2)
    assert torch.allclose(displacements_vjp(5, torch.float32, R.device, [(i, i2, g2)]), want, atol=1e-6)


@pytest.mark.parametrize("where", ["cpu", "cuda"])
def test_shuffled_lists_of_a_graph_on_either_side(where):
    """A Graph whose arrays are on the host, in any order and integer type: same energies and (reordered) gradients as grouped lists."""
    from so3lr_b200 import Graph, So3lrPotential
    Z, R, cell = _water()
    inp = _inputs(Z, R, cell)
    p, q = (np.random.default_rng(k).permutation(len(inp[a])) for k, a in enumerate(("idx_i", "idx_i_lr")))
    c = cell.astype(np.float64)
    mi = lambda d: d - np.round(d @ np.linalg.inv(c)) @ c
    d, dl = mi(R[inp["idx_j"]] - R[inp["idx_i"]].astype(np.float64)), mi(R[inp["idx_j_lr"]] - R[inp["idx_i_lr"]].astype(np.float64))
    pot = So3lrPotential(lr_cutoff=6.0)

    def energies(o, ol, dev):
        e, el = (torch.tensor(a, dtype=torch.float32, device=dev, requires_grad=True) for a in (d[o], dl[ol]))
        i, j, il, jl = (torch.tensor(inp[k][s], device=dev) for k, s in (("idx_i", o), ("idx_j", o), ("idx_i_lr", ol), ("idx_j_lr", ol)))
        E = pot(Graph(None, e, torch.tensor(Z), i, j, None, None, None, el, il, jl, None))
        return E.detach().cpu(), *(g.cpu() for g in torch.autograd.grad(E.sum(), (e, el)))

    ref = energies(np.arange(len(d)), np.arange(len(dl)), "cuda")
    got = energies(p, q, where)
    assert float((got[0] - ref[0]).abs().max()) <= 1e-5 * float(ref[0].abs().max())
    assert float((got[1] - ref[1][torch.tensor(p)]).abs().max()) <= 1e-4 and float((got[2] - ref[2][torch.tensor(q)]).abs().max()) <= 1e-5


@pytest.mark.parametrize("order", ["columns", "every_second"])
def test_strided_positions_are_read_as_what_they_show(order):
    from so3lr_b200 import So3lr
    Z, R, cell = _water()
    inputs = _inputs(Z, R, cell)
    Rt = torch.tensor(R, device="cuda")
    strided = Rt.T.contiguous().T if order == "columns" else torch.stack([Rt, Rt + 7.0], -1)[..., 0]
    assert not strided.is_contiguous()
    fn = So3lr(lr_cutoff=6.0)
    ref, got = fn({**inputs, "positions": Rt}), fn({**inputs, "positions": strided})
    assert abs(float(got["energy"] - ref["energy"])) <= 2e-6 * abs(float(ref["energy"]))
    assert float((got["forces"] - ref["forces"]).abs().max()) <= 5e-5


def test_gradients_belong_to_the_caller():
    """Gradients with respect to a graph's edges may be changed in place between two backward passes."""
    from so3lr_b200 import Graph, So3lrPotential
    Z, R, cell = _water()
    inp = _inputs(Z, R, cell)
    t = {k: torch.tensor(inp[k], device="cuda") for k in ("idx_i", "idx_j", "idx_i_lr", "idx_j_lr")}
    c = cell.astype(np.float64)
    mi = lambda d: torch.tensor(d - np.round(d @ np.linalg.inv(c)) @ c, dtype=torch.float32, device="cuda").requires_grad_(True)
    d, dl = mi(R[inp["idx_j"]] - R[inp["idx_i"]].astype(np.float64)), mi(R[inp["idx_j_lr"]] - R[inp["idx_i_lr"]].astype(np.float64))
    E = So3lrPotential(lr_cutoff=6.0)(Graph(None, d, torch.tensor(Z), t["idx_i"], t["idx_j"], None, None, None, dl, t["idx_i_lr"], t["idx_j_lr"], None)).sum()
    first = torch.autograd.grad(E, (d, dl), retain_graph=True)
    ref = [g.clone() for g in first]
    for g in first:
        g.mul_(-3.0)
    again = torch.autograd.grad(E, (d, dl), retain_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(again, ref))
    # a factor in front of the sum: the gradient's own dependence on it is not available, and that is said
    w = torch.tensor(2.5, device="cuda", requires_grad=True)
    g, = torch.autograd.grad(w * E, d, create_graph=True)
    assert torch.allclose(g.detach(), 2.5 * ref[0])
    with pytest.raises(RuntimeError):
        torch.autograd.grad(g.sum(), w)
