"""Short-range attention on one entry per undirected pair (csrc/attention_tc.cu): caller-supplied lists of every form that decides how the
entries pair up, and pair counts around the edges of a warp's share and of a tile, against the float64 oracle on the same lists.

Tolerances are those of the parity tests: energies 1e-5 relative, gradients 1e-4 eV/A; with every entry two times in the list every pair
term and its rounding error count twice: 2e-4 eV/A."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _structure(name):
    from so3lr_b200 import workloads as W
    if name.startswith("water"):
        n = int(name[5:])
        return W.water_box(n, (n * 29.9) ** (1 / 3), 3)
    Z, R = W.molecule(np.random.default_rng(7), int(name[3:]))
    return Z, R, None


def _lists(name, form):
    from oracle import so3lr_oracle as O
    Z, R, cell = _structure(name)
    R = np.asarray(R, np.float32).astype(np.float64)
    cell = None if cell is None else np.asarray(cell, np.float32).astype(np.float64)
    i, j = O.neighbor_list(R, cell, 4.5, ordered=False)
    il, jl = O.neighbor_list(R, cell, 6.0 if cell is not None else 100.0, ordered=False)
    mi = lambda d: d if cell is None else d - np.round(d @ np.linalg.inv(cell)) @ cell
    d, dl = mi(R[j] - R[i]), mi(R[jl] - R[il])
    if form == "twice":                       # every entry two times: still paired
        i, j, d = np.repeat(i, 2), np.repeat(j, 2), np.repeat(d, 2, axis=0)
    elif form == "twice_one_way":             # one entry two times, its partner once
        k = len(i) // 3
        i, j, d = (np.insert(a, k, a[k], axis=0) for a in (i, j, d))
    elif form == "one_way":                   # no entry has a partner
        m = j > i
        i, j, d = i[m], j[m], d[m]
    elif form == "images":                    # an atom beside its own periodic images
        i, j = np.append(i, [0, 0, 1, 1]), np.append(j, [0, 0, 1, 1])
        d = np.concatenate([d, [[0.0, 0.0, 4.1], [0.0, 0.0, -4.1], [-4.2, 0.3, 0.0], [4.2, -0.3, 0.0]]])
        o = np.argsort(i, kind="stable")
        i, j, d = i[o], j[o], d[o]
    elif form == "padded":                    # entries beyond the cutoff and a tail of padding
        m = len(Z)
        far = np.nonzero(i == m - 1)[0][:1]
        i, j, d = np.append(np.append(i, i[far]), [m] * 5), np.append(np.append(j, j[far]), [m] * 5), np.concatenate([d, d[far] * 9.0, np.zeros((5, 3))])
    return Z, cell, (i, j, d.astype(np.float32)), (il, jl, dl.astype(np.float32))


@pytest.mark.parametrize("name,form", [(n, "plain") for n in ("mol8", "mol11", "mol23", "mol40", "water64", "water192")] +
                         [("mol23", f) for f in ("twice", "twice_one_way", "one_way", "images", "padded")] + [("water64", f) for f in ("twice", "one_way")])
def test_list_forms_against_the_oracle(name, form):
    from oracle import so3lr_oracle as O
    from so3lr_b200.engine import System
    Z, cell, (i, j, d), (il, jl, dl) = _lists(name, form)
    n = len(Z)
    s = System(Z, cell, cutoff_lr=6.0 if cell is not None else 100.0, damping=2.0, lr_format="sparse")
    t = lambda a: torch.tensor(a, device="cuda")
    # the first evaluation of a context forms the first layer's tables
    results = [s.graph_eval(t(i), t(j), t(d), t(il), t(jl), t(dl)) for _ in range(2)]
    D, DL = torch.tensor(d, dtype=torch.float64, requires_grad=True), torch.tensor(dl, dtype=torch.float64, requires_grad=True)
    e, _ = O.energy_from_graph(O.load_params(), Z, D, i, j, DL, il, jl, lr_format="sparse", cutoff_lr=6.0 if cell is not None else 100.0, damping=2.0)
    g, = torch.autograd.grad(e.sum(), D)
    e = e.detach()
    for o in results:
        _check(o, e, g, i, j, D.detach(), n, form)


@pytest.mark.parametrize("name,rounds", [("water300", 1), ("water600", 2), ("water900", 3)])
def test_full_tiles_against_the_oracle(name, rounds):
    """Tiles of 128 pairs, what every long list runs: 16 warps with a share of 8 pairs each, in one round over the SMs and in several.  The
    lists above have shares of 1 to 5 (16 n pairs fill the share of n on every SM).  2,700 atoms take the tensor-core dense blocks."""
    from oracle import so3lr_oracle as O
    from so3lr_b200.engine import System
    Z, cell, (i, j, d), (il, jl, dl) = _lists(name, "plain")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = len(i) // 2
    assert -(-pairs // (128 * sms)) == rounds and -(-pairs // (16 * sms * rounds)) == 8
    s = System(Z, cell, cutoff_lr=6.0, damping=2.0, lr_format="sparse")
    t = lambda a: torch.tensor(a, device="cuda")
    o = s.graph_eval(t(i), t(j), t(d), t(il), t(jl), t(dl))
    D, DL = torch.tensor(d, dtype=torch.float64, requires_grad=True), torch.tensor(dl, dtype=torch.float64)
    e, _ = O.energy_from_graph(O.load_params(), Z, D, i, j, DL, il, jl, lr_format="sparse", cutoff_lr=6.0, damping=2.0)
    g, = torch.autograd.grad(e.sum(), D)
    _check(o, e.detach(), g, i, j, D.detach(), len(Z), "plain")


def _check(o, e, g, i, j, D, n, form):
    got = o["g_edges"].double().cpu()
    assert float((o["e_atom"].double().cpu() - e).abs().sum()) <= 1e-5 * float(e.abs().sum())
    if form in ("one_way", "twice_one_way"):      # lists without partners: the gradient of every entry
        assert float((got - g).abs().max()) <= 1e-4
        return
    # paired lists: what any motion of atoms or cell sees of it
    m = torch.tensor(i < n)
    ti, tj = torch.tensor(i)[m], torch.tensor(j)[m]
    f = lambda x: torch.zeros(n, 3, dtype=torch.float64).index_add(0, ti, x[m]).index_add(0, tj, -x[m])
    assert float((f(got) - f(g)).abs().max()) <= (2e-4 if form == "twice" else 1e-4)
    w, wr = D.T @ got, D.T @ g
    assert float((w - wr).abs().max()) <= 1e-4 * max(1.0, float(wr.abs().max()))
    assert float(got[~m].abs().sum()) == 0.0


def test_more_elements_than_the_tables_hold():
    """Nine elements: every evaluation of the context runs the generic first layer."""
    from oracle import so3lr_oracle as O
    from so3lr_b200.engine import System
    Z, _, (i, j, d), (il, jl, dl) = _lists("mol40", "plain")
    Z = np.array(Z)
    heavy = np.nonzero(Z > 1)[0][:8]
    Z[heavy] = [5, 6, 7, 8, 9, 15, 16, 17]
    assert len(set(Z.tolist())) == 9
    s = System(Z, None, cutoff_lr=100.0, damping=2.0, lr_format="sparse")
    t = lambda a: torch.tensor(a, device="cuda")
    D, DL = torch.tensor(d, dtype=torch.float64, requires_grad=True), torch.tensor(dl, dtype=torch.float64)
    e, _ = O.energy_from_graph(O.load_params(), Z, D, i, j, DL, il, jl, lr_format="sparse", cutoff_lr=100.0, damping=2.0)
    g, = torch.autograd.grad(e.sum(), D)
    for _ in range(2):
        o = s.graph_eval(t(i), t(j), t(d), t(il), t(jl), t(dl))
        # elements were exchanged under the same positions: strained bonds with forces far above 20 eV/A, so relative to the largest
        scale = max(1.0, float(g.abs().max()) / 20.0)
        assert float((o["e_atom"].double().cpu() - e.detach()).abs().sum()) <= 1e-5 * float(e.detach().abs().sum())
        f = lambda x: torch.zeros(len(Z), 3, dtype=torch.float64).index_add(0, torch.tensor(i), x).index_add(0, torch.tensor(j), -x)
        assert float((f(o["g_edges"].double().cpu()) - f(g)).abs().max()) <= 1e-4 * scale


@pytest.mark.parametrize("system", ["neutral", "batch"])
def test_evaluations_of_a_context_run_the_same_kernels(system):
    """Two atoms: every sum has one term, so that evaluations of the same inputs agree bit for bit, the context's first one among them, and
    the re-evaluation for another cotangent has the same energies."""
    from so3lr_b200.engine import System
    t = lambda a, **k: torch.tensor(a, device="cuda", **k)
    kw = {"graph_start": [0, 2, 2], "total_charge": [1.0, 0.0]} if system == "batch" else {}
    s = System([8, 1], None, cutoff_lr=100.0, damping=2.0, lr_format="sparse", **kw)
    i, j = t([0, 1], dtype=torch.int32), t([1, 0], dtype=torch.int32)
    d = t([[0.3, -0.8, 0.9], [-0.3, 0.8, -0.9]])
    out = [s.graph_eval(i, j, d, i, j, d, g_e_atom=g) for g in (None, None, t([1.0, 0.5]), None)]
    assert all(torch.equal(o["e_atom"], out[0]["e_atom"]) for o in out)
    assert all(torch.equal(o[k], out[0][k]) for o in (out[1], out[3]) for k in ("g_edges", "g_edges_lr", "partial_charges"))
