"""Derivatives of the jax-md adapter's displacements (Graph.edges / Graph.edges_lr of neighbor_list_featurizer) for energies that a caller
builds on them: first and second reverse-mode, forward-mode, the torch.func transforms and tracing, against the same gathers in torch.

Positions are float64 and the displacements float32 on both sides; the map is linear, so they agree to rounding of a few terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(seed=0, n=23, entries=(90, 150), cell=True):
    rng = np.random.default_rng(seed)
    t = lambda a, **k: torch.tensor(a, device="cuda", **k)
    R = t(rng.normal(size=(n, 3)) * 5.0)
    nb = [t(np.stack([np.sort(rng.integers(0, n + 1, m)), rng.integers(0, n + 1, m)]).astype(np.int32)) for m in entries]
    box = t(np.array([9.0, 11.0, 10.0])) if cell else None
    from so3lr_b200.api import neighbor_list_featurizer
    fz = neighbor_list_featurizer(None, np.ones(n, int), fractional_coordinates=False)
    ref = lambda R: _reference(R, nb, box)
    return R, (lambda R: fz(R, *nb, box=box)), ref


def _reference(R, nb, box):
    out = []
    for idx in nb:
        i, j = idx.long().clamp(max=R.shape[0] - 1)
        d = R[j] - R[i]
        if box is not None:
            d = d - torch.round((d / box).detach()) * box
        out.append(d.float())
    return out


def _energy(edges, edges_lr):
    """A caller's own energy: not linear in the displacements, finite at zero."""
    r2, r2_lr = (edges.double() ** 2).sum(-1), (edges_lr.double() ** 2).sum(-1)
    return torch.log1p(r2).sum() + 0.1 * torch.exp(-0.05 * r2_lr).sum()


def _both(cell=True):
    R, graph, ref = _setup(cell=cell)
    lib = lambda R: (lambda g: _energy(g.edges, g.edges_lr))(graph(R))
    return R, lib, lambda R: _energy(*ref(R))


def _close(a, b):
    # float32 displacements of up to 20 A on both sides: relative 1e-7 each, some tens of terms per atom
    assert float((a - b).abs().max()) <= 1e-5 * max(1.0, float(b.abs().max())), float((a - b).abs().max())


@pytest.mark.parametrize("cell", [True, False])
def test_second_derivatives(cell):
    R, lib, ref = _both(cell)
    v = torch.randn_like(R)

    def hvp(f):
        x = R.clone().requires_grad_(True)
        g, = torch.autograd.grad(f(x), x, create_graph=True)
        assert g.requires_grad
        return g.detach(), torch.autograd.grad((g * v).sum(), x)[0]

    for a, b in zip(hvp(lib), hvp(ref)):
        _close(a, b)


def test_second_derivative_through_one_list_only():
    R, graph, ref = _setup()
    x, y = (R.clone().requires_grad_(True) for _ in range(2))
    out = []
    for f, z in ((lambda z: graph(z).edges, x), (lambda z: ref(z)[0], y)):
        g, = torch.autograd.grad((f(z).double() ** 3).sum(), z, create_graph=True)
        out.append(torch.autograd.grad((g ** 2).sum(), z)[0])
    _close(*out)


def test_forward_mode():
    import torch.autograd.forward_ad as fwAD
    R, lib, ref = _both()
    v = torch.randn_like(R)

    def jvp(f):
        with fwAD.dual_level():
            return fwAD.unpack_dual(f(fwAD.make_dual(R, v))).tangent

    _close(jvp(lib), jvp(ref))


def test_function_transforms():
    R, lib, ref = _both()
    v = torch.randn_like(R)
    _close(torch.func.grad(lib)(R), torch.func.grad(ref)(R))
    _close(torch.func.jvp(lib, (R,), (v,))[1], torch.func.jvp(ref, (R,), (v,))[1])
    _close(torch.func.jvp(torch.func.grad(lib), (R,), (v,))[1], torch.func.jvp(torch.func.grad(ref), (R,), (v,))[1])
    many = torch.stack([R, R * 1.01, R - 0.3])
    _close(torch.vmap(lib)(many), torch.vmap(ref)(many))
    _close(torch.vmap(torch.func.grad(lib))(many), torch.vmap(torch.func.grad(ref))(many))


def test_derivatives_with_respect_to_the_box():
    from so3lr_b200.api import neighbor_list_featurizer
    R, _, _ = _setup()
    rng = np.random.default_rng(0)
    rng.normal(size=(23, 3))
    nb = [torch.tensor(np.stack([np.sort(rng.integers(0, 24, m)), rng.integers(0, 24, m)]).astype(np.int32), device="cuda") for m in (90, 150)]
    fz = neighbor_list_featurizer(None, np.ones(23, int), fractional_coordinates=False)
    lib = lambda R, box: (lambda g: _energy(g.edges, g.edges_lr))(fz(R, *nb, box=box))
    ref = lambda R, box: _energy(*_reference(R, nb, box))
    box = torch.tensor([9.0, 11.0, 10.0], dtype=torch.float64, device="cuda")
    for f in (torch.func.grad, lambda g, argnums: lambda R, b: torch.func.jvp(lambda x: g(R, x), (b,), (torch.ones_like(b),))[1]):
        _close(f(lib, argnums=1)(R, box), f(ref, argnums=1)(R, box))
    boxes = torch.stack([box, box * 1.1])
    _close(torch.vmap(lib, in_dims=(None, 0))(R, boxes), torch.vmap(ref, in_dims=(None, 0))(R, boxes))


def test_saved_tensor_hooks_and_tracing():
    R, lib, ref = _both()
    with torch.autograd.graph.save_on_cpu():
        x = R.clone().requires_grad_(True)
        E = lib(x)
    _close(torch.autograd.grad(E, x)[0], torch.func.grad(ref)(R))
    _, graph, _ = _setup()
    traced = torch.jit.trace(lambda R: graph(R).edges, (R,), check_trace=False)
    _close(traced(R * 1.1), graph(R * 1.1).edges)
