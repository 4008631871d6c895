"""The routes of the adjoint against one another: whole segments in one launch, the tiled
launches per step (larger lattices, last tiles thinner than the reach, a chosen variant),
the generic kernels (no compile-time shape), and lattices between the limits, whose
forward steps are one launch while the backward steps are not.  Every shape, open edges,
ragged tiles in both directions, a last segment shorter than the checkpoint spacing, a
field map and a thermal field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {"square": 1, "triangular, nearest": 2, "triangular, three shells": 3, "square, two shells": 4}


def deck_of(kind, L, periodic):
    import matjes_b200 as mj

    if kind == "triangular, nearest":
        deck = mj.triangular(L, J=(1e-3,))
    elif kind == "triangular, three shells":
        deck = mj.triangular(L)
    else:
        deck = mj.square_film((*L, 1))
        if kind == "square, two shells":
            deck.J = list(deck.J) + [(1, 1, 2, -0.2e-3)]
    deck.periodic = periodic
    return deck


def grads(kind, L, periodic, route, T, nsteps=7, every=3):
    import ctypes as C

    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = deck_of(kind, L, periodic)
    ham = mj.Hamiltonian(deck)
    v, shape = C.c_int32(), C.c_int32()
    _abi.check(_abi.lib.mj_plan_get_variant(ham.plan, C.byref(v), C.byref(shape)))
    assert shape.value == KINDS[kind]
    if route is not None:
        _abi.check(_abi.lib.mj_plan_set_variant(ham.plan, route))
    rng = np.random.default_rng(L[0] + 7 * L[1])
    m0 = torch.tensor(mj.random_sphere(ham.N, 3).T.copy(), device="cuda", requires_grad=True)
    terms = torch.tensor(mj.deck_terms(deck), requires_grad=True)
    b = torch.tensor(rng.standard_normal((3, ham.N)), device="cuda", requires_grad=True)
    gT = torch.tensor(rng.standard_normal((3, ham.N)), device="cuda")
    traj = mj.SIBTrajectory(ham, nsteps, every, timestep=0.5, alpha=0.3, temperature=T, noise="philox" if T else "off",
                            seed=5, step0=11)
    mT = traj(m0, terms, b)
    out = [mT.detach().clone()] + [g.clone() for g in torch.autograd.grad(mT, (m0, terms, b), gT)]
    ham.check_status()
    return out


def close(a, b, forward_equal):
    import torch

    if forward_equal:
        assert torch.equal(a[0], b[0])
    # 7 steps of the same arithmetic in another order: some hundred roundings, no cancellation beyond
    # the coupling sums' (their terms add at random: relative to their size still 1e-12)
    for x, y in zip(a, b):
        assert float((x - y).abs().max()) <= 1e-12 * float(y.abs().max())


@pytest.mark.parametrize("L", [(12, 10), (70, 45), (33, 9), (34, 10), (97, 61)])
@pytest.mark.parametrize("periodic", [(1, 1, 0), (0, 0, 0), (1, 0, 0)])
@pytest.mark.parametrize("kind", list(KINDS))
def test_routes_agree(kind, periodic, L):
    T = 10.0 if L[0] % 2 else 0.0
    ref = grads(kind, L, periodic, None, T)
    close(grads(kind, L, periodic, 5, T), ref, True)   # two tiled launches a step
    close(grads(kind, L, periodic, -1, T), ref, False)  # generic kernels


# 320 and 1230 tiles of 32 x 8: more than the segment launch holds, more than any launch holds
@pytest.mark.parametrize("L", [(314, 253), (950, 325)])
@pytest.mark.parametrize("kind", list(KINDS))
def test_lattices_above_the_limits(kind, L):
    ref = grads(kind, L, (1, 0, 0), -1, 10.0, nsteps=4)
    close(grads(kind, L, (1, 0, 0), None, 10.0, nsteps=4), ref, False)


@pytest.mark.parametrize("every", [1, 2, 5, 50])
def test_checkpoint_spacing(every):
    ref = grads("triangular, three shells", (70, 45), (1, 1, 0), 5, 10.0, nsteps=11, every=11)
    close(grads("triangular, three shells", (70, 45), (1, 1, 0), None, 10.0, nsteps=11, every=every), ref, True)


def test_layers():
    """Uncoupled layers: the forward steps of all of them in one launch, the backward per step."""
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi
    from matjes_b200.deck import Deck, square_areal

    deck = Deck(L=(40, 21, 3), periodic=(1, 1, 0), areal=square_areal(1.0, 5.0), atoms=[((0, 0, 0), 1, 2.0)],
                J=[(1, 1, 1, 1e-3)], K=[(1, (0.0, 0.0, 1.0), -0.1e-3)], B_ext=(0.3, 0.0, 0.5))
    out = []
    for many in (1, 0):
        ham = mj.Hamiltonian(deck)
        _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_MANY_STEPS, many))
        m0 = torch.tensor(mj.random_sphere(ham.N, 3).T.copy(), device="cuda")
        traj = mj.SIBTrajectory(ham, 6, 4, timestep=0.5, alpha=0.3)
        out.append([traj.forward(m0), *traj.backward(torch.ones_like(m0))])
    close(out[0], out[1], True)
