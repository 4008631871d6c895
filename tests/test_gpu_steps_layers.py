"""Many steps in one launch over the layers of a lattice without couplings between them,
and with a field out of the easy axis (the full form of the stencil) on every shape,
against the passes: spins bit for bit, energies to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def deck_of(kind, L, periodic):
    from matjes_b200.deck import Deck, square_areal, triangular_areal

    tri = kind.startswith("tri")
    areal = triangular_areal(1.0, 6.0) if tri else square_areal(1.0, 6.0)
    shells = {"square": 1, "square2": 2, "tri": 1, "tri3": 3}[kind]
    return Deck(L=L, periodic=periodic, areal=areal, atoms=[((0, 0, 0), 1, 2.0)],
                J=[(1, 1, s + 1, v) for s, v in enumerate([1e-3, -0.3e-3, 0.2e-3][:shells])],
                K=[(1, (0.0, 0.0, 1.0), -0.1e-3)], B_ext=(0.4, -0.2, 0.5))


@pytest.mark.parametrize("L", [(40, 21, 2), (32, 8, 5), (70, 45, 3), (300, 90, 4)])
@pytest.mark.parametrize("kind,periodic", [("square", (1, 1, 0)), ("square2", (0, 1, 0)), ("tri", (1, 0, 0)),
                                           ("tri3", (1, 1, 0)), ("tri3", (0, 0, 0))])
def test_layers_equal_the_passes(kind, periodic, L):
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = deck_of(kind, L, periodic)
    m0 = torch.tensor(mj.random_sphere(L[0] * L[1] * L[2], 3).T.copy(), device="cuda")
    out = []
    for many in (1, 0):
        ham = mj.Hamiltonian(deck)
        _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_MANY_STEPS, many))
        runs = []
        for integrator in ("sib", "heun", "euler"):
            m = m0.clone()
            _abi.check(_abi.lib.mj_profile_enable(ham.plan, 1))
            E = mj.SpinDynamics(ham, integrator=integrator, timestep=0.2, alpha=0.2, temperature=20.0, noise="philox",
                                seed=7).run(m, 5, energies=True)
            names = set(_abi.profile_read(ham.plan))
            assert ("k_steps" in names) == bool(many), names
            _abi.check(_abi.lib.mj_profile_enable(ham.plan, 0))
            e = ham.energy_distrib(m).abs().sum().item()
            runs.append((m, E, e))
        out.append(runs)
    for (m, E, e), (m1, E1, _) in zip(*out):
        assert torch.equal(m, m1)
        # sums of the same site energies in another order (as in the single-layer comparison)
        assert (E - E1).abs().max().item() <= 2.0 ** -52 * max(64, m.shape[1]) ** 0.5 * 8 * e


@pytest.mark.parametrize("kind", ["square", "square2", "tri", "tri3"])
@pytest.mark.parametrize("periodic", [(1, 1, 0), (0, 0, 0)])
def test_batch_shapes_equal_the_passes(kind, periodic):
    import torch

    import matjes_b200 as mj

    sizes = [(34, 10), (64, 48), (70, 45), (32, 8), (98, 61), (8, 16)]
    n = len(sizes)
    B = np.tile([0.3, 0.1, 0.5], (n, 1)) * np.linspace(0.5, 1.0, n)[:, None]
    out = []
    for passes in (False, True):
        b = mj.ReplicaBatch(deck_of(kind, (8, 8, 1), periodic), sizes, B, np.linspace(0.0, 40.0, n))
        if passes:
            b.set_config(3, 8)
        b.upload(mj.random_sphere(b.N, 6))
        E = b.step(b.params(timestep=0.1, alpha=0.5, noise="philox", seed=3), 9, energies=True)
        out.append((b.device_tensor().clone(), E.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
