"""Many steps in one launch (small lattices) against the same steps one call at a
time, which run the tiled passes: spins bit for bit, energies to rounding; sizes
at the edges of the 32 x 8 tiles, halos that wrap onto the own tile, last tiles
thinner than the reach, the largest lattices of both forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (5, 40), (31, 7), (32, 8), (33, 9), (34, 10), (40, 17), (65, 66), (70, 45), (256, 256),
         (300, 290), (448, 416), (511, 509)]


def lattice(kind, L, periodic):
    import matjes_b200 as mj

    if kind == "square":
        return mj.square_film((*L, 1), periodic=periodic)
    deck = mj.triangular(L)
    deck.periodic = periodic
    return deck


@pytest.mark.parametrize("L", SIZES)
@pytest.mark.parametrize("kind,periodic", [("square", (1, 1, 0)), ("square", (0, 0, 0)), ("triangular", (1, 1, 0)),
                                           ("triangular", (1, 0, 0))])
def test_steps_in_one_launch_equal_single_steps(kind, periodic, L):
    import torch

    import matjes_b200 as mj

    if not all(periodic[:2]) and min(L) < 5:
        pytest.skip("an open lattice this small has no bonds of every shell: no plan is built")
    deck = lattice(kind, L, periodic)
    ham = mj.Hamiltonian(deck)
    rng = np.random.default_rng(L[0] + 1000 * L[1])
    bmap = rng.standard_normal((deck.ncell, 3)) if L[0] % 2 else None  # every odd size with a field map
    if bmap is not None:
        ham.set_bfield(bmap)
    m0 = torch.tensor(mj.random_sphere(deck.nsites, 3).T.copy(), device="cuda")
    for integrator in ("sib", "heun", "euler"):
        for n, T in ((2, 0.0), (5, 20.0)):
            dyn = dict(integrator=integrator, timestep=0.2, alpha=0.2, temperature=T, noise="philox" if T else "off",
                       seed=7)
            one, many = m0.clone(), m0.clone()
            single = mj.SpinDynamics(ham, **dyn)
            E1 = torch.cat([single.run(one, 1, energies=True) for _ in range(n)])
            En = mj.SpinDynamics(ham, **dyn).run(many, n, energies=True)
            assert torch.equal(one, many), (integrator, n, T)
            # sums of the same site energies in another order: N roundings of the absolute sum at most
            e = ham.energy_distrib(many).abs().sum().item()
            assert (E1 - En).abs().max().item() <= 2.0 ** -52 * max(64, deck.nsites) ** 0.5 * 8 * e
            bare = m0.clone()
            mj.SpinDynamics(ham, **dyn).run(bare, n)
            assert torch.equal(bare, many)


@pytest.mark.parametrize("integrator", ["sib", "euler"])
def test_energies_over_several_launches_and_under_a_graph(integrator):
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = mj.square_film((40, 24, 1))
    ham = mj.Hamiltonian(deck)
    m0 = torch.tensor(mj.random_sphere(deck.nsites, 3).T.copy(), device="cuda")
    dyn = dict(integrator=integrator, timestep=0.2, alpha=0.2, temperature=5.0, noise="philox", seed=3)
    one, many = m0.clone(), m0.clone()
    single = mj.SpinDynamics(ham, **dyn)
    E1 = torch.cat([single.run(one, 1, energies=True) for _ in range(130)])  # 130 steps: launches of 63, 63 and 4
    En = mj.SpinDynamics(ham, **dyn).run(many, 130, energies=True)
    assert torch.equal(one, many)
    tol = 2.0 ** -52 * deck.nsites * ham.energy_distrib(many).abs().max().item() * 8
    assert (E1 - En).abs().max().item() <= tol
    before = mj.SpinDynamics(ham, **dyn)
    before.p.energy_mode = 1
    Eb = before.run(m0.clone(), 130, energies=True)
    assert (Eb[1:] - En[:-1]).abs().max().item() <= tol
    state = mj.SpinState(ham, m0)
    graph = mj.SpinDynamics(ham, **dyn)
    _abi.check(_abi.lib.mj_graph_run(ham.plan, state.handle, _abi.C.byref(graph.p), 26, 5, None,
                                     torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(state.device_tensor(), one)
