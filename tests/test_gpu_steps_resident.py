"""Many steps in one launch at three and four resident blocks per SM against the
same steps one call at a time (the tiled passes): spins bit for bit, at the tile
counts on both sides of each limit (148 SMs: 296, 444 and 592 tiles of 32 x 8)."""
import pytest

pytestmark = pytest.mark.gpu


def deck_of(kind, L):
    import matjes_b200 as mj

    if kind == "triangular, nearest":
        return mj.triangular(L, J=(1e-3,))
    if kind == "triangular, three shells":
        return mj.triangular(L)
    deck = mj.square_film((*L, 1))
    if kind == "square, two shells":
        deck.J = list(deck.J) + [(1, 1, 2, -0.2e-3)]
    return deck


# 296, 297, 444, 445, 592 and 593 tiles, the last tiles of each direction ragged
@pytest.mark.parametrize("L", [(250, 293), (95, 789), (382, 291), (157, 709), (250, 587), (31, 4738)])
@pytest.mark.parametrize("kind", ["square", "square, two shells", "triangular, nearest", "triangular, three shells"])
def test_resident_forms_equal_single_steps(kind, L):
    import torch

    import matjes_b200 as mj

    deck = deck_of(kind, L)
    ham = mj.Hamiltonian(deck)
    m0 = torch.tensor(mj.random_sphere(deck.nsites, 5).T.copy(), device="cuda")
    for integrator in ("sib", "heun", "euler"):
        for T in (0.0, 20.0):
            dyn = dict(integrator=integrator, timestep=0.2, alpha=0.2, temperature=T, noise="philox" if T else "off",
                       seed=7)
            one, many = m0.clone(), m0.clone()
            single = mj.SpinDynamics(ham, **dyn)
            for _ in range(3):
                single.run(one, 1, energies=False)
            mj.SpinDynamics(ham, **dyn).run(many, 3)
            assert torch.equal(one, many), (integrator, T)
