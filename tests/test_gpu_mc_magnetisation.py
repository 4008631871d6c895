"""The summed spins of a Monte Carlo sweep against an exact sum: blocks that walk
the lattice with a stride, at a part of a block, just below and above one walk and
at a ragged number of walks."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(10, 6), (256, 592), (256, 593), (770, 1001)])
def test_summed_spins_equal_the_exact_sum(L):
    import torch

    import matjes_b200 as mj
    from matjes_b200.montecarlo import MetropolisMC

    deck = mj.square_film((L[0], L[1], 1), Jv=1e-3, Dv=0.3e-3, Kv=-0.1e-3, Bz=0.5, periodic=(0, 0, 0))
    ham = mj.Hamiltonian(deck)
    m = torch.tensor(mj.random_sphere(deck.nsites, 3).T.copy(), device="cuda")
    chain = MetropolisMC(ham, "sphere", cone=0.5, seed=11)
    _, Mg, _ = chain.sweeps(m, 1, 20.0)
    h = m.cpu().numpy()
    want = np.array([math.fsum(c) for c in h])
    # each term passes through fewer than 1000 roundings of partial sums bounded by sum |m|
    tol = 1000 * 2.0 ** -53 * np.abs(h).sum(1)
    assert np.all(np.abs(Mg[0].cpu().numpy() - want) <= tol)
