"""What a plan holds on the device before it is asked for more: two spin arrays of scratch
(midpoint, draw) and little besides; the minimiser's velocities come with its first run."""
import pytest

pytestmark = pytest.mark.gpu


def test_scratch_of_a_plan():
    import torch

    import matjes_b200 as mj

    deck = mj.square_film((2000, 1500, 1))
    f3 = 24 * deck.nsites
    m = torch.tensor(mj.random_sphere(deck.nsites, 1).T.copy(), device="cuda")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    ham = mj.Hamiltonian(deck)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 2.5 * f3
    m1 = m.clone()
    a = mj.minimize(ham, m1, conv_torque=1e-30, max_iter=20)
    b = mj.minimize(ham, m, conv_torque=1e-30, max_iter=20)
    assert a == b and torch.equal(m, m1)
