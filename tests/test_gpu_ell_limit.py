"""ELL plans on both sides of the number of distinct tensors that are held by id: 128 go
by id (4 bytes an entry), 129 by value (76 bytes), each equal to the sum over its
couplings, written out in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def couplings(N, ntensor, seed):
    """Pairs i < j along two rings, symmetric tensors from a list of ntensor, every one of them used
    (couplings of one direction alone: the merged matrix then holds exactly these, negated)."""
    rng = np.random.default_rng(seed)
    tab = rng.standard_normal((ntensor, 3, 3))
    tab = tab + tab.transpose(0, 2, 1)
    tab[::5] = tab[::5, 0, 0][:, None, None] * np.eye(3)  # every fifth one isotropic
    i = np.concatenate([np.arange(N - 1), np.arange(N - 7)])
    j = np.concatenate([np.arange(N - 1) + 1, np.arange(N - 7) + 7])
    return i, j, tab[np.arange(i.size) % ntensor]


@pytest.mark.parametrize("ntensor", [1, 127, 128, 129])
def test_both_sides_of_the_limit(ntensor):
    import torch

    import matjes_b200 as mj

    N = 300_001
    i, j, T = couplings(N, ntensor, ntensor)
    a, b = np.meshgrid(np.arange(3), np.arange(3), indexing="ij")
    rows = (3 * i[:, None, None] + a).ravel()
    cols = (3 * j[:, None, None] + b).ravel()
    vals = T.ravel()
    keep = vals != 0.0
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    ham = mj.Hamiltonian.from_coo(N, rows[keep], cols[keep], vals[keep])
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    by_value = 4 * 76 * N  # four entries a row
    # (a plan's scratch is about 150 bytes a site, twice as much with the staging of host arrays)
    assert (held < by_value) == (ntensor <= 128)
    m = mj.random_sphere(N, 2)
    B = ham.get_eff_field(m)
    want, scale = np.zeros((N, 3)), np.zeros((N, 3))
    for p, q in ((i, j), (j, i)):  # (the tensors are symmetric)
        np.add.at(want, p, -np.einsum("kab,kb->ka", T, m[q]))
        np.add.at(scale, p, np.einsum("kab,kb->ka", np.abs(T), np.abs(m[q])))
    # twelve products a component in another order
    assert (np.abs(B - want) <= 16 * 2.0 ** -52 * scale).all()
