"""A batch's steps in many-step launches (the default) against its passes (a chosen
configuration): the spins bit for bit, with uneven sizes, single tiles, open edges,
in-plane fields, hot and cold replicas, groups larger than what is resident, swaps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(kind, sizes, periodic, inplane):
    import matjes_b200 as mj

    cell = mj.square_film((8, 8, 1), periodic=periodic) if kind == "square" else mj.triangular((8, 8))
    if kind != "square":
        cell.periodic = periodic
    n = len(sizes)
    B = np.zeros((n, 3))
    B[:, 2] = np.linspace(0.0, 1.0, n)
    if inplane:
        B[:, 0] = 0.2
    T = np.where(np.arange(n) % 3 == 0, 0.0, np.linspace(1.0, 40.0, n))
    return mj.ReplicaBatch(cell, sizes, B, T)


@pytest.mark.parametrize("kind", ["square", "triangular"])
@pytest.mark.parametrize("periodic", [(1, 1, 0), (0, 0, 0)])
@pytest.mark.parametrize("case", ["few", "uneven", "many"])
def test_many_step_launches_equal_the_passes(kind, periodic, case):
    import torch

    import matjes_b200 as mj

    sizes = {"few": [(16, 16), (16, 16)], "uneven": [(5, 40), (33, 9), (64, 48), (70, 45), (32, 8), (97, 61)],
             "many": [(256, 256)] * 5 + [(96, 64)] * 7}[case]
    out = []
    for passes in (False, True):
        b = batch(kind, sizes, periodic, inplane=case == "uneven")
        if passes:
            b.set_config(3, 8)
        b.upload(mj.random_sphere(b.N, 3))
        p = b.params(timestep=0.1, alpha=0.5, noise="philox", seed=9, step0=2)
        E = b.step(p, 7, swap_every=3, energies=True)
        out.append((b.device_tensor().clone(), E.clone(), b.temperatures()[0]))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])
