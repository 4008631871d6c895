"""Short runs of a batch between swap rounds: by themselves, and on both sides of the
step count from which the many-step launches are taken, the spins, energies and ladder
are those of the passes bit for bit.  Sizes without a last tile thinner than a reach of
two, so that the many-step launches serve every lattice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,sizes,periodic", [
    ("square", [(256, 256)] * 21 + [(64, 32)] * 3, (1, 1, 0)),
    ("square", [(320, 480)] * 5, (0, 0, 0)),
    ("triangular", [(5, 40), (34, 10), (64, 48), (70, 45), (32, 8), (98, 61)], (1, 1, 0)),
    ("triangular", [(320, 320)] * 4 + [(34, 18)], (0, 0, 0))])
def test_short_runs_equal_the_passes(kind, sizes, periodic):
    import torch

    import matjes_b200 as mj

    cell = mj.square_film((8, 8, 1), periodic=periodic) if kind == "square" else mj.triangular((8, 8))
    cell.periodic = periodic
    n = len(sizes)
    B = np.zeros((n, 3))
    B[:, 2] = np.linspace(0.0, 1.0, n)
    out = []
    for passes in (False, True):
        b = mj.ReplicaBatch(cell, sizes, B, np.linspace(1.0, 40.0, n))
        if passes:
            b.set_config(3, 8)
        b.upload(mj.random_sphere(b.N, 5))
        p = b.params(timestep=0.1, alpha=0.5, noise="philox", seed=4, step0=4)
        E = []
        for steps, swap in ((1, 0), (2, 0), (1, 1), (5, 2), (3, 0), (16, 4), (20, 0)):
            E.append(b.step(p, steps, swap_every=swap, energies=True).clone())
        b.graph_run(p, 4, 3, swap_every=2)
        out.append((torch.stack(E), b.device_tensor().clone(), torch.tensor(b.temperatures()[0])))
    for x, y in zip(*out):
        assert torch.equal(x, y)
