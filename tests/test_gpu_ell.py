"""ELL plans from COO couplings against a dense product: few distinct tensors
(held by id) and many (held per entry), rows without entries, isotropic and
full tensors side by side, site counts around a block's 256."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def couplings(N, ntensor, seed):
    """Blocks (i, j, H): up to six per row, none for every seventh row, tensors drawn from a list of ntensor."""
    rng = np.random.default_rng(seed)
    tab = rng.standard_normal((ntensor, 3, 3))
    tab[::2] = tab[::2, 0, 0][:, None, None] * np.eye(3)  # every other one isotropic
    out = []
    for i in range(N):
        if i % 7 == 0:
            continue
        for j in rng.choice(N, size=min(N, 1 + i % 6), replace=False):
            out.append((i, int(j), tab[rng.integers(ntensor)]))
    return out


@pytest.mark.parametrize("ntensor", [1, 2, 31, 2000])
@pytest.mark.parametrize("N", [1, 255, 256, 257, 700])
def test_ell_field_and_step_match_the_dense_product(N, ntensor):
    import torch

    import matjes_b200 as mj

    blocks = couplings(N, ntensor, 10 * N + ntensor)
    H = np.zeros((3 * N, 3 * N))
    rows, cols, vals = [], [], []
    for i, j, T in blocks:
        for a in range(3):
            for b in range(3):
                if T[a, b] != 0.0:
                    rows.append(3 * i + a)
                    cols.append(3 * j + b)
                    vals.append(T[a, b])
                    H[3 * i + a, 3 * j + b] += T[a, b]
    rng = np.random.default_rng(1)
    zee, b = rng.uniform(0.5, 1.5, N), rng.standard_normal((N, 3))
    ham = mj.Hamiltonian.from_coo(N, rows, cols, vals, zeeman=zee, b_site=b)
    m = mj.random_sphere(N, 3)
    B, e = ham.get_eff_field(m, with_energy=True)
    pair = -(H + H.T) @ m.ravel()
    want = pair.reshape(N, 3) - zee[:, None] * b
    # at most 2 x 6 N / N couplings of a row sum in another order: a few ulp of the row's absolute sum
    scale = (np.abs(H + H.T) @ np.abs(m.ravel())).reshape(N, 3) + np.abs(zee[:, None] * b)
    tol = 2.0 ** -52 * (4 + np.count_nonzero(H + H.T, axis=1).reshape(N, 3))
    assert (np.abs(B - want) <= tol * scale).all()
    e_want = -0.5 * (m * pair.reshape(N, 3)).sum(1) + zee * (m * b).sum(1)
    assert np.abs(e - e_want).max() <= 4 * (tol * scale).max()
    mt = torch.tensor(m.T.copy(), device="cuda")
    mj.SpinDynamics(ham, "sib", timestep=1e-3, alpha=0.1).run(mt, 2)
    assert abs(float(torch.linalg.norm(mt, dim=0).max()) - 1.0) < 1e-13
