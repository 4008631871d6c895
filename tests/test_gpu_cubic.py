"""Simple-cubic nearest neighbours (unrolled) against the oracle: one-cell and odd
sides, every mix of periodic and open edges, the axial and the full form (in-plane
field, tilted axis), and steps with the stored draw and the energies split over
the two passes."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from tests.conftest import scalar_rel_err, site_rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["axial", "full"])
@pytest.mark.parametrize("L", [(2, 2, 2), (3, 2, 5), (33, 9, 2), (31, 8, 3), (6, 17, 4)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (1, 1, 0), (0, 1, 1), (0, 0, 0)])
def test_cubic_field_and_steps_match_the_oracle(periodic, L, form):
    import torch

    import matjes_b200 as mj

    deck = mj.square_film(L, Jv=1e-3, Dv=0.15e-3, Kv=-0.02e-3, Bz=0.2, a=0.25, med_z=-0.3, periodic=periodic)
    if form == "full":
        deck = dataclasses.replace(deck, K=[(1, (1.0, 2.0, 0.5), -0.1e-3)], B_ext=(0.3, -0.2, 0.5))
    ham = mj.Hamiltonian(deck)
    M = O.Model(deck)
    m = mj.random_sphere(deck.nsites, 11)
    B, e = ham.get_eff_field(m, with_energy=True)
    Bo, eo = M.field(m)
    assert site_rel_err(B, Bo) < 1e-12 and scalar_rel_err(e, eo) < 1e-12  # the suite's field tolerance
    for integrator in ("sib", "heun", "euler"):
        dyn = dict(integrator=integrator, timestep=0.1, alpha=0.2, temperature=20.0, noise="philox", seed=5)
        mt = torch.tensor(m.T.copy(), device="cuda")
        E = mj.SpinDynamics(ham, **dyn).run(mt, 4, energies=True).cpu().numpy()
        mo = m.copy()
        Eo = M.run(mo, 4, energies=True, **dyn)
        assert np.abs(mt.cpu().numpy().T - mo).max() < 1e-11  # four steps of a few 1e-16 each, with room
        assert np.abs(E - Eo).max() <= 1e-12 * np.abs(eo).sum()
