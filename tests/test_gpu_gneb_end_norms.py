"""A path whose end images are off unit length (spins read back with a few digits): the
angles to them, and with them the spring forces, are those of their directions, on every
form of the images' field pass, as the oracle has them."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("holder", ["batch", "plan", "cubic"])
@pytest.mark.parametrize("nim", [3, 7])
def test_end_images_off_unit_length(holder, nim):
    from matjes_b200 import Hamiltonian
    from matjes_b200.deck import square_film
    from matjes_b200.gneb import GNEBInput, find_path, find_path_plan, geodesic_path

    L = (6, 6, 3) if holder == "cubic" else (35, 10, 1)
    deck = square_film(L, Jv=1e-3, Dv=0.4e-3, Kv=-0.2e-3, Bz=0.3, mu_s=2.0, periodic=(1, 1, 0),
                       **(dict(a=0.25, med_z=-0.3) if holder == "cubic" else {}))
    n = deck.nsites
    up = np.tile([0.0, 0.0, 1.0], (n, 1))
    path = geodesic_path(up, -up, nim, amp_rnd=1e-2, seed=6)
    rng = np.random.default_rng(8)
    path[0] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0, (n, 1))
    path[-1] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0, (n, 1))
    path = np.ascontiguousarray(path)
    inp = GNEBInput(spring=0.3, dt=0.02, mass=1.0, mepftol=0.0, itrmax=40, en_zero="I")
    res = find_path(deck, path, inp) if holder == "batch" else find_path_plan(Hamiltonian(deck), path, inp)
    op = path.copy()
    orx, oene, odene, oit, ofc = O.gneb_find_path(O.Model(deck), op, spring=0.3, dt=0.02, mass=1.0, ftol=0.0, itrmax=40,
                                                  en_zero="I")
    assert res.iterations == oit == 40
    # the bounds of the other comparisons with the oracle's relaxation
    assert np.abs(res.images - op).max() < 1e-10
    np.testing.assert_allclose(res.rx, orx, rtol=1e-10)
    assert np.abs(res.ene - oene).max() <= 1e-10 * np.abs(oene).max()
    assert res.max_force == pytest.approx(ofc, rel=1e-9)
