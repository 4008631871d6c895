"""The routes of the dipolar term's z part over the plans that the rule tells apart: one
plane, power-of-two z grids below and above the limit on the columns (fused z transforms
of 2 to 16 planes), other z grids, a third lattice vector that is not normal to the
planes (K without the mirror symmetry), periodic z, and the grid padded on every axis."""
import numpy as np
import pytest

from conftest import scalar_rel_err, site_rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _deck(L, periodic, tilt, dip):
    import matjes_b200 as mj

    deck = mj.square_film(L, Jv=0.0, Dv=0.0, Kv=0.0, Bz=0.0, periodic=periodic, a=0.25, med_z=-0.3, dip=dip)
    if tilt:
        areal = deck.areal.copy()
        areal[2] += 0.4 * areal[0] + 0.2 * areal[1]
        deck.areal = areal
    return deck


@pytest.mark.parametrize("L,periodic,tilt,dip", [
    ((24, 20, 1), (0, 0, 0), 0, 1), ((150, 130, 1), (1, 1, 0), 0, 1),
    ((40, 36, 2), (0, 0, 0), 0, 1), ((210, 200, 2), (0, 0, 0), 0, 1), ((200, 196, 4), (0, 0, 0), 0, 1),
    ((150, 140, 8), (0, 0, 0), 0, 1), ((60, 50, 8), (1, 1, 0), 0, 1),
    ((220, 200, 2), (1, 1, 1), 0, 1), ((220, 200, 4), (1, 1, 1), 0, 1), ((30, 28, 8), (1, 1, 1), 0, 1),
    ((190, 200, 6), (0, 0, 0), 0, 1), ((64, 60, 6), (0, 0, 0), 0, 1), ((190, 190, 5), (1, 1, 1), 0, 1),
    ((33, 31, 2), (0, 0, 0), 1, 1), ((33, 31, 4), (1, 1, 0), 1, 1), ((33, 31, 3), (0, 0, 0), 1, 1),
    ((33, 31, 7), (1, 1, 0), 1, 1), ((33, 31, 11), (0, 0, 0), 1, 1), ((33, 31, 13), (0, 0, 0), 1, 1),
    ((33, 31, 5), (1, 1, 1), 1, 1), ((40, 36, 3), (1, 1, 1), 0, 2), ((40, 36, 4), (1, 1, 0), 0, 2),
    ((150, 140, 8), (1, 1, 1), 0, 2)])
def test_every_route_gives_the_field_of_the_cufft_z_transforms(L, periodic, tilt, dip):
    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = _deck(L, periodic, tilt, dip)
    m = mj.random_sphere(deck.nsites, 7)
    ham = mj.Hamiltonian(deck)
    B, e = ham.get_eff_field(m, with_energy=True)
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_DIP_ZCONV, 0))
    Bt, et = ham.get_eff_field(m, with_energy=True)
    # sums of the same products in another order: 1e-13 of the largest field
    assert np.abs(B - Bt).max() <= 1e-13 * np.abs(Bt).max()
    assert np.abs(e - et).max() <= 1e-13 * np.abs(et).max()
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_DIP_ZCONV, 1))
    B1, e1 = ham.get_eff_field(m, with_energy=True)
    assert np.array_equal(B1, B) and np.array_equal(e1, e)


@pytest.mark.parametrize("L,periodic", [((7, 6, 2), (0, 0, 0)), ((6, 5, 3), (1, 1, 0)), ((5, 4, 7), (0, 0, 0)),
                                        ((4, 4, 11), (0, 1, 0)), ((6, 4, 4), (0, 0, 0)), ((5, 4, 3), (1, 1, 1))])
def test_tilted_third_vector_matches_the_oracle(L, periodic):
    import matjes_b200 as mj

    deck = _deck(L, periodic, 1, 1)
    m = mj.random_sphere(deck.nsites, 11)
    B, e = mj.Hamiltonian(deck).get_eff_field(m, with_energy=True)
    Bo, eo = O.Model(deck).field(m)
    assert site_rel_err(B, Bo) < 1e-12
    assert scalar_rel_err(e, eo) < 1e-12
