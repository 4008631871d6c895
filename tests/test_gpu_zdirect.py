"""The direct z sum of the dipolar term against the cuFFT z transforms: one plane to
the most it serves, open and periodic z axes, plane counts around its four warps,
column counts that are no multiple of 32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lz", [1, 2, 3, 4, 5, 8, 9, 13, 16])
@pytest.mark.parametrize("periodic", [(1, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1)])
@pytest.mark.parametrize("xy", [(5, 7), (16, 12)])
def test_direct_z_sum_equals_the_transforms(xy, periodic, Lz):
    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = mj.square_film((*xy, Lz), Jv=0.0, Dv=0.0, Kv=0.0, Bz=0.0, periodic=periodic, a=0.25, med_z=-0.3, dip=True)
    m = mj.random_sphere(deck.nsites, 3)
    ham = mj.Hamiltonian(deck)
    B, e = ham.get_eff_field(m, with_energy=True)
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, 6, 0))  # MJ_OPT_DIP_ZCONV off: cuFFT along z
    Bt, et = ham.get_eff_field(m, with_energy=True)
    # both are sums of the same products in another order: the suite's 1e-13 of the largest field
    assert np.abs(B - Bt).max() <= 1e-13 * np.abs(Bt).max()
    assert np.abs(e - et).max() <= 1e-13 * np.abs(et).max()
