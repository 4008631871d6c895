"""A film on the direct z sum holds its kernel once: the cuFFT route's K_F (6 values per
wave vector) is made when that route is asked for, not beside the planes' K."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _used():
    import torch

    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("L,periodic", [((128, 160, 13), (0, 0, 0)), ((160, 128, 7), (1, 1, 1))])
def test_kernel_is_held_once(L, periodic):
    import matjes_b200 as mj
    from matjes_b200 import _abi

    deck = mj.square_film(L, Jv=0.0, Dv=0.0, Kv=0.0, Bz=0.0, periodic=periodic, a=0.25, med_z=-0.3, dip=True)
    ham = mj.Hamiltonian(deck)
    m = mj.random_sphere(deck.nsites, 2)
    B = ham.get_eff_field(m)
    used = _used()
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_DIP_ZCONV, 0))
    n = [k if p else 2 * k for k, p in zip(L, periodic)]
    kf = 6 * 8 * (n[0] // 2 + 1) * n[1] * n[2]  # bytes of a real K_F
    assert _used() - used >= 0.9 * kf  # (allocations come in 2 MiB steps)
    Bt = ham.get_eff_field(m)
    assert np.abs(B - Bt).max() <= 1e-13 * np.abs(Bt).max()
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_DIP_ZCONV, 1))
    assert np.array_equal(ham.get_eff_field(m), B)
