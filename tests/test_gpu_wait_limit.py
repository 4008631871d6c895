"""The waits between the tiles of a many-step launch, made to run out: with
MJ_OPT_TEST_TIMEOUT no tile posts anything, every wait reaches its limit (about a
second) and the launch returns, without a fault.  The report comes once, the energies
and gradients are NaN and no numbers that could pass for results, and the same plan or
batch gives the same bits as before once the option is off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _deck(kind, L=(70, 45)):
    import matjes_b200 as mj

    return mj.triangular(L) if kind == "triangular" else mj.square_film((*L, 1))


@pytest.mark.parametrize("kind,integrator,steps", [("square", "sib", 2), ("square", "euler", 70), ("triangular", "heun", 2),
                                                   ("triangular", "sib", 70), ("square", "heun", 64)])
def test_plan(kind, integrator, steps):
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    ham = mj.Hamiltonian(_deck(kind))
    m0 = torch.tensor(mj.random_sphere(ham.N, 3).T.copy(), device="cuda")
    dyn = dict(integrator=integrator, timestep=0.1, alpha=0.1, temperature=5.0, noise="philox", seed=1)
    ref = m0.clone()
    Eref = mj.SpinDynamics(ham, **dyn).run(ref, steps, energies=True)
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_OK
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_TEST_TIMEOUT, 1))
    m = m0.clone()
    E = mj.SpinDynamics(ham, **dyn).run(m, steps, energies=True)  # every tile waits for a neighbour
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_ERR_TIMEOUT
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_OK
    assert torch.isnan(E).all()
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_TEST_TIMEOUT, 0))
    m = m0.clone()
    E = mj.SpinDynamics(ham, **dyn).run(m, steps, energies=True)
    assert torch.equal(m, ref) and torch.equal(E, Eref)
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_OK


@pytest.mark.parametrize("kind", ["square", "triangular"])
def test_adjoint(kind):
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    ham = mj.Hamiltonian(_deck(kind))
    m0 = torch.tensor(mj.random_sphere(ham.N, 4).T.copy(), device="cuda")
    gT = torch.ones_like(m0)
    traj = mj.SIBTrajectory(ham, 12, 5, timestep=0.1, alpha=0.2)
    ref = [traj.forward(m0), *traj.backward(gT)]
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_TEST_TIMEOUT, 1))
    traj.forward(m0)
    assert all(bool(torch.isnan(x).all()) for x in traj.backward(gT))
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_ERR_TIMEOUT
    assert _abi.lib.mj_plan_check_status(ham.plan) == _abi.MJ_OK
    _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_TEST_TIMEOUT, 0))
    out = [traj.forward(m0), *traj.backward(gT)]
    assert all(torch.equal(x, y) for x, y in zip(out, ref))


@pytest.mark.parametrize("swap", [0, 3])
def test_batch(swap):
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    sizes = [(64, 48), (33, 9), (70, 45)]
    b = mj.ReplicaBatch(_deck("square", (8, 8)), sizes, np.zeros((3, 3)), [1.0, 5.0, 20.0])
    m0 = mj.random_sphere(b.N, 3)

    def run():
        b.upload(m0)
        p = b.params(timestep=0.1, alpha=0.5, noise="philox", seed=9)
        return b.step(p, 6, swap_every=swap, energies=True)

    _abi.check(_abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_TEST_TIMEOUT, 1))
    assert torch.isnan(run()).all()
    with pytest.raises(mj.MatjesError, match="bounded device wait"):
        b.energies()
    b.energies()  # reported once
    _abi.check(_abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_TEST_TIMEOUT, 0))
    E = run().clone()
    assert torch.isfinite(E).all() and np.isfinite(b.download()).all()
    if not swap:  # (rounds on NaN energies may have moved temperatures)
        c = mj.ReplicaBatch(_deck("square", (8, 8)), sizes, np.zeros((3, 3)), [1.0, 5.0, 20.0])
        c.upload(m0)
        assert torch.equal(E, c.step(c.params(timestep=0.1, alpha=0.5, noise="philox", seed=9), 6, energies=True))
    assert _abi.lib.mj_batch_set_option(b.handle, 99, 1) == _abi.MJ_ERR_ARG
