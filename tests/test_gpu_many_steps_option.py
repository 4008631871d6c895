"""MJ_OPT_MANY_STEPS: the launches of many steps switched off and on again, after a chosen
variant or configuration too; the kernels that run tell which, the bits stay the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ham, m0, steps=4, **kw):
    """(spins, names of the kernels launched)"""
    import matjes_b200 as mj
    from matjes_b200 import _abi

    m = m0.clone()
    _abi.check(_abi.lib.mj_profile_enable(ham.plan, 1))
    mj.SpinDynamics(ham, integrator="sib", timestep=0.1, alpha=0.1, temperature=5.0, noise="philox", seed=3, **kw).run(m, steps)
    names = set(_abi.profile_read(ham.plan))
    _abi.check(_abi.lib.mj_profile_enable(ham.plan, 0))
    return m, names


def test_plan():
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    ham = mj.Hamiltonian(mj.triangular((70, 45)))
    m0 = torch.tensor(mj.random_sphere(ham.N, 5).T.copy(), device="cuda")
    ref, names = _run(ham, m0)
    assert names == {"k_steps"}

    def option(value):
        _abi.check(_abi.lib.mj_plan_set_option(ham.plan, _abi.MJ_OPT_MANY_STEPS, value))

    option(0)
    m, names = _run(ham, m0)
    assert names == {"k_sib1", "k_sib2"} and torch.equal(m, ref)
    option(1)
    assert _run(ham, m0)[1] == {"k_steps"}
    _abi.check(_abi.lib.mj_plan_set_variant(ham.plan, 3))
    m, names = _run(ham, m0)
    assert names == {"k_sib1", "k_sib2"} and torch.equal(m, ref)
    option(1)
    m, names = _run(ham, m0)
    assert names == {"k_steps"} and torch.equal(m, ref)
    # a captured graph follows the option
    for value in (1, 0, 1):
        option(value)
        state = mj.SpinState(ham, m0)
        d = mj.SpinDynamics(ham, integrator="sib", timestep=0.1, alpha=0.1, temperature=5.0, noise="philox", seed=3)
        _abi.check(_abi.lib.mj_graph_run(ham.plan, state.handle, _abi.C.byref(d.p), 4, 1, None,
                                         torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(state.device_tensor(), ref)


def test_batch():
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    b = mj.ReplicaBatch(mj.square_film((8, 8, 1)), [(64, 48), (40, 24)], np.zeros((2, 3)), [1.0, 9.0])
    m0 = mj.random_sphere(b.N, 4)
    out = []
    for change in (lambda: None,
                   lambda: _abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_MANY_STEPS, 0),
                   lambda: _abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_MANY_STEPS, 1),
                   lambda: b.set_config(0, 4),
                   lambda: _abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_MANY_STEPS, 1)):
        change()
        b.upload(m0)
        p = b.params(timestep=0.1, alpha=0.5, noise="philox", seed=2)
        E = b.step(p, 5, energies=True).clone()
        b.graph_run(p, 4, 2)
        out.append((E, b.device_tensor().clone()))
    assert all(torch.equal(o[1], out[0][1]) for o in out)
    assert torch.equal(out[4][0], out[3][0]) and torch.equal(out[1][0], out[0][0])
