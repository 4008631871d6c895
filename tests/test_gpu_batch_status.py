"""A batch's report of a wait that ran out: asked for by itself after asynchronous calls,
given once, and by a download for the work of the stream that it runs on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch():
    import matjes_b200 as mj

    b = mj.ReplicaBatch(mj.square_film((8, 8, 1)), [(40, 24), (16, 16)], np.zeros((2, 3)), [1.0, 5.0])
    b.upload(mj.random_sphere(b.N, 2))
    return b


def _time_out(b, stream=None):
    from matjes_b200 import _abi

    _abi.check(_abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_TEST_TIMEOUT, 1))
    b.step(b.params(timestep=0.1, alpha=0.5), 2, stream=stream)
    _abi.check(_abi.lib.mj_batch_set_option(b.handle, _abi.MJ_OPT_TEST_TIMEOUT, 0))


def test_check_status_reports_once():
    import matjes_b200 as mj

    b = _batch()
    b.check_status()
    _time_out(b)
    with pytest.raises(mj.MatjesError, match="bounded device wait"):
        b.check_status()
    b.check_status()
    b.upload(mj.random_sphere(b.N, 2))
    b.step(b.params(timestep=0.1, alpha=0.5), 2)
    b.check_status()


def test_download_reports_for_its_stream():
    import torch

    import matjes_b200 as mj
    from matjes_b200 import _abi

    b = _batch()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    out = np.empty((b.N, 3))
    _time_out(b, s.cuda_stream)
    assert _abi.lib.mj_batch_download(b.handle, out.ctypes.data, s.cuda_stream) == _abi.MJ_ERR_TIMEOUT
    b.check_status()
    assert _abi.lib.mj_batch_download(b.handle, out.ctypes.data, s.cuda_stream) == _abi.MJ_OK


def test_a_path_is_not_relaxed_from_invalid_images():
    import matjes_b200 as mj

    b = mj.ReplicaBatch(mj.square_film((8, 8, 1)), [(16, 16)] * 4, np.zeros((4, 3)), [1.0] * 4)
    m = mj.random_sphere(b.N, 2)
    b.upload(m)
    _time_out(b)
    with pytest.raises(mj.MatjesError, match="bounded device wait"):
        b.gneb_path(0.3, 0.02, 1.0, 0.0, 5, "I")
    b.upload(m)
    assert b.gneb_path(0.3, 0.02, 1.0, 0.0, 5, "I")[3] == 5
