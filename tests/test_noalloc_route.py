"""gprm_indicator_batch_device_noalloc takes the kernels of
gprm_indicator_batch_device: one launch for a small request, the same codes
at and around the sizes where the route changes."""
import ctypes as C

import numpy as np
import pytest

from gpuprm_b200 import scenes
from gpuprm_b200._abi import GPRM_MODE_FP64_BAND
from gpuprm_b200.configspace import RobotConfigspace
from test_scan import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["box4", "slots"])
def test_small_requests_take_one_launch(kind):
    import torch
    sc = scenes.make_box4(2) if kind == "box4" else make(7, 3, 6, False, 0)
    cs = RobotConfigspace(sc, dq=0.02)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND)
    q = scenes.uniform_configs(sc, 33000, 3)
    want = cs.check_configs(q)
    t = torch.tensor(np.ascontiguousarray(q.T), device="cuda:0")
    st = torch.cuda.current_stream().cuda_stream
    for n in (1, 32, 593, 32768, 32769):
        x = t[:, :n].contiguous()
        res = torch.full((n,), -7, dtype=torch.int32, device="cuda:0")
        torch.cuda.synchronize()
        s = cs.stats()
        assert cs.lib.gprm_indicator_batch_device_noalloc(cs.h, C.c_void_p(x.data_ptr()), C.c_void_p(res.data_ptr()), n,
                                                          n, C.c_void_p(st)) == 0
        np.testing.assert_array_equal(res.cpu().numpy(), want[:n])
        e = cs.stats()
        assert e["vertex_checks"] - s["vertex_checks"] == n
        assert (e["launches"] - s["launches"] == 1) == (n <= 32768 or kind == "slots")
