"""Trainings of few steps run without a graph: the same weights, bit for bit,
as the same steps from one, and no graph's cost."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data(steps, batch):
    import torch
    g = torch.Generator("cuda:0").manual_seed(steps)
    q = ((torch.rand((6, steps * batch), device="cuda:0", generator=g) * 2 - 1) * 3.14).contiguous()
    return q, (q[0] > 0).float(), torch.randperm(steps * batch, device="cuda:0", generator=g).to(torch.int32)


def train(m, q, y, perm, n, batch):
    losses = np.zeros(1, np.float32)
    rc = m.lib.gprm_mlp_train(m.h, C.c_void_p(q.data_ptr()), C.c_void_p(y.data_ptr()), n, q.shape[1],
                              C.c_void_p(perm.data_ptr()), 1, batch, 1e-3, losses.ctypes.data_as(C.POINTER(C.c_float)))
    assert rc == 0
    return float(losses[0])


@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("batch", [64, 1000])
def test_weights_equal_those_of_the_captured_steps(path, batch):
    import torch
    from gpuprm_b200.mlp import CollisionMLP
    steps = 40
    q, y, perm = data(steps, batch)
    out = []
    for cut in ((40,), (1, 32, 7)):               # one graph; three short trainings
        m = CollisionMLP(6, seed=4)
        assert m.lib.gprm_mlp_set_training(m.h, path) == 0
        at, loss = 0, 0.0
        for c in cut:
            torch.cuda.synchronize()
            loss += c * train(m, q, y, perm[at * batch:(at + c) * batch].contiguous(), c * batch, batch)
            at += c
        out.append((m.get_params(), loss / steps))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert abs(out[0][1] - out[1][1]) < 1e-5


def test_few_steps_cost_little_more_than_their_share():
    import torch
    from gpuprm_b200.mlp import CollisionMLP
    took = {}
    for steps in (8, 128):
        q, y, perm = data(steps, 1024)
        m = CollisionMLP(6, seed=4)
        best = 1e9
        for _ in range(12):
            torch.cuda.synchronize()
            t = time.perf_counter()
            train(m, q, y, perm, steps * 1024, 1024)
            best = min(best, time.perf_counter() - t)
        took[steps] = best
    assert took[8] < 2.2 * 8 / 128 * took[128]    # 3.5 with the graph of eight steps
