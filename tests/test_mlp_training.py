"""Training on the B200: the same bits whatever came before, and however many
steps one graph holds."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed=3):
    import torch
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    q = (torch.rand((6, n), device="cuda:0", generator=g) * 2 - 1) * 3
    y = (q.abs().sum(0) > 9).float()
    return q.contiguous(), y.contiguous()


def _model(path, seed=5, scale=1.0):
    from gpuprm_b200.mlp import CollisionMLP
    m = CollisionMLP(6, seed=seed)
    m.set_training(path)
    m.set_params(m.get_params() * np.float32(scale))
    return m


@pytest.mark.parametrize("path", ["tcgen05", "mma_sync"])
def test_set_params_is_seen_by_the_next_step(path):
    """The weights that set_params uploads are those that the next kernels
    read: a run's bits do not depend on the model or the run before it."""
    q, y = _data(2048)
    ref = None
    for it in range(12):
        m = _model(path, scale=1.0)
        if it % 3 == 2:
            _model(path, seed=6, scale=-2.0).train(q, y, epochs=1, batch=256)
        m.train(q, y, epochs=1, batch=256)
        p = m.get_params()
        ref = p if ref is None else ref
        np.testing.assert_array_equal(p, ref)


@pytest.mark.parametrize("path", ["tcgen05", "mma_sync"])
@pytest.mark.parametrize("steps,batch", [(1, 1), (1, 200), (7, 128), (8, 129), (9, 64), (13, 300), (16, 256)])
def test_an_epoch_is_its_steps_one_by_one(path, steps, batch):
    """The replayed graph holds the largest divisor of the step count that is
    at most 8 (1, 7, 8, 3, 1, 8 here); two epochs of it are, bit for bit, the
    same steps run as separate calls of one step each (Adam's state stays in
    the model), and the epochs' losses are the mean of the steps'."""
    import torch
    n = steps * batch + (3 if batch > 3 else 0)      # a remainder that no step uses
    q, y = _data(n)
    epochs, seed = 2, 11
    a, b = _model(path), _model(path)
    losses = a.train(q, y, epochs=epochs, batch=batch, lr=2e-3, seed=seed)
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    perm = torch.stack([torch.randperm(n, device="cuda:0", generator=g) for _ in range(epochs)]).to(torch.int32)
    for e in range(epochs):
        one = []
        for s in range(steps):
            part = perm[e, s * batch:(s + 1) * batch].contiguous()
            torch.cuda.synchronize()
            loss = np.zeros(1, np.float32)
            b._check(b.lib.gprm_mlp_train(b.h, C.c_void_p(q.data_ptr()), C.c_void_p(y.data_ptr()), batch, n,
                                          C.c_void_p(part.data_ptr()), 1, batch, 2e-3,
                                          loss.ctypes.data_as(C.POINTER(C.c_float))))
            one.append(float(loss[0]))
        # FP32 sums of up to 16 steps' block sums in another order
        assert abs(losses[e] - np.mean(one)) <= 1e-5 * abs(np.mean(one))
    np.testing.assert_array_equal(a.get_params(), b.get_params())
    assert a.device_status() == 0
