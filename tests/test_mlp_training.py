"""Training on the B200: the same bits whatever came before."""
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
