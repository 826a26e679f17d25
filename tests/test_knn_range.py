"""The cells of the k-nearest search cover the nodes' whole range, however
many that takes in one joint: results equal the oracle's, and a joint of many
cells costs no more than its share."""
import time

import numpy as np
import pytest

from test_knn_bound import same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndof,stretch", [(1, 1.0), (2, 3e5), (3, 1e6), (6, 1e12), (7, 3e37)])
def test_one_long_joint(ndof, stretch):
    rng = np.random.default_rng(ndof)
    n = 40000
    x = rng.uniform(-1, 1, (n, ndof)).astype(np.float32)
    x[:, -1] *= np.float32(stretch)
    same(x, 10, rng.choice(n, 60, replace=False))


def test_one_outlier():
    rng = np.random.default_rng(3)
    x = rng.uniform(-1, 1, (20000, 3)).astype(np.float32)
    x[77, 1] = 3e38
    same(x, 8, rng.choice(20000, 60, replace=False))


def test_many_nodes_in_one_joint_take_no_scan_of_each_other():
    import torch
    from gpuprm_b200.neighbours import NeighbourIndex
    took = []
    for ndof in (1, 2):
        x = torch.rand((ndof, 200000), device="cuda:0", generator=torch.Generator("cuda:0").manual_seed(1))
        ix = NeighbourIndex(ndof)
        ix.build(x)
        best = 1e9
        for _ in range(10):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ix.knn(1)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        took.append(best)
    assert took[0] < 5 * took[1]              # 400 times with 91 % of the nodes in the last cell
