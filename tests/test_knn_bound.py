"""The k-nearest search where its bound and its candidate buffer can go
wrong: every dimension, fewer nodes than k, more equidistant nodes than the
buffer holds, nodes on cell faces, non-finite nodes, and queries that outgrow
the first block.  Indices and float32 distances equal the oracle's."""
import numpy as np
import pytest

import nbr_oracle as NO

pytestmark = pytest.mark.gpu


def search(x, k, q=None):
    import torch
    from gpuprm_b200.neighbours import NeighbourIndex
    ix = NeighbourIndex(x.shape[1])
    ix.build(torch.tensor(np.ascontiguousarray(x.T), device="cuda:0"))
    qd = None if q is None else torch.tensor(np.ascontiguousarray(q.T), device="cuda:0")
    idx, dist = ix.knn(k, q=qd)
    torch.cuda.synchronize()
    return idx.cpu().numpy(), dist.cpu().numpy()


def same(x, k, sample):
    idx, dist = search(x, k)
    want_i, want_d = NO.knn(x, x[sample], k, exclude=sample)
    np.testing.assert_array_equal(idx[sample], want_i)
    np.testing.assert_array_equal(dist[sample], want_d)


@pytest.mark.parametrize("ndof", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("k", [1, 10, 32])
def test_every_dimension(ndof, k):
    rng = np.random.default_rng(ndof)
    n = 6000
    x = rng.uniform(-3, 3, (n, ndof)).astype(np.float32)
    x[:500] = rng.normal(0, 0.02, (500, ndof))           # a dense spot among sparse ones
    same(x, k, rng.choice(n, 150, replace=False))


def test_fewer_nodes_than_k():
    x = np.random.default_rng(1).uniform(-1, 1, (9, 4)).astype(np.float32)
    same(x, 16, np.arange(9))


@pytest.mark.parametrize("ndof", [1, 6])
def test_more_ties_than_the_buffer(ndof):
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (1500, ndof)).astype(np.float32)
    x[200:900] = x[0]                                     # 700 nodes at distance 0 of one another
    same(x, 32, np.concatenate([np.arange(195, 240), np.arange(895, 920)]))


def test_lattice_on_cell_faces():
    g = np.arange(-4, 4, dtype=np.float32)
    x = np.stack(np.meshgrid(g, g, g, g, indexing="ij"), -1).reshape(-1, 4).astype(np.float32)
    same(x, 20, np.random.default_rng(3).choice(len(x), 200, replace=False))


def test_non_finite_nodes_sort_last():
    rng = np.random.default_rng(4)
    x = rng.uniform(-2, 2, (3000, 6)).astype(np.float32)
    x[5, 2], x[6, 0], x[7] = np.nan, np.inf, -np.inf
    finite = np.setdiff1d(np.arange(3000), [5, 6, 7])
    same(x, 10, rng.choice(finite, 100, replace=False))


def test_outside_queries_with_a_bound():
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, (20000, 5)).astype(np.float32)
    q = rng.uniform(-1.6, 1.6, (300, 5)).astype(np.float32)
    idx, dist = search(x, 12, q)
    want_i, want_d = NO.knn(x, q, 12)
    np.testing.assert_array_equal(idx, want_i)
    np.testing.assert_array_equal(dist, want_d)
