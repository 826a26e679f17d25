"""The nodes' own k-nearest search by a thread per query (up to three joints,
many nodes, a short list): indices and float32 distances equal the oracle's
at the sizes where it takes over, with ties, non-finite nodes and queries
that outgrow the first block."""
import numpy as np
import pytest

from test_knn_bound import same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndof", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(65535, 10), (65536, 1), (65536, 10), (65536, 11), (100003, 7)])
def test_either_side_of_the_rule(ndof, n, k):
    rng = np.random.default_rng(ndof)
    x = rng.uniform(-3, 3, (n, ndof)).astype(np.float32)
    x[:700] = rng.normal(0, 0.02, (700, ndof))           # a dense spot
    x[700:760] = x[5]                                    # ties
    x[800, 0], x[801, -1], x[802, 0] = np.nan, np.inf, -np.inf
    x[900] = 9.0                                         # far from all others
    sample = np.concatenate([[5, 700, 759, 800, 801, 802, 900], rng.choice(n, 40, replace=False)])
    same(x, k, sample)
