"""The neighbour grid where its cell counts meet the scan's passes of 4096:
one pass, one cell more or less, many.  Indices and distances equal the
oracle's whatever the cell size."""
import numpy as np
import pytest

import nbr_oracle as NO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndof,n", [(1, 1), (1, 33), (1, 5000), (2, 5000), (3, 3000)])
@pytest.mark.parametrize("cells", [1, 3, 31, 64, 4094, 4095, 4096, 4097, 8192, 20001])
def test_cell_counts(ndof, n, cells):
    import torch
    from gpuprm_b200.neighbours import NeighbourIndex
    per = max(1, round(cells ** (1.0 / ndof)))
    rng = np.random.default_rng(cells + ndof)
    x = rng.uniform(-2, 2, (n, ndof)).astype(np.float32)
    x[0] = -2
    x[-1] = 2
    ix = NeighbourIndex(ndof)
    ix.build(torch.tensor(np.ascontiguousarray(x.T), device="cuda:0"), cell=4.0 / per)
    k = 7
    idx, dist = ix.knn(k)
    torch.cuda.synchronize()
    sample = rng.choice(n, min(n, 60), replace=False)
    want_i, want_d = NO.knn(x, x[sample], k, exclude=sample)
    np.testing.assert_array_equal(idx.cpu().numpy()[sample], want_i)
    np.testing.assert_array_equal(dist.cpu().numpy()[sample], want_d)
