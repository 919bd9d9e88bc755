"""The profiled loop reports the grid that its last iteration ran on, not the one that iteration's step chose for the next: one
iteration from a layout of known extent, at a rate that doubles the extent and more."""
import numpy as np
import pytest
import scipy.fft as sfft
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span", [10.0, 40.0])
def test_grid_of_the_last_iteration(mg, span):
    n = 2000
    Y0 = np.random.default_rng(1).uniform(0, span, (n, 2)).astype(np.float32)
    i = np.arange(n)
    P = sp.coo_matrix((np.ones(2 * n, np.float32), (np.r_[i, i], np.r_[(i + 1) % n, (i - 1) % n]))).tocsr()
    Y = Y0.copy()
    d = mg._native.optimize_tsne_profiled(P.indptr.astype(np.int32), P.indices.astype(np.int32), P.data, Y, 1, 0, 12.0, 1.0,
                                          1e6, 3, 0.7, 1.0)
    extent = lambda Z: (Z.max(0).astype(np.float64) - Z.min(0).astype(np.float64)).max() + 2e-3
    assert extent(Y) > 2 * extent(Y0)
    nb = (max(20, int(np.ceil(extent(Y0) / 0.7))) + 3) // 4 * 4
    M = sfft.next_fast_len(6 * nb, real=True)
    assert d["grid"][:2] == (nb, 3 * nb) and d["grid"][2] >= M and d["grid"][3] == d["grid"][2] // 2 + 1
