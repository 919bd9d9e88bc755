"""The fuzzy union's row forms against the oracle's union, bit for bit: neighbour rows of up to 16, 32 and more entries
(lanes per row, or a thread), union rows of up to 32, 64, 128, 256, 512 and more entries (registers per lane, or a
thread's merge), duplicate neighbours, zero memberships, empty rows past the kNN rows, a mix that drops one-way entries."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows,n,k,hubs,mix", [(5, 5, 1, 0, 1.0), (300, 300, 7, 0, 1.0), (900, 901, 16, 3, 0.5),
                                                 (1200, 1200, 17, 5, 1.0), (1500, 1500, 32, 40, 1.0), (700, 800, 33, 20, 1.0),
                                                 (2500, 2500, 90, 8, 0.3), (1300, 1300, 260, 30, 1.0), (600, 600, 14, 2, 0.0)])
def test_union_rows(mg, n_rows, n, k, hubs, mix):
    from magnet_b200 import _native
    rng = np.random.default_rng(k)
    ind = rng.integers(0, n, (n_rows, k)).astype(np.int32)
    # hub columns that most rows choose, some of them twice
    for h in range(hubs):
        rows = rng.choice(n_rows, n_rows * (h + 1) // (hubs + 1), replace=False)
        ind[rows, rng.integers(0, k, rows.size)] = h % n
    if k > 2:
        ind[::7, 1] = ind[::7, 0]
    vals = rng.random((n_rows, k)).astype(np.float32)
    vals[rng.random(vals.shape) < 0.05] = 0.0
    ip, ix, dd = _native.fuzzy_union(ind, vals, n, mix)
    op, ox, od = O.fuzzy_union(ind, vals, n, mix)
    assert np.array_equal(ip, op) and np.array_equal(ix, ox) and np.array_equal(dd, od)
