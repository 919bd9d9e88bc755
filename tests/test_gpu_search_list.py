"""knn_search on the device against a plain restatement of the beam search (two heaps, src/nndescent.cpp:585-690) on
small integer coordinates, where every squared distance is exact in any evaluation order: the same rows and distances.
Widths around the 16-float blocks and 4-float reads, lists of 1 to 8 registers, more entries than a lane keeps, repeated
landmarks, rows longer than a warp. Equal distances may be expanded in another order, so 99 % of the queries must agree
in their rows (distances in all of those)."""
import heapq

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def beam(X, gptr, gidx, land, q, k, ef, n_entry):
    d2 = ((X - q) ** 2).sum(1)
    seen, res, cand = set(), [], []

    def consider(j):
        if j in seen:
            return
        seen.add(j)
        if len(res) < ef or d2[j] < -res[0][0]:
            heapq.heappush(res, (-d2[j], -j))
            if len(res) > ef:
                heapq.heappop(res)
            heapq.heappush(cand, (d2[j], j))

    for _, j in sorted({(d2[j], j) for j in land})[:n_entry]:
        consider(j)
    while cand:
        d, c = heapq.heappop(cand)
        if len(res) >= ef and d > -res[0][0]:
            break
        for j in gidx[gptr[c]:gptr[c + 1]]:
            consider(int(j))
    out = sorted((-a, -b) for a, b in res)[:k]
    return [j for _, j in out], [d for d, _ in out]


@pytest.mark.parametrize("d,k,ef,n_entry,degree", [(64, 14, 64, 5, 25), (50, 14, 64, 5, 25), (16, 5, 33, 5, 40), (7, 3, 3, 9, 12),
                                                   (100, 10, 100, 12, 25), (33, 20, 200, 3, 70), (784, 10, 40, 5, 20)])
def test_search_equals_two_heaps(mg, d, k, ef, n_entry, degree):
    rng = np.random.default_rng(d)
    n, m = 2500, 60
    lim = 40 if d <= 100 else 12
    centres = rng.integers(-lim // 2, lim // 2, (12, d))
    draw = lambda c: (centres[rng.integers(0, 12, c)] + rng.integers(-lim // 2, lim // 2, (c, d)))
    X, Q = draw(n), draw(m)
    # a neighbour graph: each row's closest among a random third, both directions
    nb = np.empty((n, degree), np.int64)
    for i in range(n):
        pool = np.setdiff1d(rng.choice(n, n // 3, replace=False), [i])
        nb[i] = pool[np.argsort(((X[pool] - X[i]) ** 2).sum(1), kind="stable")[:degree]]
    gptr = (np.arange(n + 1) * degree).astype(np.int32)
    gidx = nb.ravel().astype(np.int32)
    land = rng.choice(n, 150).astype(np.int32)
    land[:10] = land[10:20]
    gi, gd = mg._native.knn_search(X.astype(np.float32), gptr, gidx, land, Q.astype(np.float32), k, ef, n_entry, 0, -1)
    same = 0
    for r in range(m):
        wi, wd = beam(X, gptr, gidx, land.tolist(), Q[r], k, ef, n_entry)
        wi += [-1] * (k - len(wi))
        wd += [np.inf] * (k - len(wd))
        if np.array_equal(gi[r], wi):
            same += 1
            assert np.array_equal(gd[r], np.array(wd, np.float32))
    assert same >= 0.99 * m, (same, m)
