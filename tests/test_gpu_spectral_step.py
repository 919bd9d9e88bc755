"""The spectral solver's one-launch filter steps and Cholesky orthonormalisation against the oracle's numpy solver on the
same graph and start block, both in FP64: the wanted vectors span the same subspace (float32 output: sine below 1e-5) with
the same Ritz values. Blocks of 2 to 8 columns (2, 4 and 8 lanes per row), fewer rows than a block, a row longer than
the others by far, several components with isolated nodes, a start block of nearly equal columns (1e-6 apart: the column-by-column path;
the directions left hold 10 of FP64's digits, well inside the same bound)."""
import os
import sys

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from spectral_cases import inputs, ritz_values, subspace_sine, three_components  # noqa: E402

pytestmark = pytest.mark.gpu


def ring(n, hub):
    """a path with random chords, its first node joined to `hub` others"""
    rng = np.random.default_rng(n)
    i = np.arange(n - 1)
    a, b = rng.integers(0, n, n // 3), rng.integers(0, n, n // 3)
    r = np.concatenate([i, a, np.zeros(hub, np.int64)])
    c = np.concatenate([i + 1, b, rng.choice(np.arange(1, n), hub, replace=False)])
    A = sp.coo_matrix((0.2 + rng.random(r.size), (r, c)), shape=(n, n))
    A = (A + A.T).tocsr()
    A.setdiag(0)
    A.eliminate_zeros()
    return A.astype(np.float32)


@pytest.mark.parametrize("graph,p,wanted,near", [("ring10", 3, 1, False), ("ring257", 2, 1, False), ("ring257", 5, 2, False),
                                                  ("ring3000", 4, 2, False), ("ring3000", 6, 3, False), ("ring3000", 8, 4, False),
                                                  ("three", 4, 2, False), ("three", 7, 3, False), ("ring3000", 4, 2, True)])
def test_solver_equals_the_oracle(mg, graph, p, wanted, near):
    from magnet_b200 import _native as N
    P = three_components() if graph == "three" else ring(int(graph[4:]), min(600, int(graph[4:]) // 4))
    a = list(inputs(P, 2, seed=p))
    X = np.random.default_rng(p).standard_normal((P.shape[0], p)).astype(np.float32)
    if near:
        X[:, 1:] = X[:, :1] + 1e-6 * X[:, 1:]
    a[3], a[6], a[8] = X, wanted, 3
    got = np.asarray(N.chebyshev_eigenvectors(*a[:3], X.copy(), *a[4:], -1))
    want = O.chebyshev_eigenvectors(*a[:3], X.copy(), *a[4:])
    assert np.isfinite(got).all()
    assert subspace_sine(got[:, :wanted], want[:, :wanted]) < 1e-5
    vg, vw = (ritz_values(sp.csr_matrix(P), a[4], Z[:, :wanted]) for Z in (got, want))
    assert np.allclose(vg, vw, rtol=0, atol=1e-9), (vg, vw)
