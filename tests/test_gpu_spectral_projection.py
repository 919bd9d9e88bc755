"""The spectral solver's deflation where the trivial eigenvector's weights are no eigenvector of the operator: scale factors that
are not the graph's own degrees, a directed graph, and component labels that edges cross. The oracle projects M Y itself
at every product, in FP64. Few filter steps and no stopping rule; the wanted vectors span the same subspace (float32
output: sine below 1e-5) with the same Ritz values. The solver that projected with the sums of the block before the
product was 1e-3 to 0.99 off on all but the directed one (shown in numpy)."""
import os
import sys

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from spectral_cases import inputs, ritz_values, subspace_sine, three_components  # noqa: E402

pytestmark = pytest.mark.gpu


def path_with_chords(n):
    rng = np.random.default_rng(n)
    i, a, b = np.arange(n - 1), rng.integers(0, n, n // 3), rng.integers(0, n, n // 3)
    A = sp.coo_matrix((0.2 + rng.random(n - 1 + n // 3), (np.r_[i, a], np.r_[i + 1, b])), shape=(n, n))
    A = (A + A.T).tocsr()
    A.setdiag(0)
    A.eliminate_zeros()
    return A.astype(np.float32)


@pytest.mark.parametrize("p,degree,iters", [(4, 6, 2), (4, 30, 3), (3, 2, 1), (8, 7, 2)])
@pytest.mark.parametrize("kind", ["plain", "three", "directed", "other_degrees", "labels_in_turn", "labels_in_blocks"])
def test_projection_of_the_product(mg, kind, p, degree, iters):
    from magnet_b200 import _native as N
    P = three_components() if kind == "three" else path_with_chords(900)
    n = P.shape[0]
    rng = np.random.default_rng(0)
    if kind == "directed":
        P.data = (P.data * rng.uniform(0.3, 1.7, P.nnz)).astype(np.float32)
    a = list(inputs(P, 2, seed=1))
    if kind == "other_degrees":
        a[4] = (a[4] * rng.uniform(0.7, 1.0, n)).astype(np.float32)
    if kind == "labels_in_turn":
        a[5] = (np.arange(n) % 3).astype(np.int32)
    if kind == "labels_in_blocks":
        a[5] = (np.arange(n) // 300).astype(np.int32)
    a[3] = rng.standard_normal((n, p)).astype(np.float32)
    a[6], a[7], a[8], a[9] = min(2, p - 1), degree, iters, 0.0
    got = np.asarray(N.chebyshev_eigenvectors(*a[:3], a[3].copy(), *a[4:], -1))
    want = O.chebyshev_eigenvectors(*a[:3], a[3].copy(), *a[4:])
    assert np.isfinite(got).all()
    assert subspace_sine(got[:, :a[6]], want[:, :a[6]]) < 1e-5
    vg, vw = (ritz_values(sp.csr_matrix(P), a[4], Z[:, :a[6]]) for Z in (got, want))
    assert np.allclose(vg, vw, rtol=0, atol=1e-6), (vg, vw)
