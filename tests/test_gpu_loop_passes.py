"""The grid passes at the lengths and rows where their packing and tiling change, and the launches that cover many
layouts against the loop of one.

Spectra: any real half spectrum is accepted by set_kernels, so the values here are random (they are not even in k2, which
tells apart the columns read mirrored, averaged and plain). Tolerance against the FP64 restatement: a single-precision
transform's relative RMS error is below log2(M) 2^-24 per pass; four passes, the spread and the gather (each a few
roundings) stay below 8 log2(M) 2^-24 of the norm of the two terms whose difference F is.
Batch: two single-precision runs differ in the order of the spread's atomics, about 1e-5 of the gradient's two terms,
which may cancel to a tenth: 1e-3 of the step over both iterations."""
import numpy as np
import pytest
import scipy.fft as sfft
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def restated(Y, xmin, ymin, width, nb, ni, M, K1h, K2h):
    n, N = len(Y), nb * ni
    W = np.empty((3, N, N), np.float64)
    O.lib().orc_spread(Y.ctypes.data, n, xmin, ymin, width, nb, ni, W.ctypes.data)
    Wh = np.fft.rfft2(W, s=(M, M), axes=(1, 2))
    phi = np.empty((4, N, N), np.float64)
    phi[0] = np.fft.irfft2(K1h * Wh[0], s=(M, M))[:N, :N]
    phi[1:] = np.fft.irfft2(K2h[None] * Wh, s=(M, M), axes=(1, 2))[:, :N, :N]
    phi = np.ascontiguousarray(phi)
    F = np.empty((n, 2), np.float64)
    sumQ = O.lib().orc_gather(Y.ctypes.data, n, xmin, ymin, width, nb, ni, phi.ctypes.data, F.ctypes.data)
    # the size of the two terms of F: |y| phi_2 and the potentials of x W, y W
    rms = [np.sqrt(np.mean(phi[q] ** 2)) for q in range(4)]
    scale = np.sqrt(n) * np.hypot(np.abs(Y).max() * rms[1], max(rms[2], rms[3]))
    return float(sumQ), F, scale


# (boxes, nodes): M = 4, 15 (odd), 24, 30 (odd rows), 45, 125, 270, 450, 729 (odd), 1536 and 1600 (either block size), 2400
@pytest.mark.parametrize("nb,ni", [(2, 1), (7, 1), (4, 3), (5, 3), (11, 2), (31, 2), (27, 5), (75, 3), (91, 4), (256, 3),
                                   (200, 4), (400, 3)])
def test_any_real_spectrum(mg, nb, ni):
    rng = np.random.default_rng(100 * nb + ni)
    width = 0.7
    M = sfft.next_fast_len(2 * nb * ni, real=True)
    K1, K2 = (rng.uniform(0.5, 1.5, (M, M // 2 + 1)).astype(np.float32) for _ in range(2))
    Y = rng.uniform(0.01, nb * width - 0.01, (max(200, 20 * nb), 2)).astype(np.float32)
    conv = mg.FFTConv2D(M, ni)
    conv.set_kernels(K1, K2)
    sq, F = conv.compute(Y, 0.0, 0.0, width, nb)
    sq64, F64, scale = restated(Y, 0.0, 0.0, width, nb, ni, M, K1.astype(np.float64), K2.astype(np.float64))
    tol = 8 * np.log2(M) * 2.0 ** -24
    assert abs(sq - sq64) <= tol * (abs(sq64) + len(Y))
    assert np.linalg.norm(F - F64) <= tol * scale


# one set, two sets, and more layouts than points per side differ; rows of 1 to 40 edges run different lane counts
@pytest.mark.parametrize("count,branches,ni", [(1, 1, 3), (3, 1, 3), (37, 2, 3), (37, 8, 4)])
def test_many_layouts_in_a_launch(mg, count, branches, ni):
    rng = np.random.default_rng(count)
    Ps, Ys = [], []
    for i in range(count):
        n = int(rng.integers(2, 60)) if i % 3 == 0 else int(rng.integers(60, 1500))
        k = min(n - 1, int(rng.integers(1, 40)))
        A = sp.random(n, n, density=min(1.0, k / n), format="csr", random_state=i, dtype=np.float32)
        A = A + A.T + sp.csr_matrix((np.ones(n, np.float32), (np.arange(n), (np.arange(n) + 1) % n)), shape=(n, n))
        A = (A + A.T).tocsr()
        A.setdiag(0); A.eliminate_zeros(); A.sort_indices()
        A = (A / A.sum()).tocsr().astype(np.float32)
        Ps.append(A)
        Ys.append((rng.uniform(-1, 1, (n, 2)) * 0.4 * np.sqrt(n)).astype(np.float32))
    out = mg.optimize_tsne_batch(Ps, [Y.copy() for Y in Ys], n_iter=2, early_iter=1, learning_rate=1.0, n_interp=ni,
                                 threads_per_row=8, branches=branches)
    for P, Y0, Yb in zip(Ps, Ys, out):
        Y1 = mg.optimize_tsne(P, Y0.copy(), n_iter=2, early_iter=1, learning_rate=1.0, n_interp=ni, threads_per_row=8)
        C = Y0 - Y0.mean(0)
        assert np.linalg.norm(Yb - Y1) <= 1e-3 * np.linalg.norm(Y1 - C) + 1e-6 * np.linalg.norm(C)
