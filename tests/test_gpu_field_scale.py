"""The two columns of F each keep their own precision where a layout's columns differ in scale (a strip, a layout off the
origin), although x W and y W share a transform: a strip's or an offset layout's F, column by column, against FP64 on
the same spectra, and the step that the device loop takes from it.

Tolerance: column c of F is the difference of |y_c| phi_1 and the potential of the charge y_c, so its error is bounded on
the scale of these two alone, 8 log2(M) 2^-24 of their norm as for any spectrum of one field (four passes, spread and
gather); the shared transform adds the other column's rounding, at most 1.42 times as large after the scaling, which
leaves the bound at less than twice that. Unscaled, the narrow column of a 1:100 strip is 20 times further off."""
import numpy as np
import pytest
import scipy.fft as sfft
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu
WIDTH = 0.7


def problem(mg, Y, nb, ni):
    """F and the kernel's sum on the device, F in 64 bits, and the bound of each column's error"""
    n, N, M = len(Y), nb * ni, sfft.next_fast_len(2 * nb * ni, real=True)
    o = np.minimum(np.arange(M), M - np.arange(M)) * (WIDTH / ni)
    b = 1 + o[:, None] ** 2 + o[None] ** 2
    K1, K2 = (np.fft.rfft2(k).real.astype(np.float32) for k in (1 / b, 1 / b ** 2))
    x0, y0 = (float(np.float32(Y[:, c].min().astype(np.float64) - 1e-3)) for c in (0, 1))
    conv = mg.FFTConv2D(M, ni)
    conv.set_kernels(K1, K2)
    sq, F = conv.compute(Y, x0, y0, WIDTH, nb)
    W = np.empty((3, N, N))
    O.lib().orc_spread(Y.ctypes.data, n, x0, y0, WIDTH, nb, ni, W.ctypes.data)
    Wh = np.fft.rfft2(W, s=(M, M), axes=(1, 2))
    phi = np.empty((4, N, N))
    phi[0] = np.fft.irfft2(K1.astype(np.float64) * Wh[0], s=(M, M))[:N, :N]
    phi[1:] = np.fft.irfft2(K2.astype(np.float64)[None] * Wh, s=(M, M), axes=(1, 2))[:, :N, :N]
    F64 = np.empty((n, 2))
    O.lib().orc_gather(Y.ctypes.data, n, x0, y0, WIDTH, nb, ni, phi.ctypes.data, F64.ctypes.data)
    rms = [np.sqrt(np.mean(p ** 2)) for p in phi]
    bound = [16 * np.log2(M) * 2.0 ** -24 * np.sqrt(n) * np.hypot(np.abs(Y[:, c]).max() * rms[1], rms[2 + c]) for c in (0, 1)]
    return sq, F, F64, bound


# boxes, nodes, extents, offsets; the last three: no scale to speak of, and columns of zeros (F is 0 there)
@pytest.mark.parametrize("nb,ni,extent,offset", [(100, 3, (1, 0.01), (0, 0)), (100, 3, (0.01, 1), (0, 0)),
                                                  (60, 3, (1, 0.2), (0, 0)), (60, 3, (1, 0.7), (0, 0)),
                                                  (61, 5, (1, 1), (1000, 0)), (61, 5, (1, 1), (0, -1000)),
                                                  (31, 2, (1, 1e-25), (0, 0)), (31, 2, (1, 0), (0, 0)),
                                                  (31, 2, (0, 1), (0, 0))])
def test_columns_of_unequal_scale(mg, nb, ni, extent, offset):
    rng = np.random.default_rng(nb)
    n = 20000
    r, t = np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n)
    half = 0.49 * nb * WIDTH
    Y = (np.stack([r * np.cos(t), r * np.sin(t)], 1) * half * extent + offset).astype(np.float32)
    _, F, F64, bound = problem(mg, Y, nb, ni)
    for c in (0, 1):
        assert np.linalg.norm(F[:, c] - F64[:, c]) <= bound[c], c


@pytest.mark.parametrize("batch", [False, True])
def test_a_strip_in_the_loop(mg, batch):
    """one iteration of rate 2000 from a 1:100 strip against the plain calls' step with F in 64 bits: the forces' bound, times
    the rate and the largest gain 1.2 over the kernel's sum, and four roundings of a position"""
    rng = np.random.default_rng(3)
    n, lr = 3000, 2000.0
    Y = (rng.uniform(-1, 1, (n, 2)) * (30, 0.3)).astype(np.float32)
    i = np.arange(n)
    P = sp.coo_matrix((np.ones(2 * n, np.float32), (np.r_[i, i], np.r_[(i + 1) % n, (i - 1) % n]))).tocsr()
    P = (P / P.sum()).tocsr().astype(np.float32)
    span = (Y.max(0).astype(np.float64) - Y.min(0).astype(np.float64) + 2e-3).max()
    nb = (int(np.ceil(span / WIDTH)) + 3) // 4 * 4
    sq, _, F64, bound = problem(mg, Y, nb, 3)
    A = mg.tsne_attraction(P.indptr, P.indices, P.data, Y, 1.0)
    Z, U, G = Y.copy(), np.zeros_like(Y), np.ones_like(Y)
    mg.tsne_step(Z, U, G, A, F64.astype(np.float32), 1.0, 1.0 / sq, lr, 0.5)
    kw = dict(n_iter=1, early_iter=0, learning_rate=lr)
    if batch:
        L = mg.optimize_tsne_batch([P, P], [Y.copy(), Y.copy()], threads_per_row=2, branches=1, **kw)[1]
    else:
        L = mg.optimize_tsne(P, Y.copy(), **kw)
    for c in (0, 1):
        slack = 1.2 * lr / sq * bound[c] + 4 * np.sqrt(n) * np.spacing(np.abs(Y[:, c]).max())
        assert np.linalg.norm(L[:, c] - Z[:, c]) <= slack, c
