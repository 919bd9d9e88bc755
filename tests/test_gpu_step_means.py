"""tsne_step / tsne_update with the column means taken in the same pass: rows that end inside a block, a block of rows
exactly, several blocks, and dimensions that do and do not divide the block. The update itself is the reference's single
precision arithmetic (src/fftrep.cpp:245-253), so the only difference allowed is one rounding of the mean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2, 3, 7, 64])
@pytest.mark.parametrize("n", [1, 85, 128, 257, 40001])
def test_step_and_means(mg, n, dim):
    rng = np.random.default_rng(n * 100 + dim)
    f32 = np.float32
    Y, U, A, F = (rng.normal(0, 3, (n, dim)).astype(f32) for _ in range(4))
    G = rng.uniform(0.005, 2, (n, dim)).astype(f32)
    rho, inv, lr, mom = f32(1.5), f32(0.25), f32(2.0), f32(0.8)
    for fused in (True, False):
        y, u, g = Y.copy(), U.copy(), G.copy()
        grad = rho * A - F * inv if fused else A
        if fused:
            mg.tsne_step(y, u, g, A, F, float(rho), float(inv), float(lr), float(mom))
        else:
            mg.tsne_update(y, u, g, A, float(lr), float(mom))
        gain = np.where((grad > 0) == (U > 0), G * f32(0.8), G + f32(0.2)).astype(f32)
        gain = np.maximum(gain, f32(0.01))
        un = mom * U - lr * gain * grad
        yn = Y + un
        mean = (yn.astype(np.float64).sum(0) / n).astype(f32)
        assert np.array_equal(g, gain) and np.array_equal(u, un)
        assert np.all(np.abs(y - (yn - mean)) <= 2.0 ** -22 * (np.abs(mean) + np.abs(yn)))
