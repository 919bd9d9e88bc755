"""Owner mode's grid barriers and work that keeps them waiting: how long the others wait for a thread has no bound of its own,
so a wait ends only where nothing moves any more, and a run that gave up is reported by the call that reads its layout."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_a_long_replay_is_waited_for(mg):
    """8,000 edges are one chunk of the reference's; a distance-0 negative makes one thread replay it, 16 million draws one after
    another (some seconds), while the other blocks wait. +, *, / and sqrt only: equal to the oracle bit for bit."""
    rng = np.random.default_rng(0)
    n, rate = 8000, 2000.0
    head = np.arange(n, dtype=np.int32)
    tail = ((head + rng.integers(1, n, n)) % n).astype(np.int32)
    eps = np.ones(n, np.float32)
    Y = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    Y[:50] = Y[50:100]
    Yo, Yd = Y.copy(), Y.copy()
    eo, eno = eps.copy(), (eps / rate).astype(np.float32)
    ed, end = eo.copy(), eno.copy()
    O.sgd_owner(Yo, head, tail, eps, eo, eno, a=1.7, b=1.0, rep_a=1.7, rep_b=1.0, negative_sample_rate=rate, epoch_start=0,
                epoch_end=2, alpha0=1.0, alpha1=0.3, mid_w0=0.0, mid_w1=0.0, clip_mode=0, n_fixed=0, seed=11)
    z, z2 = np.zeros(0, np.int32), np.zeros((0, 2), np.float32)
    mg.optimize_layout(Yd, head, tail, eps, ed, end, z, z, 0, 2, 1.0, 0.3, 0.0, 0.0, 1.7, 1.0, 1.7, 1.0, rate, 0, 1.0, 2.0, 4,
                       0.25, 0, 0, 0, z2, z2, z, 0.9, 0.999, z, z.reshape(0, 1), z, z, 0.0, 0, np.zeros(0, np.float32), 11,
                       -1, 1)
    assert np.array_equal(Yd, Yo), np.abs(Yd - Yo).max()


def test_transform_reports_a_run_that_gave_up(mg, cuda, monkeypatch):
    """the library's answer is a stand-in's; the request raises it instead of returning positions"""
    from magnet_b200 import serve as S
    rng = np.random.default_rng(1)
    X, Y = rng.normal(size=(300, 4)).astype(np.float32), rng.normal(size=(300, 2)).astype(np.float32)
    layout = S.FittedLayout(X, Y, a=1.577, b=0.895, transform_epochs=5)
    assert np.isfinite(layout.transform(X[:7] + 0.01)).all()
    real = S._lib()

    class GaveUp:
        def __getattr__(self, name):
            return getattr(real, name)

        def mg_synchronize(self):
            return 4

        def mg_last_error(self):
            return ctypes.c_char_p(b"a grid barrier gave up").value

    monkeypatch.setattr(S, "_lib", lambda: GaveUp())
    with pytest.raises(RuntimeError, match="gave up"):
        layout.transform(X[:7] + 0.01)
