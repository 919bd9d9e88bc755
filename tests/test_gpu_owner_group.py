"""Owner mode's batched epochs (schedule and draws made ahead, eight lanes per head, one launch for many epochs) against
the oracle's owner run. Power kernel at b = rep_b = 1 under plain steps: +, *, / and sqrt only, so the layout, eons and
eonns are equal bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

#        nodes, fixed, row lengths, epochs, negative rate, norm clip, duplicate positions, mid-range phase
CASES = {
    "one_row": (40, 39, (5, 5), 3, 5.0, 0, False, False),
    "short_rows": (700, 0, (0, 8), 4, 5.0, 0, False, False),
    "window_edges": (600, 100, (7, 18), 5, 5.0, 1, False, False),      # rows of 7 to 17 edges around windows of 8
    "many_negatives": (500, 0, (6, 20), 4, 20.0, 0, False, False),     # over 8 negatives per edge
    "transform": (5000, 4400, (14, 15), 21, 5.0, 0, False, False),     # edges of the new rows only, 2 chunks
    "replayed": (900, 0, (9, 12), 5, 5.0, 0, True, False),             # distance-0 negatives: chunks replayed
    "phases": (800, 0, (6, 14), 9, 5.0, 0, False, True),               # mid-range pulls fade out inside the call
}


@pytest.mark.parametrize("name", CASES)
def test_owner_batches_equal_the_oracle(mg, name):
    n, fixed, (lo, hi), epochs, rate, clip, dup, mid = CASES[name]
    rng = np.random.default_rng(len(name))
    length = np.zeros(n, np.int64)
    first = fixed if name in ("transform", "one_row") else 0
    length[first:] = rng.integers(lo, max(hi, lo + 1), n - first)
    head = np.repeat(np.arange(n, dtype=np.int32), length)
    tail = rng.integers(0, n, head.size).astype(np.int32)
    tail = np.where(tail == head, (tail + 1) % n, tail).astype(np.int32)
    eps = rng.uniform(1.0, 3.0, head.size).astype(np.float32)
    Y = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    if dup:
        Y = Y[np.arange(n) % 16].copy()
    pairs = rng.integers(0, n, (n, 3)).astype(np.int32)
    Yo, Yd = Y.copy(), Y.copy()
    eo, eno = eps.copy(), (eps / rate).astype(np.float32)
    ed, end = eo.copy(), eno.copy()
    mw = (0.2, -0.1) if mid else (0.0, 0.0)
    kw = dict(a=1.7, b=1.0, rep_a=1.7, rep_b=1.0, negative_sample_rate=rate, epoch_start=0, epoch_end=epochs, alpha0=1.0,
              alpha1=0.3, mid_w0=mw[0], mid_w1=mw[1], clip_mode=clip, n_fixed=fixed, seed=9)
    if mid:
        kw.update(mid_pairs=pairs)
    O.sgd_owner(Yo, head, tail, eps, eo, eno, **kw)
    z, z2 = np.zeros(0, np.int32), np.zeros((0, 2), np.float32)
    mg.optimize_layout(Yd, head, tail, eps, ed, end, z, z, 0, epochs, 1.0, 0.3, mw[0], mw[1], 1.7, 1.0, 1.7, 1.0, rate, 0,
                       1.0, 2.0, 4, 0.25, 0, clip, fixed, z2, z2, z, 0.9, 0.999, z, pairs if mid else z.reshape(0, 1), z, z,
                       0.0, 0, np.zeros(0, np.float32), 9, -1, 1)
    assert np.array_equal(ed, eo) and np.array_equal(end, eno)
    assert np.array_equal(Yd, Yo), np.abs(Yd - Yo).max()
