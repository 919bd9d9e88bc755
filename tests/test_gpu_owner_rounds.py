"""Owner mode's pipelined node pass at the ends of its rounds: rows listed 32 edges at a time (rows of 31 to 70 edges, 32, 33 and
64 among them), rounds of 48 positions, an edge of more negatives than a round holds (drawn while it is computed) beside
ordinary ones in the same row, and the groups of a warp ending their rows after different numbers of rounds. Node counts
at which a head has 8, 4, 2 and 1 lanes. Power kernel at b = rep_b = 1 under plain steps: +, *, / and sqrt only, so the
layout, eons and eonns equal the oracle's owner run bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

#         row lengths, lengths that are there, negative rate, positions shared
KINDS = {
    "refill": ((31, 71), (32, 33, 64), 5.0, False),
    "wide": ((1, 24), (0, 1, 23), 45.0, False),       # 43 to 90 negatives an edge: about half the edges past a round
    "very_wide": ((1, 12), (0, 11), 160.0, False),    # every edge past a round
    "wide_replayed": ((1, 40), (32, 33), 45.0, True),
}


@pytest.mark.parametrize("n", [90, 2368, 2369, 4737, 9473])
@pytest.mark.parametrize("kind", KINDS)
def test_rounds_equal_the_oracle(mg, kind, n):
    (lo, hi), there, rate, shared = KINDS[kind]
    rng = np.random.default_rng(n + len(kind))
    length = rng.integers(lo, hi, n)
    length[:len(there)] = there
    head = np.repeat(np.arange(n, dtype=np.int32), length)
    tail = ((head + rng.integers(1, n, head.size)) % n).astype(np.int32)
    eps = rng.uniform(1.0, 3.0, head.size).astype(np.float32)
    Y = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    if shared:
        Y[: n // 8] = Y[n // 8: 2 * (n // 8)]
    Yo, Yd = Y.copy(), Y.copy()
    eo, eno = eps.copy(), (eps / rate).astype(np.float32)
    ed, end = eo.copy(), eno.copy()
    kw = dict(a=1.7, b=1.0, rep_a=1.7, rep_b=1.0, negative_sample_rate=rate, epoch_start=0, epoch_end=5, alpha0=1.0, alpha1=0.3,
              mid_w0=0.0, mid_w1=0.0, clip_mode=0, n_fixed=0, seed=11)
    O.sgd_owner(Yo, head, tail, eps, eo, eno, **kw)
    z, z2 = np.zeros(0, np.int32), np.zeros((0, 2), np.float32)
    mg.optimize_layout(Yd, head, tail, eps, ed, end, z, z, 0, 5, 1.0, 0.3, 0.0, 0.0, 1.7, 1.0, 1.7, 1.0, rate, 0, 1.0, 2.0, 4,
                       0.25, 0, 0, 0, z2, z2, z, 0.9, 0.999, z, z.reshape(0, 1), z, z, 0.0, 0, np.zeros(0, np.float32), 11,
                       -1, 1)
    assert np.array_equal(ed, eo) and np.array_equal(end, eno)
    assert np.array_equal(Yd, Yo), np.abs(Yd - Yo).max()
