"""The counter mode's sample lists: epochs over more than one counting window, runs of one and of several words, edge counts
that end inside a word, edges that lag behind the epoch or are sampled in every one of them, layouts with fewer samples
than threads.

The bookkeeping (eons / eonns) equals the oracle's bit for bit. The layout: at a step size so small that positions stay
where they are to first order, the displacement is the sum of every sample's steps at the starting positions, whatever
their order. With steps of 3e-5 |g| on coordinates up to 2, a step's rounding is below 1 % of it (6e-8 / 1e-5) and averages
out, and the positions move by less than 1 % of the distances: 2 % of the displacement's norm."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
ALPHA, A, B, REP_A, RATE, GAMMA = 3e-5, 1.7, 0.8, 1.74, 5.0, 1.0


def problem(n, k, dim, seed):
    rng = np.random.default_rng(seed)
    head = np.sort(rng.integers(0, n, n * k)).astype(np.int32)
    tail = ((head + rng.integers(1, n, n * k)) % n).astype(np.int32)
    E = len(head)
    eps = rng.uniform(1.0, 12.0, E).astype(np.float32)
    eps[rng.random(E) < 0.02] = 0.4                      # every epoch, falling behind
    eons = (7 + eps * rng.random(E)).astype(np.float32)
    eons[rng.random(E) < 0.05] = -3.0                    # lagging at the start
    eons[rng.random(E) < 0.05] = 1e6                     # never
    eonns = (7 - rng.random(E)).astype(np.float32)
    return rng.uniform(0, 2, (n, dim)).astype(np.float32), head, tail, eps, eons, eonns


# (n, k, dim): one word, a ragged word, one-word runs, two-word runs; fewer samples than threads
@pytest.mark.parametrize("n,k,dim", [(3, 1, 2), (301, 5, 2), (301, 5, 3), (5000, 12, 2), (20011, 17, 2)])
def test_lists_against_oracle(mg, n, k, dim):
    Y0, head, tail, eps, eons, eonns = problem(n, k, dim, n + dim)
    e0, e1 = 7, 7 + (45 if n < 10000 else 36)
    z, zf = np.zeros(0, np.int32), np.zeros((0, dim), np.float32)
    Y, ed, nd = Y0.copy(), eons.copy(), eonns.copy()
    mg.optimize_layout(Y, head, tail, eps, ed, nd, z, z, e0, e1, ALPHA, ALPHA, 0.0, 0.0, A, B, REP_A, 1.0, RATE, 0, 1.0,
                       GAMMA, 4, 0.25, 0, 0, 0, zf, zf, z, 0.9, 0.999, z, np.zeros((0, 1), np.int32), z, z, 0.0, 0,
                       np.zeros(0, np.float32), 99, 1, 0, None, None, 0)
    eo, no, D, P = eons.copy(), eonns.copy(), np.zeros((n, dim)), Y0.astype(np.float64)
    for e in range(e0, e1):
        smp, nn, off, negs, _ = O.sgd_schedule(Y0.copy(), head, tail, eps, eo, no, e, per_edge_stream=True, a=A, b=B,
                                               rep_a=REP_A, negative_sample_rate=RATE, seed=99, epoch_start=e0,
                                               epoch_end=e1, alpha0=ALPHA, alpha1=ALPHA, negs_cap=60 * len(head) + 64)
        i = np.flatnonzero(smp)
        if not len(i):
            continue
        u, v = head[i], tail[i]
        d = P[u] - P[v]
        d2 = (d * d).sum(1)[:, None]
        pw = d2 ** B
        g = -2 * A * B * pw / (d2 * (A * pw + 1)) * d
        gu = g.copy()
        np.add.at(D, v, np.clip(-g, -4, 4))
        row = np.repeat(np.arange(len(i)), nn[i])
        kk = np.concatenate([negs[off[j]:off[j] + nn[j]] for j in i]) if nn[i].sum() else np.zeros(0, np.int32)
        d = P[u[row]] - P[kk]
        d2 = (d * d).sum(1)[:, None]
        g = np.where(kk[:, None] == u[row][:, None], 0.0, 2 * GAMMA / ((0.001 + d2) * (REP_A * d2 + 1)) * d)
        np.add.at(gu, row, g)
        np.add.at(D, u, np.clip(gu, -4, 4))
    assert np.array_equal(ed, eo) and np.array_equal(nd, no)
    D *= ALPHA
    assert np.linalg.norm((Y - P) - D) <= 0.02 * np.linalg.norm(D)
