"""The sample pass of large layouts (one thread per walker), at sizes a test can hold: n / 1 walkers at 30,011 points (more walkers
than its eight-lane form takes: positions read as they are needed) and n / 8 at 232,003 (few enough walkers for their
points that positions are read a sample ahead). The displacement check of the sample lists: at a step size so small that
positions stay where they are to first order, the displacement is the sum of every sample's steps at the starting
positions. Steps of 3e-5 |g| on coordinates up to 2: a step's rounding is below 1 % of it (6e-8 / 1e-5) and averages out,
and the positions move by less than 1 % of the distances: 2 % of the displacement's norm. The bookkeeping equals the
oracle's bit for bit. A sample left out or taken twice at the walkers' ends (three per walker are under way) is 1 / 8 of
the samples of a walker or more, 5 % of the displacement at least."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
ALPHA, A, RATE, GAMMA = 3e-5, 1.7, 5.0, 1.0

#        n / walkers, n, edges a row, dim, b, rep_b, mid-range pairs, b of its own per node
CASES = {
    "plain": (1, 30011, 7, 2, 0.8, 1.0, False, False),
    "plain_b1": (1, 30011, 7, 2, 1.0, 1.0, False, False),
    "plain_rep": (1, 30011, 7, 2, 0.8, 0.9, True, False),
    "plain_3d": (1, 30011, 7, 3, 1.0, 0.9, False, False),
    "plain_node_b": (1, 30011, 7, 2, 0.8, 1.0, False, True),
    "ahead": (8, 232003, 4, 2, 0.8, 1.0, False, False),
    "ahead_b1": (8, 232003, 4, 2, 1.0, 1.0, True, False),
    "ahead_rep": (8, 232003, 4, 2, 1.0, 0.9, False, False),
    "ahead_3d": (8, 232003, 4, 3, 0.8, 0.9, False, False),
    "ahead_node_b": (8, 232003, 4, 3, 0.8, 1.0, True, True),
}


@pytest.mark.parametrize("name", CASES)
def test_thread_form_against_the_schedule(mg, monkeypatch, name):
    div, n, k, dim, b, rep_b, mid, own_b = CASES[name]
    monkeypatch.setenv("MGB_SGD_INFLIGHT_DIV", str(div))
    rng = np.random.default_rng(n + dim)
    head = np.sort(rng.integers(0, n, n * k)).astype(np.int32)
    tail = ((head + rng.integers(1, n, n * k)) % n).astype(np.int32)
    E = len(head)
    eps = rng.uniform(1.0, 6.0, E).astype(np.float32)
    eons = (3 + eps * rng.random(E)).astype(np.float32)
    eonns = (3 - rng.random(E)).astype(np.float32)
    Y0 = rng.uniform(0, 2, (n, dim)).astype(np.float32)
    pairs = rng.integers(0, n, (n, 3)).astype(np.int32)
    node_b = rng.uniform(0.6, 1.1, n).astype(np.float32)
    e0, e1, mw = 3, 9, 0.3 if mid else 0.0
    z, zf = np.zeros(0, np.int32), np.zeros((0, dim), np.float32)
    Y, ed, nd = Y0.copy(), eons.copy(), eonns.copy()
    mg.optimize_layout(Y, head, tail, eps, ed, nd, z, z, e0, e1, ALPHA, ALPHA, mw, mw, A, b, A, rep_b, RATE, 0, 1.0, GAMMA, 4,
                       0.25, 0, 0, 0, zf, zf, z, 0.9, 0.999, z, pairs if mid else z.reshape(0, 1), z, z, 0.0, 0,
                       node_b if own_b else np.zeros(0, np.float32), 99, 1, 0, None, None, 0)
    kw = dict(mid_pairs=pairs, mid_w0=mw, mid_w1=mw) if mid else {}
    eo, no, D, P = eons.copy(), eonns.copy(), np.zeros((n, dim)), Y0.astype(np.float64)
    for e in range(e0, e1):
        smp, nn, off, negs, midp = O.sgd_schedule(Y0.copy(), head, tail, eps, eo, no, e, per_edge_stream=True, a=A, b=b,
                                                  rep_a=A, rep_b=rep_b, negative_sample_rate=RATE, seed=99, epoch_start=e0,
                                                  epoch_end=e1, alpha0=ALPHA, alpha1=ALPHA, negs_cap=20 * E + 64, **kw)
        i = np.flatnonzero(smp)
        u, v = head[i], tail[i]
        bb = (0.5 * (node_b[u].astype(np.float64) + node_b[v]) if own_b else np.full(len(i), b))[:, None]
        d = P[u] - P[v]
        d2 = (d * d).sum(1)[:, None]
        pw = d2 ** bb
        g = -2 * A * bb * pw / (d2 * (A * pw + 1)) * d
        gu = g.copy()
        np.add.at(D, v, np.clip(-g, -4, 4))
        cnt = np.maximum(nn[i], 0)
        row = np.repeat(np.arange(len(i)), cnt)
        first = np.cumsum(cnt) - cnt
        kk = negs[np.repeat(off[i], cnt) + np.arange(len(row)) - np.repeat(first, cnt)]
        d = P[u[row]] - P[kk]
        d2 = (d * d).sum(1)[:, None]
        g = np.where(kk[:, None] == u[row][:, None], 0.0, 2 * rep_b * GAMMA / ((0.001 + d2) * (A * d2 ** rep_b + 1)) * d)
        np.add.at(gu, row, g)
        if mid:
            w = midp[i]
            has = w >= 0
            g = np.where(has[:, None], -mw * (P[u] - P[np.maximum(w, 0)]), 0.0)
            gu += g
            np.add.at(D, w[has], np.clip(-g[has], -4, 4))
        np.add.at(D, u, np.clip(gu, -4, 4))
    assert np.array_equal(ed, eo) and np.array_equal(nd, no)
    D *= ALPHA
    assert np.linalg.norm((Y - P) - D) <= 0.02 * np.linalg.norm(D)
