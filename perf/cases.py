"""Timed cases of the layout pass: the calls a program makes into this package, with inputs on the device.

Families (a case's "kind"):
  tsne       the whole FFT t-SNE loop (`optimize_tsne` of the native surface): the "tsne" pass and the full-batch
             refinement of "hybrid"
  batch      many t-SNE layouts of uneven size together (`TsneBatch`)
  iteration  one iteration as the reference's own Python loop drives it: bbox_2d, FFTConv2D.compute,
             tsne_attraction, tsne_step
  sgd        one segment of the sampled SGD (`optimize_layout`, hogwild)
  transform  placing new rows into a resident layout (`FittedLayout.transform`): search, memberships, edge
             schedule, owner-mode SGD; host rows in, host positions out
  graph      a fit's graph on the device through the C ABI: smooth_knn, fuzzy union, edge schedule
  spectral   the spectral initialisation's solver (`chebyshev_eigenvectors`)

The layouts here are not at the end of an optimisation, so the optimisers run at learning rates that move them by
steps as small as a nearly finished layout makes. At larger ones the sign rule of the t-SNE gains (and the clipped
steps of racing threads in the SGD) turn a rounding into another path after a few iterations.

listed() and draw() give cases, prepare() makes a case's inputs from a seed, run() is one pass, work() counts what a
pass cannot do without, exact() gives the same outputs in 64 bits from plain torch."""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "lib-magnet_b200") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "lib-magnet_b200"))

DEV = "cuda"
A_UMAP, B_UMAP = 1.577, 0.895          # the kernel of min_dist 0.1, spread 1


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a small t-SNE layout (the low end of the batched sizes), where launches count; perplexity 30
        dict(name="tsne_2k", kind="tsne", n=2000, k=90, n_iter=60, early=10, ni=3, dof=1.0),
        # the 70,000-point perplexity-30 t-SNE configuration, a stretch across the end of early exaggeration
        dict(name="tsne_70k", kind="tsne", n=70000, k=90, n_iter=30, early=10, ni=3, dof=1.0),
        # the full-batch refinement of the million-point hybrid layout, the headline workload (k = 15)
        dict(name="hybrid_1m", kind="tsne", n=1000000, k=14, n_iter=10, early=0, ni=3, dof=1.0),
        # the batched form: many small layouts of log-uniform size in one graph per iteration
        dict(name="batch_24", kind="batch", count=24, lo=500, hi=5000, k=60, n_iter=30),
        # the drop-in per-iteration calls on a 10,000-point layout: latency of each call
        dict(name="iteration_10k", kind="iteration", n=10000, k=14, ni=3, dof=1.0),
        # the same calls on a large ragged layout with 5 interpolation nodes and heavy tails
        dict(name="iteration_400k", kind="iteration", n=399989, k=14, ni=5, dof=0.7),
        # the 10,000-point "umap" configuration: the last tenth of its 500 epochs (a late segment)
        dict(name="sgd_10k", kind="sgd", n=10000, k=14, dim=2, total=500, e0=450, e1=500),
        # the sampled SGD of the million-point layout: the last tenth of its 200 epochs
        dict(name="sgd_1m", kind="sgd", n=1000000, k=14, dim=2, total=200, e0=180, e1=200),
        # serving: a small request, and the largest one against 200,000 fitted rows of 64 features
        dict(name="transform_48", kind="transform", n=60000, d=64, m=48),
        dict(name="transform_4096", kind="transform", n=200000, d=64, m=4096),
        # the graph and edge schedule of a 300,000-row fit
        dict(name="graph_300k", kind="graph", n=300000, k=14, epochs=200),
        # the spectral initialisation of a 200,000-row fit
        dict(name="spectral_200k", kind="spectral", n=200000, k=14, p=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tsne", "tsne", "batch", "iteration", "iteration", "sgd", "sgd", "transform", "graph", "spectral"])
    if kind == "tsne":
        n = _log(rng, 500, 600000)
        k = rng.choice([14, 14, 30, 90]) if n <= 100000 else 14
        return dict(kind=kind, n=n, k=k, n_iter=max(8, min(40, 3000000 // n)), early=rng.choice([0, 4]),
                    ni=rng.choice([3, 3, 3, 4]), dof=rng.choice([1.0, 1.0, 0.8]))
    if kind == "batch":
        lo = _log(rng, 500, 1000)
        return dict(kind=kind, count=rng.randint(8, 24), lo=lo, hi=_log(rng, 2000, 5000), k=rng.choice([14, 30, 60]),
                    n_iter=rng.randint(10, 30))
    if kind == "iteration":
        return dict(kind=kind, n=_log(rng, 700, 400000), k=rng.choice([14, 14, 30]), ni=rng.choice([3, 3, 3, 4, 5]),
                    dof=rng.choice([1.0, 1.0, 0.7]))
    if kind == "sgd":
        n = _log(rng, 3000, 1000000)
        total = 500 if n <= 10000 else (300 if n <= 100000 else 200)
        return dict(kind=kind, n=n, k=14, dim=rng.choice([2, 2, 3]), total=total, e0=total - total // 10, e1=total)
    if kind == "transform":
        return dict(kind=kind, n=_log(rng, 20000, 200000), d=rng.choice([50, 64]), m=_log(rng, 1, 4096))
    if kind == "graph":
        return dict(kind=kind, n=_log(rng, 5000, 300000), k=rng.choice([9, 14, 19, 29]), epochs=rng.choice([200, 300, 500]))
    return dict(kind=kind, n=_log(rng, 5000, 200000), k=rng.choice([9, 14]), p=rng.choice([4, 4, 6]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)


def _disc(m, g):
    r = torch.sqrt(torch.rand(m, 1, generator=g, device=DEV))
    t = torch.rand(m, 1, generator=g, device=DEV) * (2 * math.pi)
    return torch.cat([r * torch.cos(t), r * torch.sin(t)], 1)


def _layout(n, std, g):
    """a layout of about n / 5000 + 5 round patches in a disc (a finished layout spans a little over 4 times its
    spread, 712 boxes at a million points), column 0 of the given spread, and its points' order along a Z-order curve"""
    c = 5 + n // 5000
    which = torch.randint(0, c, (n,), generator=g, device=DEV)
    Y = 0.9 * _disc(c, g)[which] + _disc(n, g) * (1.2 / math.sqrt(c))
    Y -= Y.mean(0)
    Y *= std / float(Y[:, 0].std())
    lo = Y.min(0).values
    q = ((Y - lo) / (Y.max(0).values - lo) * 32767).long()
    code = torch.zeros(n, dtype=torch.int64, device=DEV)
    for b in range(15):
        code |= ((q[:, 0] >> b) & 1) << (2 * b) | ((q[:, 1] >> b) & 1) << (2 * b + 1)
    return Y.contiguous(), torch.argsort(code)


def _neighbours(order, k, g):
    """k neighbours of every point among those near it along the curve, and their ascending distances"""
    n = order.numel()
    k = min(k, n // 4)
    off = torch.cumsum(torch.randint(1, 4, (n, k), generator=g, device=DEV), 1) % (n // 2)
    sign = torch.randint(0, 2, (n, k), generator=g, device=DEV) * 2 - 1
    rank = (torch.arange(n, device=DEV)[:, None] + off.clamp(min=1) * sign) % n
    ind = torch.empty((n, k), dtype=torch.int32, device=DEV)
    ind[order] = order[rank].int()
    first = 0.5 + torch.rand(n, 1, generator=g, device=DEV)
    gaps = torch.rand(n, k, generator=g, device=DEV) * (2.0 / k)
    gaps[:, 0] = 0
    dist = (first * (1 + torch.cumsum(gaps, 1))).float().contiguous()
    return ind.contiguous(), dist


def _symmetric(ind, vals):
    """CSR of a + a^T - a a^T over the neighbours' memberships a, columns sorted"""
    n, k = ind.shape
    rows = torch.arange(n, device=DEV).repeat_interleave(k)
    cols = ind.reshape(-1).long()
    v = vals.reshape(-1)
    keys, inv = torch.unique(torch.cat([rows * n + cols, cols * n + rows]), return_inverse=True)
    e = v.numel()
    keep = torch.zeros(keys.numel(), device=DEV)
    a = keep.index_put((inv[:e],), v)
    t = keep.index_put((inv[e:],), v)
    data = a + t - a * t
    r = keys // n
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    return indptr.int(), (keys % n).int(), data.float().contiguous()


def _graph(n, k, std, g):
    Y, order = _layout(n, std, g)
    ind, dist = _neighbours(order, k, g)
    vals = torch.exp(-(dist - dist[:, :1]) / (0.6 * dist[:, :1]))
    return Y, _symmetric(ind, vals)


def _spread(n):
    return 31.0 * math.sqrt(n / 70000.0)   # the hand-off of hybrid, and about where a t-SNE layout ends


def _rate(n):
    return n / (200.0 if n >= 20000 else 2000.0)


def _fft_len(m):
    while True:
        x = m
        for f in (2, 3, 5):
            while x % f == 0:
                x //= f
        if x == 1:
            return m
        m += 1


def _choose_grid(box, ni, max_boxes=1000, box_width=0.7, min_boxes=20):
    """the grid of magnet/tsne.py:30-46 for a bounding box"""
    lo = [float(box[0]) - 1e-3, float(box[1]) - 1e-3]
    hi = [float(box[2]) + 1e-3, float(box[3]) + 1e-3]
    span = max(hi[0] - lo[0], hi[1] - lo[1])
    nb = min(max(math.ceil(span / box_width), min_boxes), max_boxes)
    nb = min(max_boxes, -(-nb // 4) * 4)
    width = box_width if nb * box_width >= span else max(span / nb, 1e-12)
    return lo[0], lo[1], width, nb


def _spectra(nb, width, ni, dof):
    """M and the real half spectra (M, M / 2 + 1) of the two kernels on the wrapped grid, in 64 bits"""
    M = _fft_len(2 * nb * ni)
    off = torch.arange(M, device=DEV)
    off = torch.where(off <= M // 2, off, off - M).double() * (width / ni)
    base = 1.0 + (off[:, None] ** 2 + off[None, :] ** 2) / dof
    return M, torch.fft.rfft2(base ** -dof).real, torch.fft.rfft2(base ** (-dof - 1.0)).real


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    import magnet_b200 as mg
    g = _gen(seed)
    kind = case["kind"]
    if kind == "tsne":
        Y, (ip, ix, dd) = _graph(case["n"], case["k"], _spread(case["n"]), g)
        return _State(kind=kind, case=case, N=mg._native, Y=Y, ip=ip, ix=ix, dd=dd)
    if kind == "batch":
        graphs, Ys = [], []
        for i in range(case["count"]):
            f = (i + 0.5) / case["count"]
            n = int(case["lo"] * (case["hi"] / case["lo"]) ** f)
            Y, csr = _graph(n, case["k"], _spread(n), g)
            graphs.append(csr)
            Ys.append(Y)
        batch = mg._native.TsneBatch(graphs, n_iter=case["n_iter"], early_iter=case["n_iter"] // 3, learning_rate=0.5,
                                     threads_per_row=0, branches=32)
        return _State(kind=kind, case=case, batch=batch, graphs=graphs, Ys=Ys)
    if kind == "iteration":
        n = case["n"]
        Y, (ip, ix, dd) = _graph(n, case["k"], _spread(n), g)
        dd = (dd / dd.double().sum()).float()
        update = torch.randn(n, 2, generator=g, device=DEV) * 0.05
        gains = 0.2 + 1.5 * torch.rand(n, 2, generator=g, device=DEV)
        box = torch.cat([Y.min(0).values, Y.max(0).values]).tolist()
        _, _, width, nb = _choose_grid(box, case["ni"])
        M, K1, K2 = _spectra(nb, width, case["ni"], case["dof"])
        conv = mg.FFTConv2D(M, case["ni"])
        conv.set_kernels(K1.float().contiguous(), K2.float().contiguous())
        return _State(kind=kind, case=case, mg=mg, Y=Y, ip=ip, ix=ix, dd=dd, update=update, gains=gains,
                      convs={(nb, round(width, 6)): conv})
    if kind == "sgd":
        n, dim, total = case["n"], case["dim"], case["total"]
        Y, (ip, ix, w) = _graph(n, case["k"], 5.0, g)
        if dim == 3:
            Y = torch.cat([Y, torch.randn(n, 1, generator=g, device=DEV) * 2.0], 1).contiguous()
        # the edge schedule: freq = min(1, s w) summing to 5 n, edges below one visit dropped
        lo, hi = 0.0, 1e4
        wd = w.double()
        for _ in range(60):
            s = 0.5 * (lo + hi)
            if float(torch.clamp(s * wd, max=1.0).sum()) < 5.0 * n:
                lo = s
            else:
                hi = s
        freq = torch.clamp(lo * wd, max=1.0)
        keep = freq >= 1.0 / total
        head = torch.repeat_interleave(torch.arange(n, device=DEV), (ip[1:] - ip[:-1]).long())[keep].int()
        tail = ix[keep].contiguous()
        eps = (1.0 / freq[keep]).float()
        # where the schedule stands at epoch e0: the next visit, and the negatives drawn up to the last one
        last = eps * torch.floor((case["e0"] - 1) / eps)
        # (kept in arrays that hold every edge there can be, used up to the schedule's count)
        eons, eonns = (torch.zeros(2 * n * case["k"], device=DEV) for _ in range(2))
        eons[:eps.numel()] = last + eps
        eonns[:eps.numel()] = torch.ceil(last) - eps / 5.0 * torch.rand(eps.shape, generator=g, device=DEV)
        pairs = torch.randint(0, n, (n, 5), generator=g, device=DEV, dtype=torch.int32)
        z = torch.zeros(0, dtype=torch.int32, device=DEV)
        zf = torch.zeros(0, dtype=torch.float32, device=DEV)
        z2 = torch.zeros((0, dim), dtype=torch.float32, device=DEV)
        return _State(kind=kind, case=case, mg=mg, Y=Y, head=head, tail=tail, eps=eps, eons=eons, eonns=eonns,
                      pairs=pairs, z=z, zf=zf, z2=z2, seed=int(seed) % 65536)
    if kind == "transform":
        import scipy.sparse as sp
        from magnet_b200.serve import FittedLayout
        n, d, c = case["n"] // 50 * 50, case["d"], 50
        means = torch.randn(c, 1, d, generator=g, device=DEV) * 5.0
        X = means + torch.randn(c, n // c, d, generator=g, device=DEV)
        ind = torch.empty((c, n // c, 14), dtype=torch.int64, device=DEV)
        dist = torch.empty((c, n // c, 14), device=DEV)
        for j in range(c):      # neighbours lie in the row's own blob
            d2 = torch.cdist(X[j], X[j])
            d2.fill_diagonal_(float("inf"))
            dist[j], ind[j] = torch.topk(d2, 14, dim=1, largest=False)
            ind[j] += j * (n // c)
        mix = torch.randperm(n, generator=g, device=DEV)     # rows come in no order
        inv = torch.empty_like(mix)
        inv[mix] = torch.arange(n, device=DEV)
        ind = inv[ind.reshape(n, 14)][mix].int()
        dist = dist.reshape(n, 14)[mix]
        vals = torch.exp(-(dist - dist[:, :1]) / (0.3 * dist[:, :1]))
        ip, ix, dd = _symmetric(ind, vals)
        centres = torch.randn(c, 1, 2, generator=g, device=DEV) * 6.0
        Y = (centres + 0.5 * (X[:, :, :2] - means[:, :, :2])).reshape(n, 2)[mix]
        P = sp.csr_matrix((dd.cpu().numpy(), ix.cpu().numpy(), ip.cpu().numpy()), shape=(n, n))
        fitted = FittedLayout(X.reshape(n, d)[mix].cpu().numpy(), Y.cpu().numpy(), a=A_UMAP, b=B_UMAP, graph=P)
        which = torch.randint(0, c, (case["m"],), generator=g, device=DEV)
        Q = means[which, 0] + torch.randn(case["m"], d, generator=g, device=DEV)
        return _State(kind=kind, case=case, fitted=fitted, Q=Q.cpu().numpy(), seed=int(seed) % 65536)
    if kind == "graph":
        n = case["n"]
        _, order = _layout(n, 10.0, g)
        ind, dist = _neighbours(order, case["k"], g)
        k = ind.shape[1]
        cap = 2 * n * k
        f32 = dict(dtype=torch.float32, device=DEV)
        i32 = dict(dtype=torch.int32, device=DEV)
        return _State(kind=kind, case=case, lib=_c_abi(mg), ind=ind, dist=dist, vals=torch.empty((n, k), **f32),
                      indptr=torch.zeros(n + 1, **i32), indices=torch.zeros(cap, **i32), data=torch.zeros(cap, **f32),
                      head=torch.zeros(cap, **i32), tail=torch.zeros(cap, **i32), eps=torch.zeros(cap, **f32))
    n, p = case["n"], case["p"]
    _, (ip, ix, dd) = _graph(n, case["k"], 10.0, g)
    deg = torch.zeros(n, dtype=torch.float64, device=DEV)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (ip[1:] - ip[:-1]).long())
    deg.index_add_(0, rows, dd.double())
    X = torch.randn(n, p, generator=g, device=DEV)
    return _State(kind=kind, case=case, N=mg._native, ip=ip, ix=ix, dd=dd, X=X, sd=(1.0 / deg.sqrt()).float(),
                  comp=torch.zeros(n, dtype=torch.int32, device=DEV))


_LIB = None


def _c_abi(mg):
    """the C ABI, as a program that holds device arrays calls it"""
    global _LIB
    if _LIB is None:
        lib = ctypes.CDLL(mg.LIBRARY)
        P, I64, I, D = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_double
        lib.mg_smooth_knn.argtypes = [P, I64, I, I, ctypes.c_float, I, P]
        lib.mg_fuzzy_union.argtypes = [P, P, I64, I, I64, D, P, P, P, I64, ctypes.POINTER(I64)]
        lib.mg_edge_schedule.argtypes = [P, P, P, I64, I64, D, I, P, P, P, ctypes.POINTER(I64)]
        _LIB = lib
    return _LIB


def _ok(rc):
    if rc != 0:
        raise RuntimeError("C ABI call failed with status %d" % rc)


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    c = s.case
    if s.kind == "tsne":
        Y = s.Y.clone()
        s.N.optimize_tsne(s.ip, s.ix, s.dd, Y, n_iter=c["n_iter"], early_iter=c["early"], learning_rate=_rate(c["n"]),
                          n_interp=c["ni"], dof=c["dof"])
        return Y
    if s.kind == "batch":
        Ys = [Y.clone() for Y in s.Ys]
        s.batch.run(Ys)
        return torch.cat(Ys)
    if s.kind == "iteration":
        mg, Y, update, gains = s.mg, s.Y.clone(), s.update.clone(), s.gains.clone()
        xmin, ymin, width, nb = _choose_grid(mg.bbox_2d(Y), c["ni"])
        sumQ, F = s.convs[(nb, round(width, 6))].compute(Y, xmin, ymin, width, nb)
        attr = mg.tsne_attraction(s.ip, s.ix, s.dd, Y, c["dof"])
        mg.tsne_step(Y, update, gains, attr, F, 1.0, 1.0 / max(sumQ, 1e-12), max(200.0, c["n"] / 12.0), 0.8)
        # (the gains follow the gradient's sign alone; what they do shows in the update)
        return {"sumQ": sumQ, "F": F, "attr": attr, "Y": Y, "update": update}
    if s.kind == "sgd":
        Y, eons, eonns = s.Y.clone(), s.eons.clone(), s.eonns.clone()
        a0, a1 = 0.002 * (1.0 - c["e0"] / c["total"]), 0.002 * (1.0 - c["e1"] / c["total"])
        m = s.head.numel()
        s.mg.optimize_layout(Y, s.head, s.tail, s.eps, eons[:m], eonns[:m], s.z, s.z, c["e0"], c["e1"], a0, a1, 0.05, 0.0,
                             A_UMAP, B_UMAP, A_UMAP, 1.0, 5.0, 0, 1.0, 2.0, 4, 0.25, 0, 0, 0, s.z2, s.z2, s.z, 0.9,
                             0.999, s.z, s.pairs, s.z, s.z, 0.0, 0, s.zf, s.seed, -1)
        return {"Y": Y, "eons": eons, "eonns": eonns}
    if s.kind == "transform":
        return s.fitted.transform(s.Q, seed=s.seed)
    if s.kind == "graph":
        n, k = s.ind.shape
        nnz, kept = ctypes.c_int64(0), ctypes.c_int64(0)
        _ok(s.lib.mg_smooth_knn(s.dist.data_ptr(), n, k, k + 1, 1.0, 64, s.vals.data_ptr()))
        _ok(s.lib.mg_fuzzy_union(s.ind.data_ptr(), s.vals.data_ptr(), n, k, n, 1.0, s.indptr.data_ptr(),
                                 s.indices.data_ptr(), s.data.data_ptr(), s.indices.numel(), ctypes.byref(nnz)))
        _ok(s.lib.mg_edge_schedule(s.indptr.data_ptr(), s.indices.data_ptr(), s.data.data_ptr(), n, nnz.value, 5.0,
                                   c["epochs"], s.head.data_ptr(), s.tail.data_ptr(), s.eps.data_ptr(),
                                   ctypes.byref(kept)))
        return {"vals": s.vals, "indptr": s.indptr, "indices": s.indices, "data": s.data, "head": s.head,
                "tail": s.tail, "eps": s.eps, "nnz": nnz.value, "kept": kept.value}
    X = s.X.clone()
    # magnet/spectral.py: 2 wanted vectors of p columns (4 of 6 in 3-d), degree 30, its iteration budget, tol 0.05
    s.N.chebyshev_eigenvectors(s.ip, s.ix, s.dd, X, s.sd, s.comp, c["p"] // 2, 30, 3, 0.05)
    return X


# ------------------------------------------------------------------------------------------------ work
def work(case):
    kind, n, k = case["kind"], case.get("n", 0), case.get("k", 14)
    row = 1.7 * k               # entries per row of the symmetric graph, about

    def tsne_iteration(n, row, ni):
        # positions, update, gains in and out, the affinities; the charges' and potentials' grid once each way,
        # and the transforms of 3 charge and 3 potential channels
        N = ni * max(20, math.ceil(4.3 * _spread(n) / 0.7))
        b = n * (48 + 8 * row) + 24.0 * N * N
        f = n * (12 * row + 20 * ni * ni) + 6 * 2.5 * (2 * N) ** 2 * math.log2((2 * N) ** 2)
        return b, f

    if kind == "tsne":
        b, f = tsne_iteration(n, row, case["ni"])
        return {"bytes": b * case["n_iter"], "flops": f * case["n_iter"]}
    if kind == "batch":
        b = f = 0.0
        for i in range(case["count"]):
            m = int(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / case["count"]))
            x, y = tsne_iteration(m, row, 3)
            b, f = b + x, f + y
        return {"bytes": b * case["n_iter"], "flops": f * case["n_iter"]}
    if kind == "iteration":
        b, f = tsne_iteration(n, row, case["ni"])
        return {"bytes": b + 24.0 * n, "flops": f}
    if kind == "sgd":
        # per epoch: the schedule of every edge read, and 5 n samples of an edge, its state and 7 positions
        epochs = case["e1"] - case["e0"]
        return {"bytes": epochs * n * (4.0 * row + 5 * (16 + 8 + 8 * case["dim"] / 2 * 7)), "flops": epochs * n * 5 * 120.0}
    if kind == "transform":
        m, d = case["m"], case["d"]
        visited = min(n, 1600)
        return {"bytes": m * (4.0 * d * visited + 100 * 5 * 7 * 8) + 8.0 * n, "flops": m * (3.0 * d * visited + 100 * 5 * 120)}
    if kind == "graph":
        return {"bytes": n * (12.0 * k + 8 * row + 12 * row), "flops": n * k * 20.0}
    products = 31.0 * 3
    return {"bytes": products * n * (8 * row + 16 * case["p"]), "flops": products * n * row * 2 * case["p"]}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _weights(u, ni):
    w = torch.ones((u.numel(), ni), dtype=torch.float64, device=DEV)
    for k in range(ni):
        for m in range(ni):
            if m != k:
                w[:, k] *= (u - (m + 0.5) / ni) / ((k - m) / ni)
    return w


def _repulsion(Y, xmin, ymin, width, nb, ni, spectra):
    """sumQ and F of positions Y by interpolation on the grid; the boxes as 32-bit positions fall into them"""
    M, K1, K2 = spectra
    N = nb * ni
    inv_w = torch.tensor(1.0, dtype=torch.float32) / torch.tensor(width, dtype=torch.float32)
    y32 = Y.float()
    x0, y0 = torch.tensor(xmin, dtype=torch.float32).item(), torch.tensor(ymin, dtype=torch.float32).item()
    w32 = torch.tensor(width, dtype=torch.float32).item()
    bx = ((y32[:, 0] - x0) * inv_w.item()).int().clamp(0, nb - 1).long()
    by = ((y32[:, 1] - y0) / w32).int().clamp(0, nb - 1).long()
    wx = _weights(((Y[:, 0] - x0) / w32 - bx).clamp(0.0, 1.0), ni)
    wy = _weights(((Y[:, 1] - y0) / w32 - by).clamp(0.0, 1.0), ni)
    W = torch.zeros((3, M, M), dtype=torch.float64, device=DEV)
    for a in range(ni):
        for b in range(ni):
            at = (bx * ni + a) * M + by * ni + b
            w = wx[:, a] * wy[:, b]
            for c, q in enumerate((w, w * Y[:, 0], w * Y[:, 1])):
                W[c].view(-1).index_add_(0, at, q)
    phi = []
    for c in range(3):
        h = torch.fft.rfft2(W[c])
        if c == 0:
            phi.append(torch.fft.irfft2(h * K1, s=(M, M)))
        phi.append(torch.fft.irfft2(h * K2, s=(M, M)))
        del h
    p = torch.zeros((4, Y.shape[0]), dtype=torch.float64, device=DEV)
    for a in range(ni):
        for b in range(ni):
            at = (bx * ni + a) * M + by * ni + b
            w = wx[:, a] * wy[:, b]
            for c in range(4):
                p[c] += w * phi[c].reshape(-1)[at]
    return p[0].sum() - Y.shape[0], p[1][:, None] * Y - p[2:4].T


def _attraction(rows, ix, p, Y, dof):
    diff = Y[rows] - Y[ix.long()]
    w = p / (1.0 + (diff * diff).sum(1) / dof)
    return torch.zeros_like(Y).index_add_(0, rows, diff * w[:, None])


def _step(Y, u, gains, grad, lr, mom):
    gains = torch.where((grad > 0) == (u > 0), gains * 0.8, gains + 0.2).clamp(min=0.01)
    u = mom * u - lr * gains * grad
    Y = Y + u
    return Y - Y.mean(0), u, gains


def _loop(Y, csr, n_iter, early, lr, ni, dof):
    ip, ix, dd = csr
    n = Y.shape[0]
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (ip[1:] - ip[:-1]).long())
    p = dd.double()
    p /= p.sum()
    Y = Y.double()
    u, gains = torch.zeros_like(Y), torch.ones_like(Y)
    spectra, key = None, None
    for it in range(n_iter):
        box = torch.cat([Y.min(0).values, Y.max(0).values]).float().tolist()
        xmin, ymin, width, nb = _choose_grid(box, ni)
        if key != (nb, round(width, 6)):
            key, spectra = (nb, round(width, 6)), _spectra(nb, width, ni, dof)
        sumQ, F = _repulsion(Y, xmin, ymin, width, nb, ni, spectra)
        rho, mom = (12.0, 0.5) if it < early else (1.0, 0.8)
        Y, u, gains = _step(Y, u, gains, rho * _attraction(rows, ix, p, Y, dof) - F / sumQ, lr, mom)
    return Y


def _memberships(dist, k):
    """the bisection of src/graph.cpp:29-78 in 64 bits"""
    d = dist.double()
    n = d.shape[0]
    target = math.log2(k + 1)
    rho = d[:, :1]
    lo = torch.zeros((n, 1), dtype=torch.float64, device=DEV)
    hi = torch.full_like(lo, float("inf"))
    mid = torch.ones_like(lo)
    done = torch.zeros_like(lo, dtype=torch.bool)
    for _ in range(64):
        t = d - rho
        psum = torch.where(t > 0, torch.exp(-t / mid), 1.0).sum(1, keepdim=True)
        done |= (psum - target).abs() < 1e-5
        over = psum > target
        hi = torch.where(over & ~done, mid, hi)
        lo = torch.where(~over & ~done, mid, lo)
        mid = torch.where(done, mid, torch.where(torch.isinf(hi), mid * 2, (lo + hi) * 0.5))
    t = d - rho
    return torch.where(t > 0, torch.exp(-t / torch.maximum(mid, 1e-3 * d.mean(1, keepdim=True))), 1.0)


def _jacobi(H):
    """eigenvalues, descending, and vectors of a small symmetric matrix by cyclic Jacobi rotations, which also settle
    the vectors' signs"""
    A, p = H.cpu().numpy().copy(), H.shape[0]
    V = np.eye(p)
    for _ in range(100):
        if (np.triu(A, 1) ** 2).sum() < 1e-22:
            break
        for i in range(p):
            for j in range(i + 1, p):
                if abs(A[i, j]) < 1e-300:
                    continue
                q = (A[j, j] - A[i, i]) / (2 * A[i, j])
                t = (1.0 if q >= 0 else -1.0) / (abs(q) + math.sqrt(q * q + 1))
                c = 1 / math.sqrt(t * t + 1)
                J = np.eye(p)
                J[i, i] = J[j, j] = c
                J[i, j], J[j, i] = t * c, -t * c
                A, V = J.T @ A @ J, V @ J
    order = np.argsort(-np.diag(A))
    return torch.tensor(np.diag(A)[order].copy(), device=DEV), torch.tensor(V[:, order].copy(), device=DEV)


def _ritz(X, apply, n_wanted):
    Z = apply(X)
    H = X.T @ Z
    theta, V = _jacobi(torch.triu(H) + torch.triu(H, 1).T)
    X, Z = X @ V, Z @ V
    return X, theta.tolist(), float((Z - theta * X)[:, :n_wanted].norm(dim=0).max())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sgd", "transform", "batch") or (kind == "tsne" and case["n"] < 20000):
        # races and draws (sgd, transform); in a small layout one gain that a rounding turns shows: no value in 64 bits
        return None
    s = prepare(case, seed)
    if kind == "tsne":
        return _loop(s.Y, (s.ip, s.ix, s.dd), case["n_iter"], case["early"], _rate(case["n"]), case["ni"], case["dof"])
    if kind == "iteration":
        n, ni, dof = case["n"], case["ni"], case["dof"]
        Y = s.Y.double()
        xmin, ymin, width, nb = _choose_grid(torch.cat([s.Y.min(0).values, s.Y.max(0).values]).tolist(), ni)
        sumQ, F = _repulsion(Y, xmin, ymin, width, nb, ni, _spectra(nb, width, ni, dof))
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), (s.ip[1:] - s.ip[:-1]).long())
        attr = _attraction(rows, s.ix, s.dd.double(), Y, dof)
        Y, u, _ = _step(Y, s.update.double(), s.gains.double(), attr - F / sumQ, max(200.0, n / 12.0), 0.8)
        return {"sumQ": float(sumQ), "F": F, "attr": attr, "Y": Y, "update": u}
    if kind == "graph":
        vals = _memberships(s.dist, s.dist.shape[1])
        n, k = s.ind.shape
        rows = torch.arange(n, device=DEV).repeat_interleave(k)
        cols = s.ind.reshape(-1).long()
        keys, inv = torch.unique(torch.cat([rows * n + cols, cols * n + rows]), return_inverse=True)
        zero = torch.zeros(keys.numel(), dtype=torch.float64, device=DEV)
        a = zero.index_add(0, inv[:n * k], vals.reshape(-1))
        t = zero.index_add(0, inv[n * k:], vals.reshape(-1))
        data = torch.zeros(s.data.numel(), dtype=torch.float64, device=DEV)
        data[:keys.numel()] = a + t - a * t
        return {"vals": vals, "indptr": None, "indices": None, "data": data, "head": None, "tail": None, "eps": None,
                "nnz": None, "kept": None}
    n, p, nw = case["n"], case["p"], case["p"] // 2
    sd = s.sd.double()[:, None]
    trivial = 1.0 / sd
    P = torch.sparse_csr_tensor(s.ip.long(), s.ix.long(), s.dd.double(), size=(n, n))

    def deflate(X):
        return X - trivial * (trivial * X).sum(0) / (trivial * trivial).sum()

    def apply(X):
        return deflate(0.5 * (X + sd * (P @ (sd * X))))

    def orthonormal(X):
        X = deflate(X).clone()
        for _ in range(2):
            for k in range(p):
                if k:
                    X[:, k] -= X[:, :k] @ (X[:, :k].T @ X[:, k])
                X[:, k] /= X[:, k].norm()
        return X

    X, theta, res = _ritz(orthonormal(s.X.double()), apply, nw)
    prev = -1.0
    for _ in range(3):
        gap = max(theta[nw - 1] - theta[nw], 1e-3)
        total = sum(theta[:nw])
        if res < 0.05 * gap or res < 1e-9 or (prev >= 0 and abs(total - prev) < 1e-9 * nw):
            break
        prev = total
        alpha = max(min(theta[p - 1], theta[nw - 1] - 0.5 * gap), 1e-3)
        e = 0.5 * alpha
        sigma1 = e / (min(1.0, theta[0] + 1e-9) - e)
        sigma = sigma1
        Y = (apply(X) - e * X) * (sigma1 / e)
        for _ in range(2, 31):
            new = 1.0 / (2.0 / sigma1 - sigma)
            X, Y = Y, (apply(Y) - e * Y) * (2.0 * new / e) - sigma * new * X
            sigma = new
        X, theta, res = _ritz(orthonormal(Y), apply, nw)
    return X
