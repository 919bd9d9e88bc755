"""A t-SNE step in a caller's graph: captured at a larger size than the calls before it had, and replayed after calls of other
sizes, it does what the plain call does, bit for bit. (A thread of its own: the library's scratch is per thread, and other
tests' calls would have grown it.)"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def arrays(torch, n, dim, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda: torch.randn(n, dim, generator=g, device="cuda")
    return [r(), r() * 0.1, 0.5 + torch.rand(n, dim, generator=g, device="cuda"), r() * 1e-4, r()]


@pytest.mark.parametrize("dim", [2, 7])
def test_captured_step(mg, cuda, dim):
    import torch
    out = {}

    def work():
        try:
            s = torch.cuda.Stream()
            mg._native.set_stream(s.cuda_stream)
            step = lambda a: mg.tsne_step(*a, 12.0, 1e-3, 200.0, 0.5)
            with torch.cuda.stream(s):
                step(arrays(torch, 50, dim, 0))
                ref, cap = arrays(torch, 300000, dim, 1), arrays(torch, 300000, dim, 1)
                s.synchronize()
                graph = torch.cuda.CUDAGraph()
                graph.capture_begin(capture_error_mode="thread_local")
                step(cap)
                graph.capture_end()
                big = arrays(torch, 1000000, dim, 2)
                step(big)
                mg.bbox_2d(big[0][:, :2].contiguous())
                graph.replay()
                step(ref)
            torch.cuda.synchronize()
            out["same"] = all(torch.equal(a, b) for a, b in zip(ref[:3], cap[:3]))
            del graph
        except BaseException as e:
            out["error"] = e
        finally:
            mg._native.set_stream(0)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert "error" not in out, out["error"]
    assert out["same"]
