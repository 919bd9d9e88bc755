"""The batch autotuner times each launch shape once: the batch runs its layouts as at most two sets, so a branch count above
two is the run of two again. The batch is a stand-in that records how it was made (no GPU)."""
import numpy as np
import pytest


@pytest.fixture
def recorded(monkeypatch, tmp_path):
    native = pytest.importorskip("magnet_b200._native")
    made = []

    class Batch:
        def __init__(self, graphs, n_iter, threads_per_row, branches, **params):
            made.append((threads_per_row, branches))

        def run(self, Ys):
            pass

    monkeypatch.setattr(native, "TsneBatch", Batch)
    monkeypatch.setenv("MAGNET_B200_CACHE", str(tmp_path))
    return made


def test_no_shape_is_timed_twice(recorded):
    from magnet_b200 import autotune as A
    graphs = [(np.array([0, 1, 2], np.int32), np.array([1, 0], np.int32), np.ones(2, np.float32))]
    choice = A.tune_tsne_batch(graphs, [np.zeros((2, 2), np.float32)], {}, key="k")
    shapes = [(t, min(b, 2)) for t, b in recorded]
    assert len(set(shapes)) == len(shapes), recorded
    assert {b for _, b in shapes} == {1, 2}
    assert choice["branches"] in A.BRANCHES and A.lookup("k") == choice
