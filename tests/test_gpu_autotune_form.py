"""The launch-shape autotuner's cache keeps the two ways of growing a tree apart: a learner that grows
in rounds does not take a shape timed on single splits, nor the other way round.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _constrained(L):
    L.set_interaction_constraints([[0, 1, 2, 3], [3, 4, 5, 6]])


SINGLE = {"constraints": (_constrained, 1), "bynode": (lambda L: L.set_bynode(0.5, False, 3), 1),
          "timing": (lambda L: L.set_timing(True), 1), "plain form": (lambda L: None, 0)}


@pytest.mark.parametrize("first", ["single", "rounds"])
@pytest.mark.parametrize("i,why", list(enumerate(SINGLE)))
def test_shapes_are_cached_by_growth(i, why, first):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    n, F = 3000, 7
    leaves = 20 + 2 * i + (first == "rounds")  # a shape class of its own
    rng = np.random.default_rng(i)
    X = rng.standard_normal((n, F))
    ds = BinnedDataset.from_dense(X)
    g, h = (X[:, 0] + 0.3 * rng.standard_normal(n)).astype(np.float32), np.ones(n, np.float32)
    setup, mode = SINGLE[why]

    def tune(single):
        """Whether the shape came from trial trees (the learner has trained none itself)."""
        L = GpuTreeLearner(ds, LearnerConfig(num_leaves=leaves, use_quantized_grad=1), loop_mode=mode if single else 1)
        if single:
            setup(L)
        shape = L.autotune(g, h, trials=1)
        assert shape == L.launch_shape() and shape[4] == 1
        timed = L.last_timing()["total_ms"] > 0.0
        L.close()
        return timed

    order = (True, False) if first == "single" else (False, True)
    assert [tune(s) for s in order] == [True, True]
    assert [tune(s) for s in order] == [False, False]
