"""Histograms and row partitions where their inner loops change form, against the oracle bit for bit:
feature counts around the 4, 8, 16 and 32 steps of a tile, 8- and 4-bit bins, the packed and the wide
integer counters; leaf sizes around a CTA's tile of the partition.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _learner(n, F, max_bin, levels=4, K=1, leaves=3, seed=1):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, F))
    X[:, ::3] = rng.integers(0, 12, size=(n, len(range(0, F, 3))))
    ds = BinnedDataset.from_dense(X, max_bin=max_bin)
    g = (X[:, 0] - X[:, -1] + rng.standard_normal((K, n))).astype(np.float32)
    h = (0.05 + 0.2 * rng.random((K, n))).astype(np.float32)
    cfg = LearnerConfig(num_leaves=leaves, min_data_in_leaf=1, min_sum_hessian_in_leaf=0.0, use_quantized_grad=1,
                        num_grad_quant_bins=levels, stochastic_rounding=0, num_threads=2)
    return ds, GpuTreeLearner(ds, cfg, num_jobs=K), g, h


@pytest.mark.parametrize("F", [1, 4, 5, 8, 9, 16, 17, 31, 33, 36, 40, 48, 49])
@pytest.mark.parametrize("max_bin,levels", [(255, 4), (15, 4), (63, 64), (255, 254)])
def test_integer_tiles_match_oracle(F, max_bin, levels):
    import harness
    n = 20000 + F
    ds, L, g, h = _learner(n, F, max_bin, levels, K=2, leaves=7)
    tree = L.train_raw(g, h)
    for j in range(2):
        rec, values = harness.OracleLearner(ds, L.cfg).train(g[j], h[j])[:2]
        k = int(tree[3][j])
        assert k == len(rec) + 1
        for name in ("leaf", "inner_feature", "threshold", "left_count", "left_int_sum", "gain"):
            assert np.array_equal(tree[0][j, :k - 1][name], rec[name]), name
        assert np.array_equal(tree[1][j, :k], values)


@pytest.mark.parametrize("n", [100, 255, 256, 257, 1023, 1024, 1025, 2049, 70000])
def test_partition_tiles_match_oracle(n):
    """Each leaf holds the rows that its splits send there, whatever its size and the bagged rows."""
    import harness
    ds, L, g, h = _learner(n, 6, 255, leaves=31)
    orc = harness.OracleLearner(ds, L.cfg)
    bag = np.nonzero(np.random.default_rng(2).random(n) < 0.6)[0].astype(np.int32)
    for rows in (None, bag):
        nl = int(L.train_raw(g, h, rows=rows)[3][0])
        assert nl == len(orc.train(g[0], h[0], rows=rows)[1])
        used = np.arange(n) if rows is None else rows
        assert np.array_equal(L.row_leaf()[used], orc.row_leaf()[used])
