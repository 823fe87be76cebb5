"""Root sums of gradient levels that are no power of two, which the reference adds row after row in f64:
equal to the oracle's around the batches of 32 rows, with and without bagging, at the pace of one chain of
additions for each of the two sums.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _learner(n, bins, **kw):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(n + bins)
    X = rng.standard_normal((n, 3))
    ds = BinnedDataset.from_dense(X, min_data_in_leaf=1, min_data_in_bin=1, feature_pre_filter=False)
    g = (X[:, 0] + rng.standard_normal(n)).astype(np.float32)
    h = (0.1 + rng.random(n)).astype(np.float32)
    cfg = LearnerConfig(num_leaves=4, min_data_in_leaf=1, min_sum_hessian_in_leaf=0.0, use_quantized_grad=1,
                        num_grad_quant_bins=bins, seed=4, num_threads=2, **kw)
    return ds, GpuTreeLearner(ds, cfg), g, h


@pytest.mark.parametrize("bins", [3, 5, 127])
@pytest.mark.parametrize("n", [33, 64, 65, 96, 1000, 4097])
def test_root_sums_match_oracle(n, bins):
    import harness
    ds, L, g, h = _learner(n, bins)
    orc = harness.OracleLearner(ds, L.cfg)
    bag = np.nonzero(np.random.default_rng(2).random(n) < 0.6)[0].astype(np.int32)
    for rows in (None, bag, bag[:len(bag) // 32 * 32]):
        if rows is not None and len(rows) < 2:
            continue
        a, b = L.train(g, h, rows), orc.train(g, h, rows)
        assert a[2] == b[2] and len(a[0]) == len(b[0])
        assert a[0].tobytes() == b[0].tobytes() and np.array_equal(a[1], b[1])


def test_root_sums_take_one_chain_each():
    n = 200000
    ds, L, g, h = _learner(n, 5)
    t = []
    for _ in range(4):
        L.train(g, h)
        t.append(L.last_timing()["total_ms"])
    assert min(t) * 1e6 / n < 170.0  # ns a row: 104; with both sums on one lane 233
    L.close()
