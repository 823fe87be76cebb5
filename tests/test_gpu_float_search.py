"""The plain float search from exact fixed-point sums, against the oracle's f64 search, where its
integers, bounds and queue can go wrong: leaves whose mean gradient is far from zero (thresholds that
differ in the last digits), lambda_l2, ties of empty bins, hessians near min_sum_hessian, missing values
of each kind with both scan directions, few and many bins, constant hessians; and trees whose values
span too much for the fixed point, which the f64 search takes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("kw", [dict(), dict(lambda_l2=5.0), dict(min_sum_hessian_in_leaf=40.0, min_data_in_leaf=1),
                                dict(min_gain_to_split=2.0)], ids=lambda k: "-".join(k) or "plain")
@pytest.mark.parametrize("grad", ["normal", "shifted", "const", "wide"])
@pytest.mark.parametrize("max_bin,missing", [(255, "nan"), (255, "none"), (255, "zero"), (63, "nan"), (15, "zero")])
def test_float_trees_match_oracle(kw, grad, max_bin, missing):
    import harness
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    n, F = 12011, 9
    rng = np.random.default_rng(max_bin + len(grad))
    X = rng.standard_normal((n, F))
    X[:, :3] = rng.integers(0, 12, size=(n, 3))
    X[:, 3] = np.where(rng.random(n) < 0.6, 1.5, X[:, 3])  # the most frequent bin inside the slice
    z = 0.4 * X[:, 0] + X[:, 4] * (X[:, 5] > 0.3) - np.abs(X[:, 6])
    if missing == "nan":
        X[rng.random((n, F)) < 0.1] = np.nan
    ds = BinnedDataset.from_dense(X, max_bin=max_bin, zero_as_missing=missing == "zero")
    g = (z + 0.5 * rng.standard_normal(n)).astype(np.float32)
    h = (0.05 + 0.2 * rng.random(n)).astype(np.float32)
    if grad == "shifted":
        g = (g + np.float32(50.0)).astype(np.float32)
    elif grad == "const":
        h[:] = 1.0
    elif grad == "wide":
        g[::7] *= np.float32(2.0 ** -100)
    cfg = LearnerConfig(num_leaves=15, use_quantized_grad=0, is_constant_hessian=grad == "const", num_threads=2, fused_madd=1,
                        **kw)
    ro = harness.OracleLearner(ds, cfg).train(g, h)
    for timed in (False, True):  # grow rounds, one split at a time
        L = GpuTreeLearner(ds, cfg)
        L.set_timing(timed)
        rg = L.train(g, h)
        e = harness.gain_errors(rg[0], ro[0])
        # both searches take the f64 gain of the chosen threshold from sums good to about 1e-13 of a bin's
        # mass; a gain is the difference of terms up to 1e4 times as large
        assert e["max_rel"] <= 1e-6, e
        if e["splits_compared"] == len(ro[0]):
            assert len(rg[0]) == len(ro[0])
            np.testing.assert_allclose(rg[1], ro[1], rtol=1e-9)
        else:  # a tie: the two splits gain the same
            tie = e["near_ties"][0]
            assert abs(tie["gpu"][3] - tie["oracle"][3]) <= 1e-9 * abs(tie["oracle"][3]) + 1e-9, tie


def test_many_searches_match_single_splits():
    """The launch form for more than two waves of searches (2 x 40 features x 16 leaves)."""
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(8)
    n, F = 40000, 40
    X = rng.standard_normal((n, F))
    ds = BinnedDataset.from_dense(X)
    g = (X @ rng.standard_normal(F) + rng.standard_normal(n)).astype(np.float32)
    h = (0.1 + rng.random(n)).astype(np.float32)
    cfg = LearnerConfig(num_leaves=255, use_quantized_grad=0, num_threads=2)
    a, b = GpuTreeLearner(ds, cfg), GpuTreeLearner(ds, cfg)
    b.set_timing(True)
    x, y = a.train(g, h), b.train(g, h)
    assert len(x[0]) == len(y[0])
    np.testing.assert_allclose(x[0]["gain"], y[0]["gain"], rtol=1e-9)
    np.testing.assert_allclose(x[1], y[1], rtol=1e-9)
