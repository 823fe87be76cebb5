"""The quantized categorical search's scans against the oracle, where the warp form can go wrong: category
counts around one and several warps of positions, groups that every category fills and that take many,
few and no categories with enough data, short and long scans, both children.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("cats", [3, 31, 33, 64, 150, 254])
@pytest.mark.parametrize("kw", [dict(), dict(min_data_per_group=1), dict(min_data_per_group=900), dict(max_cat_threshold=200),
                                dict(max_cat_threshold=5, min_data_in_leaf=300), dict(cat_smooth=120.0),
                                dict(max_cat_threshold=128, min_data_per_group=333, min_sum_hessian_in_leaf=60.0)],
                         ids=lambda k: "-".join("%s%g" % x for x in k.items()) or "plain")
def test_categorical_scans_match_oracle(cats, kw):
    import harness
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(cats)
    n = 20011
    c = np.floor(rng.random(n) ** 1.5 * cats)
    X = np.stack([c, rng.integers(0, cats, n).astype(float), rng.standard_normal(n)], axis=1)
    ds = BinnedDataset.from_dense(X, categorical=[0, 1])
    effect = rng.standard_normal(cats)
    g = (effect[c.astype(int)] + 0.3 * X[:, 2] + rng.standard_normal(n)).astype(np.float32)
    h = (0.1 + 0.2 * rng.random(n)).astype(np.float32)
    cfg = LearnerConfig(num_leaves=12, use_quantized_grad=1, num_grad_quant_bins=16, stochastic_rounding=1, seed=5,
                        num_threads=2, **kw)
    ro = harness.OracleLearner(ds, cfg).train(g, h)
    for timed in (False, True):  # grow rounds, one split at a time
        L = GpuTreeLearner(ds, cfg)
        L.set_timing(timed)
        rg = L.train(g, h)
        assert len(rg[0]) == len(ro[0])
        for name in ("leaf", "inner_feature", "categorical", "left_count", "left_int_sum", "gain", "cat_bins"):
            assert np.array_equal(rg[0][name], ro[0][name]), name
        assert np.array_equal(rg[1], ro[1])
