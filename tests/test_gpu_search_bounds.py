"""The quantized search's bounds hold, and leave few thresholds to be evaluated in full, whatever the
leaf's smallest side, the gradients' unit and how many of them are zero: trees equal to the oracle's, at
about the time of an ordinary one (a search that evaluates every threshold takes a tree four times as
long).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _data():
    from lgbm_gb300 import BinnedDataset
    rng = np.random.default_rng(1)
    X = rng.standard_normal((30000, 40))
    ds = BinnedDataset.from_dense(X)
    g = (0.3 * rng.standard_normal(30000) - np.sin(X[:, 0] + X[:, 1] * (X[:, 2] > 0))).astype(np.float32)
    h = (0.2 + 0.8 * rng.random(30000)).astype(np.float32)
    return ds, X, g, h


def _tree(ds, g, h, **kw):
    """The tree (checked against the oracle's) and the device time of growing it."""
    import harness
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    cfg = LearnerConfig(num_leaves=63, use_quantized_grad=1, seed=5, num_threads=2, fused_madd=1, **kw)
    L = GpuTreeLearner(ds, cfg)
    want = harness.OracleLearner(ds, cfg).train(g, h)
    got = L.train(g, h)
    assert len(got[0]) == len(want[0]) > 10
    for name in ("leaf", "inner_feature", "threshold", "left_count", "left_int_sum", "gain"):
        assert np.array_equal(got[0][name], want[0][name]), name
    assert np.array_equal(got[1], want[1])
    t = []
    for _ in range(7):
        L.train(g, h)
        t.append(L.last_timing()["total_ms"])
    L.close()
    return float(np.median(t))


@pytest.mark.parametrize("kw", [dict(min_sum_hessian_in_leaf=0.0, min_data_in_leaf=1),
                                dict(min_sum_hessian_in_leaf=0.0, min_data_in_leaf=0),
                                dict(min_sum_hessian_in_leaf=0.0, min_data_in_leaf=0, lambda_l2=1e-9)],
                         ids=lambda k: "-".join("%s" % v for v in k.values()))
def test_leaves_without_a_least_hessian(kw):
    ds, X, g, h = _data()
    assert _tree(ds, g, h, **kw) < 2.0 * _tree(ds, g, h)


@pytest.mark.parametrize("min_gain", [0.0, 1e-3])
def test_leaves_without_gradients(min_gain):
    """Only the rows of a corner have gradients; most leaves and features have none to split by."""
    ds, X, g, h = _data()
    g = np.where((X[:, 0] > 1.0) & (X[:, 1] > 0.0), g, 0.0).astype(np.float32)
    g[:600] *= np.float32(0.1)
    kw = dict(min_gain_to_split=min_gain, min_data_in_leaf=3)
    assert _tree(ds, g, h, **kw) < 1.6 * _tree(*_data()[:1], *_data()[2:], **kw)


@pytest.mark.parametrize("unit", [1e-30, 1e-20, 1e-13, 1e13, 1e16])
@pytest.mark.parametrize("l2", [0.0, 3.0])
def test_units_of_the_gradients(unit, l2):
    ds, X, g, h = _data()
    assert _tree(ds, (g * np.float32(unit)).astype(np.float32), h, lambda_l2=l2) < 2.0 * _tree(ds, g, h, lambda_l2=l2)
