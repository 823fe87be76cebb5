"""Quantized leaf renewal against the oracle, which adds every leaf's gradients and hessians one after
the other in f64: leaf values bit for bit, in grow rounds (rows grouped again) and one split at a time,
for gradients whose sums are exact, that round now and then, that round nearly always, and that span
too many binary orders for the integer sums; bagged rows in an order of their own; class trees.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _grad(kind, n, rng, z):
    if kind == "normal":
        return (z + rng.standard_normal(n)).astype(np.float32), (0.05 + 0.2 * rng.random(n)).astype(np.float32)
    if kind == "integers":
        return rng.integers(-3, 4, n).astype(np.float32), np.ones(n, np.float32)
    if kind == "tiny":  # a thousandth of the rows far below the rest
        s = np.where(rng.random(n) < 1e-3, 2.0 ** -30, 1.0)
        return ((z + rng.standard_normal(n)) * s).astype(np.float32), ((0.05 + 0.2 * rng.random(n)) * s).astype(np.float32)
    if kind == "wide":
        s = np.exp2(-rng.integers(0, 90, n).astype(np.float64))
        return ((z + rng.standard_normal(n)) * s).astype(np.float32), (rng.random(n) * s).astype(np.float32)
    s = np.exp2(-rng.integers(0, 20, n).astype(np.float64))  # "mixed"
    return ((z + rng.standard_normal(n)) * s).astype(np.float32), ((0.1 + rng.random(n)) * s).astype(np.float32)


@pytest.mark.parametrize("kind", ["normal", "integers", "tiny", "mixed", "wide"])
@pytest.mark.parametrize("n,leaves", [(300, 2), (5003, 7), (70001, 31), (70001, 520)])
def test_renewed_leaves_match_oracle(kind, n, leaves):
    import harness
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(n + leaves)
    X = rng.standard_normal((n, 6))
    X[:, 0] = rng.integers(0, 9, n)
    ds = BinnedDataset.from_dense(X, max_bin=63)
    z = np.where(X[:, 1] > 1.5, 3.0, -0.2) + 0.3 * X[:, 0]
    g, h = _grad(kind, n, rng, z)
    cfg = LearnerConfig(num_leaves=leaves, min_data_in_leaf=5, use_quantized_grad=1, num_grad_quant_bins=16,
                        stochastic_rounding=1, quant_train_renew_leaf=1, min_sum_hessian_in_leaf=1e-9, seed=4, num_threads=2)
    a, b, orc = GpuTreeLearner(ds, cfg), GpuTreeLearner(ds, cfg), harness.OracleLearner(ds, cfg)
    b.set_timing(True)  # one split at a time
    bag = np.nonzero(rng.random(n) < 0.7)[0].astype(np.int32)
    for rows in (None, bag, rng.permutation(bag).astype(np.int32)):
        ra, rb, ro = (x.train(g, h, rows=rows) for x in (a, b, orc))
        assert len(ra[0]) == len(ro[0]) and np.array_equal(ra[0]["threshold"], ro[0]["threshold"])
        assert np.array_equal(ra[1], ro[1]) and np.array_equal(rb[1], ro[1])


def test_renewed_class_trees_match_single_trees():
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(3)
    n, K = 30011, 3
    X = rng.standard_normal((n, 5))
    ds = BinnedDataset.from_dense(X, max_bin=63)
    G, H = (np.stack(v) for v in zip(*(_grad("normal", n, rng, X[:, k]) for k in range(K))))
    cfg = LearnerConfig(num_leaves=40, use_quantized_grad=1, stochastic_rounding=0, quant_train_renew_leaf=1, num_threads=2)
    want = GpuTreeLearner(ds, cfg, num_jobs=K)
    want.set_timing(True)
    x, y = GpuTreeLearner(ds, cfg, num_jobs=K).train_raw(G, H), want.train_raw(G, H)
    assert np.array_equal(x[3], y[3]) and np.array_equal(x[1], y[1])
