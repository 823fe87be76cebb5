"""The row-wise kernels around a tree: device gradients computed as fp32 pairs equal the f64 arithmetic
rounded to fp32 (torch's f64 on the device, operation for operation), discretization next to whole
numbers equals the oracle's, and the score update and row lookup reach every row at the sizes where
their grids change.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _learner(n, K=1, **cfg):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(0)
    ds = BinnedDataset.from_dense(rng.standard_normal((n, 2)), bin_construct_sample_cnt=2000)
    return GpuTreeLearner(ds, LearnerConfig(num_leaves=4, **cfg), num_jobs=K)


def _gradients(L, kind, score, label, sigmoid=1.0):
    import torch
    L.objective_gradients(kind, score.data_ptr(), label.data_ptr(), sigmoid)
    torch.cuda.synchronize()
    g, h = L.gradient_buffers()

    class View:
        def __init__(self, ptr):
            self.__cuda_array_interface__ = {"shape": (score.numel(),), "typestr": "<f4", "data": (ptr, False),
                                             "version": 3, "strides": None}
    return torch.as_tensor(View(g), device="cuda").clone(), torch.as_tensor(View(h), device="cuda").clone()


def _scores(n, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    s[: n // 4] *= 8.0
    s[n // 4: n // 3] *= 1e-6
    s[n // 3: n // 3 + n // 20] *= 200.0
    edge = torch.tensor([0.0, -0.0, 1.0, -1.0, 59.999, 60.0, 60.001, -60.0, -61.0, 700.0, -700.0, 800.0, 1e-300, 1e300,
                         float("inf"), float("-inf"), 0.6931471805599453, 0.010830424696249145], dtype=torch.float64)
    s[: len(edge)] = edge.cuda()
    return s


def _equal(a, b):
    import torch
    same = (a == b) | (torch.isnan(a) & torch.isnan(b))
    assert bool(same.all()), (int((~same).sum()), a[~same][:5], b[~same][:5])


@pytest.mark.parametrize("weighted", [False, True])
def test_l2_gradients_equal_f64(weighted):
    import torch
    n = 200003
    L = _learner(n)
    s = _scores(n, 1)
    label = (s + 0.1 * _scores(n, 2)).float()
    label[::3] = s[::3].float()
    w = torch.rand(n, device="cuda") + 0.5
    if weighted:
        L.set_objective_weights(w.data_ptr())
    torch.cuda.synchronize()
    g, h = _gradients(L, 0, s, label)
    want = (s - label.double()).float()
    _equal(g, want * w if weighted else want)
    _equal(h, w if weighted else torch.ones_like(w))


@pytest.mark.parametrize("sigmoid,lw,weighted", [(1.0, (1.0, 1.0), False), (0.7, (1.0, 2.5), False),
                                                 (1.0, (0.3, 1.7), True), (2.0, (1.0, 1.0), True)])
def test_binary_gradients_equal_f64(sigmoid, lw, weighted):
    import torch
    n = 400009
    L = _learner(n)
    s = _scores(n, 3)
    label = (torch.rand(n, device="cuda") < 0.4).float()
    w = torch.rand(n, device="cuda") + 0.5
    L.set_objective_weights(w.data_ptr() if weighted else 0, *lw)
    torch.cuda.synchronize()
    g, h = _gradients(L, 1, s, label, sigmoid)
    lab = torch.where(label > 0, 1.0, -1.0).double()
    lwr = torch.tensor(lw, dtype=torch.float64, device="cuda")[(label > 0).long()]
    t = -lab * sigmoid
    resp = t / (1.0 + torch.exp(lab * sigmoid * s))
    ar = resp.abs()
    q = ar * (sigmoid - ar)
    wd = w.double() if weighted else None
    _equal(g, (resp * lwr * wd).float() if weighted else (resp * lwr).float())
    _equal(h, (q * lwr * wd).float() if weighted else (q * lwr).float())


@pytest.mark.parametrize("K,weighted", [(2, False), (3, True), (10, False), (32, False)])
def test_softmax_gradients_equal_f64(K, weighted):
    import torch
    n = 100003
    L = _learner(n, K)
    s = torch.stack([_scores(n, 10 + k).clamp(-1e3, 1e3) for k in range(K)]).contiguous()
    s[:, n // 2:] *= 0.5
    label = torch.randint(0, K, (n,), device="cuda").float()
    w = torch.rand(n, device="cuda") + 0.5
    L.set_objective_weights(w.data_ptr() if weighted else 0)
    torch.cuda.synchronize()
    g, h = (x.view(K, n) for x in _gradients(L, 2, s, label))
    rec = torch.exp(s - s.max(0).values)
    wsum = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(K):
        wsum = wsum + rec[k]
    factor = K / (K - 1.0)
    for k in range(K):
        p = rec[k] / wsum
        gi = torch.where(label == k, p - 1.0, p)
        hi = (factor * p) * (1.0 - p)
        wd = w.double()
        _equal(g[k], (gi * wd).float() if weighted else gi.float())
        _equal(h[k], (hi * wd).float() if weighted else hi.float())


@pytest.mark.parametrize("stochastic,bins", [(0, 4), (1, 4), (1, 16), (0, 127)])
def test_discretization_next_to_whole_numbers(stochastic, bins):
    """Gradients on exact multiples of the scale and of half of it, and one fp32 step either side."""
    import harness
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    n = 30011
    rng = np.random.default_rng(4)
    ds = BinnedDataset.from_dense(rng.standard_normal((n, 4)))
    k = rng.integers(-bins // 2, bins // 2 + 1, n)
    g = (k + 0.5 * rng.integers(0, 2, n)).astype(np.float32)
    g = np.where(rng.random(n) < 0.3, np.nextafter(g, np.float32(9e9)), g)
    g = np.clip(g, -(bins // 2), bins // 2).astype(np.float32)
    g[0] = bins // 2
    h = (rng.integers(0, 2 * bins + 1, n) * 0.5).astype(np.float32)
    h[1] = bins
    cfg = LearnerConfig(num_leaves=31, use_quantized_grad=1, num_grad_quant_bins=bins, stochastic_rounding=stochastic,
                        seed=5, num_threads=2)
    gpu, orc = GpuTreeLearner(ds, cfg), harness.OracleLearner(ds, cfg)
    rows = np.sort(rng.choice(n, n // 2, replace=False)).astype(np.int32)
    for r in (None, rows, None):
        a, b = gpu.train(g, h, r), orc.train(g, h, r)
        assert len(a[0]) == len(b[0]) > 0
        for name in ("inner_feature", "threshold", "left_count", "left_int_sum", "right_int_sum"):
            assert np.array_equal(a[0][name], b[0][name]), name
        assert np.array_equal(a[1], b[1])


@pytest.mark.parametrize("n", [255, 256, 257, 5001, 311296, 311297])
def test_score_update_reaches_every_row(n):
    import torch
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 3))
    ds = BinnedDataset.from_dense(X, min_data_in_leaf=1, feature_pre_filter=False)
    L = GpuTreeLearner(ds, LearnerConfig(num_leaves=300 if n > 5000 else 31, min_data_in_leaf=1, use_quantized_grad=1))
    g, h = (X[:, 0] + 0.1 * X[:, 1]).astype(np.float32), np.ones(n, np.float32)
    rows = np.nonzero(rng.random(n) < 0.7)[0].astype(np.int32)
    for r in (None, rows):
        out = L.train_raw(g[None], h[None], rows=r)
        leaf = L.row_leaf()
        bagged = np.ones(n, bool) if r is None else np.isin(np.arange(n), r)
        assert np.array_equal(leaf >= 0, bagged)
        counts = np.bincount(leaf[leaf >= 0], minlength=int(out[3][0]))
        assert counts.min() > 0 and counts.sum() == bagged.sum()
        score = torch.from_numpy(rng.standard_normal(n)).cuda()
        want = score.cpu().numpy().copy()
        want[bagged] += out[1][0][leaf[bagged]]
        torch.cuda.synchronize()
        L.add_prediction_to_score(out[1], score.data_ptr(), on_device=True)
        assert np.array_equal(score.cpu().numpy(), want)
