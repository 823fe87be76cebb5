"""Device gradients where results lie at and beside powers of two (scores near zero: a binary hessian of
0.25, K equal classes): the f64 arithmetic's result rounded to fp32, as quickly as elsewhere.
"""
import numpy as np
import pytest

from test_gpu_row_kernels import _equal, _gradients, _learner

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _time(L, kind, s, label):
    import torch
    st = torch.cuda.ExternalStream(L.stream())
    t = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        L.objective_gradients(kind, s.data_ptr(), label.data_ptr())
        b.record(st)
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b))
    return float(np.median(t))


def _scores(K, n, scale):
    rng = np.random.default_rng(3)
    s = rng.standard_normal((K, n)) * scale
    s[:, ::3] = 0.0  # equal classes
    return s


@pytest.mark.parametrize("scale", [0.0, 1e-9, 1e-6, 1e-5, 1e-4, 3e-4, 1e-3])
def test_binary_gradients_beside_a_quarter(scale):
    import torch
    n = 1 << 20
    L = _learner(n)
    s = torch.from_numpy(_scores(1, n, scale)[0]).cuda()
    label = (torch.arange(n, device="cuda") % 3 == 1).float()
    torch.cuda.synchronize()
    g, h = _gradients(L, 1, s, label)
    lab = torch.where(label > 0, 1.0, -1.0).double()
    resp = -lab / (1.0 + torch.exp(lab * s))
    ar = resp.abs()
    _equal(g, resp.float())
    _equal(h, (ar * (1.0 - ar)).float())
    ordinary = torch.from_numpy(np.random.default_rng(1).standard_normal(n)).cuda()
    torch.cuda.synchronize()
    assert _time(L, 1, s, label) < 1.8 * _time(L, 1, ordinary, label) + 0.01


@pytest.mark.parametrize("K", [2, 3, 4, 8, 32])
@pytest.mark.parametrize("scale", [0.0, 1e-6, 1e-4])
def test_softmax_gradients_beside_equal_classes(K, scale):
    import torch
    n = 100000
    L = _learner(n, K)
    s = torch.from_numpy(_scores(K, n, scale)).cuda()
    label = (torch.arange(n, device="cuda") % K).float()
    torch.cuda.synchronize()
    g, h = (x.view(K, n) for x in _gradients(L, 2, s, label))
    rec = torch.exp(s - s.max(0).values)
    wsum = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(K):
        wsum = wsum + rec[k]
    factor = K / (K - 1.0)
    for k in range(K):
        p = rec[k] / wsum
        _equal(g[k], torch.where(label == k, p - 1.0, p).float())
        _equal(h[k], ((factor * p) * (1.0 - p)).float())
    ordinary = torch.from_numpy(np.random.default_rng(1).standard_normal((K, n))).cuda()
    torch.cuda.synchronize()
    assert _time(L, 2, s, label) < 1.6 * _time(L, 2, ordinary, label) + 0.01
