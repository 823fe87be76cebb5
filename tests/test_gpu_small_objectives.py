"""Device gradients of values far below 1: scores, labels, the sigmoid and label weights down to the
smallest fp32 numbers give the f64 arithmetic's result rounded to fp32 (torch's f64 on the device).
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


def _mixed(n, seed, scale):
    """N(0, 1) times 10^-8 .. 1 of the scale, with zeros."""
    import torch
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n) * scale * 10.0 ** rng.uniform(-8, 0, n)
    x[rng.random(n) < 0.1] = 0.0
    return torch.from_numpy(x).cuda()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("scale", [1e-3, 1e-10, 1e-12, 1e-17, 1e-18, 1e-20, 1e-30, 1e-37])
def test_l2_gradients_of_small_values(scale, weighted):
    import torch
    n = 50021
    L = _learner(n)
    s = _mixed(n, 1, scale)
    label = _mixed(n, 2, scale).float()
    label[::5] = s[::5].float()
    label[1::5] = (s[1::5] * 0.25).float()
    known = torch.tensor([[5e-19, 1.6e-19], [8e-19, 1e-20], [1e-20, 1e-20], [5e-19, 1e-12]], dtype=torch.float64)
    s[:4], label[:4] = known[:, 0].cuda(), known[:, 1].float().cuda()
    w = torch.rand(n, device="cuda") + 0.5
    if weighted:
        L.set_objective_weights(w.data_ptr())
    torch.cuda.synchronize()
    g, h = _gradients(L, 0, s, label)
    want = (s - label.double()).float()
    _equal(g, want * w if weighted else want)
    _equal(h, w if weighted else torch.ones_like(w))


@pytest.mark.parametrize("sigmoid,lw", [(1.0, (1.0, 1.0)), (1e-20, (1.0, 1.0)), (1e-12, (1.0, 1.0)),
                                        (1.0, (1e-20, 1.0)), (1.0, (1.0, 3e-25)), (1e-19, (1e-19, 1e-3))])
@pytest.mark.parametrize("scale", [1.0, 1e-18, 1e-30])
def test_binary_gradients_of_small_values(sigmoid, lw, scale):
    import torch
    n = 50021
    L = _learner(n)
    s = _mixed(n, 3, scale)
    label = (torch.arange(n, device="cuda") % 3 == 0).float()
    L.set_objective_weights(0, *lw)
    torch.cuda.synchronize()
    g, h = _gradients(L, 1, s, label, sigmoid)
    lab = torch.where(label > 0, 1.0, -1.0).double()
    lwr = torch.tensor(lw, dtype=torch.float64, device="cuda")[(label > 0).long()]
    resp = (-lab * sigmoid) / (1.0 + torch.exp(lab * sigmoid * s))
    ar = resp.abs()
    _equal(g, (resp * lwr).float())
    _equal(h, ((ar * (sigmoid - ar)) * lwr).float())


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e-36, 1e-38, 1e-41])
def test_gradients_of_small_row_weights(K, scale):
    """Products down to the subnormal fp32 numbers, and rows of no weight."""
    import torch
    n = 100003
    L = _learner(n, K)
    rng = np.random.default_rng(7)
    s = torch.from_numpy(rng.standard_normal((K, n)) * 4.0).cuda()
    label = torch.from_numpy(rng.integers(0, max(K, 2), n)).float().cuda()
    w = (torch.rand(n, device="cuda") + 0.5) * scale
    w[::7] = 0.0
    L.set_objective_weights(w.data_ptr())
    torch.cuda.synchronize()
    wd = w.double()
    if K == 1:
        g, h = _gradients(L, 1, s, label)
        lab = torch.where(label > 0, 1.0, -1.0).double()
        resp = -lab / (1.0 + torch.exp(lab * s[0]))
        ar = resp.abs()
        _equal(g, (resp * wd).float())
        _equal(h, ((ar * (1.0 - ar)) * wd).float())
        return
    g, h = (x.view(K, n) for x in _gradients(L, 2, s, label))
    rec = torch.exp(s - s.max(0).values)
    wsum = rec[0] + rec[1] + rec[2]
    for k in range(K):
        p = rec[k] / wsum
        _equal(g[k], (torch.where(label == k, p - 1.0, p) * wd).float())
        _equal(h[k], ((K / (K - 1.0) * p) * (1.0 - p) * wd).float())
