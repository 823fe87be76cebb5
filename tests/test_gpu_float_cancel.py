"""The float search where large positive and negative bins cancel: the f64 sums of the thresholds round
differently from their exact values, and the split goes by the f64 sums, added in the search's order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINS = 255


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _case(seed, big):
    """One feature of 255 bins (bin 0 the most frequent, not in the slice): 400 rows in bin 0, one of
    almost no hessian in each of the others, 100 more in bin 252, and +big / -big in bins 253 and 254, whose
    rows are too few to split off. Every sum but those across +big is exact in f64, the root's too (the
    two big rows are 16 lanes apart)."""
    rng = np.random.default_rng(seed)
    unit = 2.0 ** -20
    bins = np.concatenate([[253], np.zeros(15), [254], np.zeros(385), np.arange(1, 253), np.full(99, 252)]).astype(np.uint8)
    n = len(bins)
    g, h = np.zeros(n), np.full(n, 2.0 ** -24)
    h[bins == 0] = 1.0
    h[-100:] = 1.0
    g[0], g[16] = big, -big
    inner = (bins > 0) & (bins < 252)
    above = rng.integers(0, 3, int(inner.sum()))  # the inner bins' sum from each on, in units
    above[1::2] = 0  # the top warp's odd lanes add across +big
    g[inner] = (above - np.append(above[1:], 0)) * unit
    g[-1] = 0.5 + (8 * rng.integers(0, 8) + rng.integers(4, 8)) * unit
    return bins, g.astype(np.float32), h.astype(np.float32)


def _f64_choice(bins, g, h):
    """The reverse scan as the search adds it: within a warp of 32 bins by doubling, then the warps above
    from the top down."""
    sg, sh = (np.bincount(bins, w.astype(np.float64), BINS)[1:] for w in (g, h))
    total_g, total_h = float(np.sum(g.astype(np.float64)[np.argsort(-np.abs(g), kind="stable")])), float(h.astype(np.float64).sum())
    sum_h = total_h + 2 * float(np.float32(1e-15))
    eps = float(np.float32(1e-15))
    suffix = []
    for v in (sg, sh):
        x = np.zeros(256)
        x[:len(v)] = v
        x = x.reshape(8, 32)
        for o in (1, 2, 4, 8, 16):
            y = x.copy()
            y[:, :32 - o] += x[:, o:]
            x = y
        above = np.zeros(8)
        for w in range(8):
            a = 0.0
            for i in range(7, w, -1):
                a += x[i, 0]
            above[w] = a
        suffix.append((x + above[:, None]).reshape(-1)[:len(v)])
    rg, rh = suffix[0], eps + suffix[1]
    best, at = -np.inf, -1
    for t in range(len(rg) - 1, -1, -1):
        cf = len(bins) / sum_h
        cnt = np.floor(np.bincount(bins, h.astype(np.float64), BINS)[1:] * cf + 0.5)[t:].sum()
        if cnt < 20 or rh[t] < 1e-3:
            continue
        if len(bins) - cnt < 20 or sum_h - rh[t] < 1e-3:
            break
        lg, lh = total_g - rg[t], sum_h - rh[t]
        gain = lg * lg / lh + rg[t] * rg[t] / rh[t]
        if gain > best:
            best, at = gain, t
    return at


@pytest.mark.parametrize("rounds", [True, False])
@pytest.mark.parametrize("big", [0.0, 2.0 ** 20, 2.0 ** 34, 2.0 ** 35])
def test_threshold_is_the_f64_sums_choice(big, rounds):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    from lgbm_gb300.dataset import FeatureInfo
    f = FeatureInfo()
    f.real, f.num_bin, f.missing_type, f.default_bin, f.most_freq_bin, f.penalty = 0, BINS, 0, 0, 0, 1.0
    f.upper_bounds = np.append(np.arange(BINS - 1) + 0.5, np.inf)
    for seed in range(12):
        bins, g, h = _case(seed, big)
        ds = BinnedDataset(bins[None, :].copy(), [f], 1)
        L = GpuTreeLearner(ds, LearnerConfig(num_leaves=2, fused_madd=1))
        L.set_timing(not rounds)
        rec = L.train(g, h)[0]
        L.close()
        assert len(rec) == 1
        assert int(rec[0]["threshold"]) == _f64_choice(bins, g, h), seed
