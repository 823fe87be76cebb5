"""Device binning where its bucketed search can go wrong, against numpy's searchsorted over the bin
mappers' bounds: bounds crowded into one bucket, far from zero, spread over many orders of magnitude
or at the ends of the range, values on the bounds and next to them, infinities, NaN, few bounds, row
counts around a tile and a store word.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows", [1, 255, 256, 259, 5003])
@pytest.mark.parametrize("max_bin", [3, 15, 255])
def test_bins_match_searchsorted(dtype, rows, max_bin):
    import torch
    from lgbm_gb300 import BinnedDataset
    rng = np.random.default_rng(max_bin)
    n = 6000
    u = rng.standard_normal(n)
    cols = [u, 1e6 + 1e-2 * u, np.exp(4 * u), np.where(rng.random(n) < 0.9, 1e-3 * u, 1e5 * u),
            np.sign(u) * np.exp2(60 * rng.random(n)), 1e-38 * u, 1e38 * np.tanh(u), np.sign(u) * 1e-30 * np.exp(9 * u),
            rng.integers(0, 3, n).astype(float), rng.integers(-40, 200, n).astype(float),
            np.where(rng.random(n) < 0.2, np.nan, u), np.where(rng.random(n) < 0.2, np.nan, np.exp(8 * u)),
            np.where(rng.random(n) < 0.5, 0.0, u), np.where(rng.random(n) < 0.6, -2.0, u), u ** 9, 1.0 / u, -np.exp(5 * u), u ** 3, 0.5 - u]
    X = np.stack(cols, axis=1).astype(dtype)
    ds = BinnedDataset.from_dense(X.astype(np.float64), max_bin=max_bin)
    assert ds.num_features > 16  # more than one group of features
    probe = X[rng.integers(0, n, rows)]
    for fi in ds.features:  # on and next to the bounds
        b = fi.upper_bounds[np.isfinite(fi.upper_bounds)]
        if len(b):
            at = rng.random(rows) < 0.5
            with np.errstate(over="ignore"):
                pick = rng.choice(b, rows).astype(dtype)
            near = np.nextafter(pick, rng.choice([-np.inf, np.inf], rows).astype(dtype))
            probe[at, fi.real] = np.where(rng.random(rows) < 0.5, pick, near)[at]
    odd = rng.random(probe.shape)
    for k, v in enumerate((np.inf, -np.inf, np.nan, 0.0, -0.0)):
        probe[(odd >= 0.01 * k) & (odd < 0.01 * (k + 1))] = v
    got = ds.bin_like_device(torch.from_numpy(probe).cuda()).cpu().numpy()
    for j, fi in enumerate(ds.features):
        v = probe[:, fi.real].astype(np.float64)
        nan_bin = fi.missing_type == 2
        searched = fi.upper_bounds[:fi.num_bin - 1 - nan_bin]
        want = np.searchsorted(searched, np.where(np.isnan(v), 0.0, v), side="left")
        if nan_bin:
            want = np.where(np.isnan(v), fi.num_bin - 1, want)
        want = np.where(want == fi.most_freq_bin, 0, want + (fi.most_freq_bin != 0))
        assert np.array_equal(got[j], want), j
