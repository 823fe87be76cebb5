"""Histograms and row partitions where their inner loops change form, against the oracle bit for bit:
feature counts around the 4, 8, 16 and 32 steps of a tile, 8- and 4-bit bins, the packed and the wide
integer counters; leaf sizes around a CTA's tile of the partition. Float histograms at the same tiles,
with gradients inside and outside the range of the fixed-point sums, against extended-precision sums.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _learner(n, F, max_bin, levels=4, K=1, leaves=3, seed=1):
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, F))
    X[:, ::3] = rng.integers(0, 12, size=(n, len(range(0, F, 3))))
    ds = BinnedDataset.from_dense(X, max_bin=max_bin)
    g = (X[:, 0] - X[:, -1] + rng.standard_normal((K, n))).astype(np.float32)
    h = (0.05 + 0.2 * rng.random((K, n))).astype(np.float32)
    cfg = LearnerConfig(num_leaves=leaves, min_data_in_leaf=1, min_sum_hessian_in_leaf=0.0, use_quantized_grad=1,
                        num_grad_quant_bins=levels, stochastic_rounding=0, num_threads=2)
    return ds, GpuTreeLearner(ds, cfg, num_jobs=K), g, h


@pytest.mark.parametrize("F", [1, 4, 5, 8, 9, 16, 17, 31, 33, 36, 40, 48, 49])
@pytest.mark.parametrize("max_bin,levels", [(255, 4), (15, 4), (63, 64), (255, 254)])
def test_integer_tiles_match_oracle(F, max_bin, levels):
    import harness
    n = 20000 + F
    ds, L, g, h = _learner(n, F, max_bin, levels, K=2, leaves=7)
    tree = L.train_raw(g, h)
    for j in range(2):
        rec, values = harness.OracleLearner(ds, L.cfg).train(g[j], h[j])[:2]
        k = int(tree[3][j])
        assert k == len(rec) + 1
        for name in ("leaf", "inner_feature", "threshold", "left_count", "left_int_sum", "gain"):
            assert np.array_equal(tree[0][j, :k - 1][name], rec[name]), name
        assert np.array_equal(tree[1][j, :k], values)


@pytest.mark.parametrize("n", [100, 255, 256, 257, 1023, 1024, 1025, 2049, 70000])
def test_partition_tiles_match_oracle(n):
    """Each leaf holds the rows that its splits send there, whatever its size and the bagged rows."""
    import harness
    ds, L, g, h = _learner(n, 6, 255, leaves=31)
    orc = harness.OracleLearner(ds, L.cfg)
    bag = np.nonzero(np.random.default_rng(2).random(n) < 0.6)[0].astype(np.int32)
    for rows in (None, bag):
        nl = int(L.train_raw(g, h, rows=rows)[3][0])
        assert nl == len(orc.train(g[0], h[0], rows=rows)[1])
        used = np.arange(n) if rows is None else rows
        assert np.array_equal(L.row_leaf()[used], orc.row_leaf()[used])


# With n rows a fixed-point value has 94 - ceil(log2(n + 1)) bits, 24 of them the mantissa: 55 binary
# orders between the largest and the smallest value for 30011 rows.
_SPAN = 55


@pytest.mark.parametrize("F,max_bin", [(1, 255), (4, 15), (7, 255), (12, 63), (16, 15), (30, 255), (35, 15), (41, 255)])
@pytest.mark.parametrize("const", [False, True])
@pytest.mark.parametrize("values", ["normal", "spread", "edge", "beyond", "wide"])
def test_float_tiles_match_extended_sums(F, max_bin, const, values):
    """A root whose split gains too little keeps its histogram. Fixed-point sums are exact per CTA; then each of at
    most 152 CTAs' sums is rounded once and added with one more rounding: 304 * 2^-53 < 4e-14 of the bin's
    mass. fp32 pairs (values beyond the range) keep the bound of the leaf-histogram comparison, 1e-10."""
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    n = 30011
    rng = np.random.default_rng(F)
    X = rng.standard_normal((n, F))
    X[:, ::3] = rng.integers(0, 12, size=(n, len(range(0, F, 3))))
    ds = BinnedDataset.from_dense(X, max_bin=max_bin)
    z = rng.standard_normal((2, n))
    z[:, rng.random(n) < 0.1] = 0.0
    if values == "spread":
        z = np.ldexp(z, -rng.integers(0, 30, size=z.shape))
    elif values in ("edge", "beyond"):  # magnitudes in [1, 2), a few at the far end of the range
        z = np.sign(z) * (1.0 + rng.random(z.shape))
        z[:, rng.random(n) < 0.05] *= 2.0 ** -(_SPAN if values == "edge" else _SPAN + 1)
    elif values == "wide":
        z = np.ldexp(z, -rng.integers(0, 110, size=z.shape))
    g, h = z[0].astype(np.float32), np.abs(z[1]).astype(np.float32)
    if const:
        h[:] = 0.7
    cfg = LearnerConfig(num_leaves=2, min_gain_to_split=1e300, use_quantized_grad=0,
                        is_constant_hessian=const, num_threads=2)
    L = GpuTreeLearner(ds, cfg)
    assert len(L.train(g, h)[1]) == 1
    hist = L.leaf_histogram(0)
    tol = 4e-14 if values in ("normal", "spread", "edge") else 1e-10
    at = 0
    for j, fi in enumerate(ds.features):
        col = np.asarray(ds.bins[j], dtype=np.int64)
        for c, v in enumerate((g, h)):
            want = np.zeros(fi.group_bins, np.longdouble)
            mass = np.zeros(fi.group_bins, np.longdouble)
            np.add.at(want, col, v.astype(np.longdouble))
            np.add.at(mass, col, np.abs(v).astype(np.longdouble))
            for b in range(1, fi.group_bins):
                if not (fi.most_freq_bin > 0 and b == fi.most_freq_bin + 1):  # that one is the total minus the others
                    assert abs(hist[at + b, c] - want[b]) <= tol * mass[b], (j, c, b)
        at += fi.group_bins
