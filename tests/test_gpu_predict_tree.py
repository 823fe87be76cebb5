"""Held-out rows through one tree: both forms of the walk (columns staged in shared memory up to 96 of
them, global loads above) against a numpy replay of the routing rule, over missing types, most
frequent bins, two-valued and categorical columns, odd row counts and unaligned bins. A score is one
addition of a leaf value, so the results are equal.
"""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _left(fi, gbins, thr, dleft, b):
    """data_partition.rs:299-410 for stored bins b of a feature of its own group."""
    mfb, top = fi.most_freq_bin, gbins - 1
    zero, na = fi.missing_type == 1, fi.missing_type == 2
    mfb_zero, mfb_na = zero and fi.default_bin == mfb, na and top == mfb + 1 and mfb > 0
    shift = 0 if mfb == 0 else 1
    th, zbin = thr + shift, fi.default_bin + shift
    miss = (zero or na) and dleft
    rest = np.full(b.shape, miss if (mfb_zero or mfb_na) else mfb <= thr)
    if top > 1:
        out = np.where(b == 0, rest, b <= th)
        if na and not mfb_na:
            out = np.where(b == top, miss, out)
    else:
        out = np.where(b == top, miss if (na and not mfb_na) else top <= th, rest)
    if zero and not mfb_zero:
        out = np.where(b == zbin, miss, out)
    return out


@pytest.mark.parametrize("F,leaves,m,offset", [(1, 2, 1, 0), (8, 31, 497, 1), (40, 255, 5003, 7), (96, 255, 992, 0),
                                               (97, 300, 2011, 15), (140, 600, 3000, 3)])
@pytest.mark.parametrize("missing", ["none", "nan", "zero"])
def test_predict_matches_replay(F, leaves, m, offset, missing):
    import torch
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    rng = np.random.default_rng(F + leaves)
    n = 3000
    X = rng.standard_normal((n, F))
    X[:, 1::4] = rng.random((n, len(range(1, F, 4)))) < 0.3          # two values
    X[:, 2::4] = rng.choice([-2.0, 0.0, 3.0, 5.0], p=[0.1, 0.2, 0.6, 0.1], size=(n, len(range(2, F, 4))))
    cat = list(range(3, F, 4))
    X[:, 3::4] = rng.integers(0, 40, size=(n, len(cat)))
    if missing == "nan":
        num = [c for c in range(F) if c not in cat]
        X[np.ix_(np.arange(n), num)] = np.where(rng.random((n, len(num))) < 0.2, np.nan, X[:, num])
    ds = BinnedDataset.from_dense(X, zero_as_missing=missing == "zero", categorical=cat)
    L = GpuTreeLearner(ds, LearnerConfig(num_leaves=max(leaves, 2)))
    nf, ni = ds.num_features, leaves - 1
    gb = np.array([fi.group_bins for fi in ds.features])
    bins = (rng.integers(0, 256, size=(nf, m)) % np.where(rng.random((nf, m)) < 0.95, gb[:, None], 256)).astype(np.uint8)
    # a random tree: a random leaf is split each time
    lc, rc = np.zeros(ni, np.int32), np.zeros(ni, np.int32)
    at = [None]
    for i in range(ni):
        k = int(rng.integers(0, len(at)))
        if at[k] is not None:
            at[k][0][at[k][1]] = i
        at[k] = (lc, i)
        at.append((rc, i))
    for j, (arr, i) in enumerate(at):
        arr[i] = ~j
    sf = np.concatenate([np.arange(nf), rng.integers(0, nf, size=ni)])[:ni].astype(np.int32)
    is_cat = np.array([ds.features[f].categorical for f in sf])
    thr = np.array([rng.integers(0, ds.features[f].num_bin) for f in sf]).astype(np.uint32)
    dleft = rng.random(ni) < 0.5
    bits = rng.integers(0, 1 << 32, size=(ni, 8), dtype=np.uint64).astype(np.uint32)
    tree = SimpleNamespace(num_leaves=leaves, left_child=lc, right_child=rc, split_feature_inner=sf, threshold_in_bin=thr,
                           decision_type=(is_cat * 1 + dleft * 2).astype(np.int8), cat_bin_bits=bits,
                           leaf_value=rng.standard_normal(leaves))
    node = np.zeros(m, np.int64)
    for _ in range(leaves):
        for i in np.unique(node[node >= 0]):
            r = np.flatnonzero(node == i)
            fi, b = ds.features[sf[i]], bins[sf[i], r].astype(np.int64)
            if is_cat[i]:
                pos = np.where(b == 0, fi.most_freq_bin, b - 1 + (fi.most_freq_bin == 0))
                inside = (pos < 256) & (b < fi.group_bins) & ((b != 0) | (fi.most_freq_bin > 0))
                pos = np.minimum(pos, 255)
                left = inside & (((bits[i][pos >> 5] >> (pos & 31).astype(np.uint32)) & 1) != 0)
            else:
                left = _left(fi, fi.group_bins, int(thr[i]), bool(dleft[i]), b)
            node[r] = np.where(left, lc[i], rc[i])
    start = rng.standard_normal(m)
    buf = torch.zeros(nf * m + 32, dtype=torch.uint8, device="cuda")
    buf[offset:offset + nf * m] = torch.from_numpy(bins.ravel()).cuda()
    score = torch.from_numpy(start).cuda()
    torch.cuda.synchronize()
    L.predict_add(tree, buf.data_ptr() + offset, m, score.data_ptr())
    assert np.array_equal(score.cpu().numpy(), start + tree.leaf_value[~node])
    one = SimpleNamespace(num_leaves=1, left_child=lc, right_child=rc, split_feature_inner=sf, threshold_in_bin=thr,
                          decision_type=tree.decision_type, leaf_value=np.array([0.25]))
    L.predict_add(one, buf.data_ptr() + offset, m, score.data_ptr())
    assert np.array_equal(score.cpu().numpy(), (start + tree.leaf_value[~node]) + 0.25)
