"""Grow rounds (several leaves expanded at once, splits committed in the reference's order) against
the same learner growing one split at a time (phase timing on) and against the oracle: quantized
trees bit for bit (records, leaf values, partition, searched leaves' histograms), at the sizes where
the rounds' bookkeeping can go wrong — trees of two leaves up to more than a decision holds, feature
counts around a search group and a tile, leaves of a few rows, chains of splits that need more rounds
than were captured, several class trees, categorical columns and constraints.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _data(n, F, seed, max_bin=255, cat=(), chain=False, nan=0.1):
    from lgbm_gb300 import BinnedDataset
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, F))
    X[:, : F // 3] = rng.integers(0, 16, size=(n, F // 3))
    for c in cat:
        X[:, c] = rng.integers(0, 30, size=n)
    z = np.nan_to_num(X) @ (rng.standard_normal(F) * (rng.random(F) < 0.4)) + 0.5
    if chain:  # every next best leaf is a child of the last split one
        z = np.exp2(np.clip(X[:, -1], -3, 3) * 8.0) / 256.0
    if nan:
        X[rng.random((n, F)) < nan] = np.nan
    ds = BinnedDataset.from_dense(X, max_bin=max_bin, categorical=list(cat))
    g = (0.3 * rng.standard_normal(n) - z).astype(np.float32)
    h = (0.05 + 0.2 * rng.random(n)).astype(np.float32)
    return ds, g, h


def _same(a, b):
    assert int(a[3][0]) == int(b[3][0])
    k = int(a[3][0])
    for name in a[0].dtype.names:
        x, y = a[0][0, :k - 1][name], b[0][0, :k - 1][name]
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f"), name
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


CASES = [
    dict(n=400, F=1, leaves=2), dict(n=3000, F=3, leaves=3), dict(n=5000, F=7, leaves=31),
    dict(n=20000, F=8, leaves=31, max_bin=15), dict(n=20011, F=9, leaves=63, max_bin=63),
    dict(n=30000, F=33, leaves=255), dict(n=3000, F=40, leaves=255, min_data=1), dict(n=60000, F=17, leaves=512),
    dict(n=30000, F=5, leaves=513), dict(n=40000, F=4, leaves=40, chain=True, nan=0.0),
    dict(n=40000, F=12, leaves=100, chain=True, max_bin=63), dict(n=30000, F=20, leaves=31, cat=(0, 7, 19)),
    dict(n=30000, F=24, leaves=63, lambda_l2=3.0, min_gain=0.5), dict(n=30000, F=24, leaves=63, lambda_l1=0.5),
    dict(n=30000, F=24, leaves=63, max_depth=4), dict(n=30000, F=24, leaves=63, quant=0),
    dict(n=30000, F=12, leaves=63, constraints=[[0, 1, 2, 3], [3, 4, 5, 6, 7], [8, 9, 10, 11]]),
]


@pytest.mark.parametrize("c", CASES, ids=lambda c: "-".join("%s%s" % (k, v) for k, v in c.items() if k != "constraints"))
def test_rounds_equal_one_split_at_a_time(c):
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    quant = c.get("quant", 1)
    ds, g, h = _data(c["n"], c["F"], 5, c.get("max_bin", 255), c.get("cat", ()), c.get("chain", False), c.get("nan", 0.1))
    cfg = LearnerConfig(num_leaves=c["leaves"], min_data_in_leaf=c.get("min_data", 20), use_quantized_grad=quant,
                        stochastic_rounding=1, seed=3, num_threads=2, lambda_l2=c.get("lambda_l2", 0.0),
                        lambda_l1=c.get("lambda_l1", 0.0), min_gain_to_split=c.get("min_gain", 0.0),
                        max_depth=c.get("max_depth", -1))
    a, b = GpuTreeLearner(ds, cfg), GpuTreeLearner(ds, cfg)
    b.set_timing(True)  # one split at a time
    if "constraints" in c:
        for x in (a, b):
            x.set_interaction_constraints(c["constraints"])
    rows = np.nonzero(np.random.default_rng(1).random(c["n"]) < 0.8)[0].astype(np.int32)
    for it, r in enumerate((None, rows, None)):
        ra, rb = (x.train_raw(g[None], h[None], rows=r) for x in (a, b))
        if quant:
            _same(ra, rb)
            assert np.array_equal(a.row_leaf(), b.row_leaf())
            for leaf in range(0, int(ra[3][0]) - 2, 7):
                ha, hb = a.leaf_histogram(leaf), b.leaf_histogram(leaf)
                if leaf not in (int(ra[0][0][int(ra[3][0]) - 2]["leaf"]),):  # the last split's children: not searched
                    assert (ha is None) == (hb is None) and (ha is None or np.array_equal(ha, hb))
        else:
            k = int(ra[3][0])
            assert k == int(rb[3][0])
            np.testing.assert_allclose(ra[0][0, :k - 1]["gain"], rb[0][0, :k - 1]["gain"], rtol=1e-6)
            np.testing.assert_allclose(ra[1], rb[1], rtol=1e-6)


@pytest.mark.parametrize("chain", [False, True])
def test_class_trees_and_score_update(chain):
    """Class trees of one call need different numbers of rounds; the device score update comes once,
    after the last of them, in a batch call and in a group."""
    import torch
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig, LearnerGroup, train_batch
    ds, g, h = _data(20000, 10, 9, chain=chain, nan=0.0)
    K, n = 3, 20000
    rng = np.random.default_rng(2)
    G = np.stack([g, (0.2 * rng.standard_normal(n)).astype(np.float32) + 0.1, -g])
    H = np.stack([h, h, h])
    cfg = LearnerConfig(num_leaves=48, use_quantized_grad=1, seed=3, num_threads=2)
    one = GpuTreeLearner(ds, cfg, num_jobs=K)
    one.set_timing(True)
    want = one.train_raw(G, H)
    # the returned leaf values, shrunk as the device update does
    v = want[1] * 0.1
    v[np.abs(v) <= float(np.float32(1e-35))] = 0.0
    score0 = np.stack([v[j][one.row_leaf()[j]] for j in range(K)])
    for form in ("train", "batch", "group"):
        L = GpuTreeLearner(ds, cfg, num_jobs=K)
        score = torch.zeros((K, n), dtype=torch.float64, device="cuda")
        dg, dh = torch.from_numpy(G).cuda(), torch.from_numpy(H).cuda()
        torch.cuda.synchronize()
        if form == "train":
            got = L.train_raw(G, H)
        elif form == "batch":
            got = train_batch([L], [G], [H], shrinkage=0.1, scores=[score.data_ptr()])[0]
        else:
            grp = LearnerGroup([L])
            got = grp.train([dg.data_ptr()], [dh.data_ptr()], shrinkage=0.1, scores=[score.data_ptr()])[0]
        assert np.array_equal(got[3], want[3]) and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
        for j in range(K):
            k = int(want[3][j])
            assert got[0][j, :k - 1].tobytes() == want[0][j, :k - 1].tobytes()
        if form != "train":
            assert np.array_equal(score.cpu().numpy(), score0)


def test_rounds_match_oracle():
    import harness
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    ds, g, h = _data(50000, 30, 11)
    cfg = LearnerConfig(num_leaves=127, use_quantized_grad=1, seed=7, num_threads=2)
    gpu, orc = GpuTreeLearner(ds, cfg), harness.OracleLearner(ds, cfg)
    for _ in range(2):
        a, b = gpu.train(g, h), orc.train(g, h)
        assert len(a[0]) == len(b[0])
        for name in ("leaf", "right_leaf", "inner_feature", "threshold", "left_count", "left_int_sum", "gain"):
            assert np.array_equal(a[0][name], b[0][name]), name
        assert np.array_equal(a[1], b[1]) and np.array_equal(gpu.row_leaf(), orc.row_leaf())
