"""Integer histograms at the ends of their counters: the wide form with every bin of a tile in use,
and a histogram CTA whose hessian sum needs all 32 bits.
"""
import numpy as np
import pytest

from test_gpu_hist_tiles import _learner

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("F", [1, 5, 9, 17, 33, 49])
def test_wide_counters_of_255_bins_match_oracle(F):
    """127 gradient levels fill a packed counter in 511 rows, fewer than a round of the CTA's."""
    import harness
    n = 20000 + F
    ds, L, g, h = _learner(n, F, 255, 127, K=2, leaves=7)
    tree = L.train_raw(g, h)
    for j in range(2):
        rec, values = harness.OracleLearner(ds, L.cfg).train(g[j], h[j])[:2]
        k = int(tree[3][j])
        assert k == len(rec) + 1 and np.any(tree[0][j, 0]["left_int_sum"] != 0)
        for name in ("leaf", "inner_feature", "threshold", "left_count", "left_int_sum", "gain"):
            assert np.array_equal(tree[0][j, :k - 1][name], rec[name]), name
        assert np.array_equal(tree[1][j, :k], values)


@pytest.mark.parametrize("loop_mode", [1, 0])
def test_hessian_sum_of_one_cta_above_31_bits(loop_mode):
    import torch
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig
    n = 17_200_000
    x = (torch.arange(n, device="cuda") % 1000).clamp(max=2).float()
    X = (2.0 - x).reshape(n, 1).contiguous()  # zeros but for two rows in a thousand
    ds = BinnedDataset.from_dense_device(X, bin_construct_sample_cnt=20000)
    assert ds.features[0].most_freq_bin == 0
    L = GpuTreeLearner(ds, LearnerConfig(num_leaves=2, use_quantized_grad=1, num_grad_quant_bins=127,
                                         stochastic_rounding=0, min_gain_to_split=1e12), loop_mode=loop_mode)
    L.set_launch_shape((32, 1, 8, 0, 1))
    g = torch.full((n,), -1.0, device="cuda")
    h = torch.ones(n, device="cuda")
    torch.cuda.synchronize()
    assert int(L.train_raw(g.data_ptr(), h.data_ptr(), on_device=True)[3][0]) == 1
    got = L.leaf_histogram(0)
    rows = np.array([int((X == v).sum()) for v in (0.0, 1.0, 2.0)], dtype=np.int64)
    assert rows[0] * 127 >= 2 ** 31
    assert np.array_equal(got[:, 0], -63 * rows)
    assert np.array_equal(got[:, 1], 127 * rows)
    L.close()
