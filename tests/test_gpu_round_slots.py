"""Histogram slots of grow rounds: an expanded leaf's slot goes to its larger child, and its own
histogram is still there to be asked for.
"""
import numpy as np
import pytest

from test_gpu_rounds import _data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("c", [dict(F=4, leaves=31), dict(F=40, leaves=63), dict(F=40, leaves=255, max_bin=63),
                               dict(F=20, leaves=63, cat=(0, 7, 19)), dict(F=12, leaves=40, lambda_l1=0.5),
                               dict(F=24, leaves=63, max_depth=5), dict(F=24, leaves=63, mask=True),
                               dict(F=24, leaves=63, quant=0), dict(F=8, leaves=63, quant=0, max_bin=31)],
                         ids=lambda c: "-".join("%s%s" % kv for kv in c.items()))
def test_every_leaf_keeps_its_histogram(c):
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    quant = c.get("quant", 1)
    ds, g, h = _data(30000, c["F"], 3, c.get("max_bin", 255), c.get("cat", ()), nan=0.1 if quant else 0.0)
    cfg = LearnerConfig(num_leaves=c["leaves"], use_quantized_grad=quant, seed=3, num_threads=2,
                        lambda_l1=c.get("lambda_l1", 0.0), max_depth=c.get("max_depth", -1))
    a, b = GpuTreeLearner(ds, cfg), GpuTreeLearner(ds, cfg)
    b.set_timing(True)  # one split at a time
    if c.get("mask"):
        for x in (a, b):
            x.set_feature_mask(np.arange(c["F"]) % 3 != 1)
    ra, rb = (x.train_raw(g[None], h[None]) for x in (a, b))
    k = int(ra[3][0])
    assert k == int(rb[3][0]) > 3
    last = ra[0][0, k - 2]
    mass = float(np.abs(g).sum())
    compared = 0
    for leaf in range(k):
        if leaf in (int(last["leaf"]), int(last["right_leaf"])):  # the last split's children: not searched
            continue
        ha, hb = a.leaf_histogram(leaf), b.leaf_histogram(leaf)
        assert (ha is None) == (hb is None)
        if ha is None:
            continue
        compared += 1
        if quant:
            assert np.array_equal(ha, hb), leaf
        else:  # sums of doubles in another order, and a subtraction taken back
            np.testing.assert_allclose(ha, hb, rtol=0, atol=64 * 2.0 ** -53 * mass)
    assert compared >= (k - 2) // 2 or c.get("max_depth")


def test_device_memory_is_near_one_slot_a_leaf():
    import torch
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    ds, g, h = _data(3000, 512, 4, nan=0.0)
    slot = 16 * 256 * 32 * 16  # tiles x bins x features x (gradient, hessian)
    assert max(f.group_bins for f in ds.features) > 248
    GpuTreeLearner(ds, LearnerConfig(num_leaves=4)).train(g, h)  # the library's own startup
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    L = GpuTreeLearner(ds, LearnerConfig(num_leaves=255))
    used = before - torch.cuda.mem_get_info()[0]
    assert used <= 1.35 * 255 * slot, (used, 255 * slot)
    L.close()


@pytest.mark.parametrize("quant", [1, 0])
def test_learner_without_room_for_rounds_grows_one_split_at_a_time(quant):
    """With less free memory than a learner with grow rounds takes, but enough for one without, creation
    succeeds and the trees are the same."""
    import torch
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    ds, g, h = _data(4000, 2000, 6, nan=0.0)
    cfg = LearnerConfig(num_leaves=255, use_quantized_grad=quant, seed=2, num_threads=2)
    GpuTreeLearner(ds, cfg).train(g, h)  # the library's own startup
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    a = GpuTreeLearner(ds, cfg)
    used = before - torch.cuda.mem_get_info()[0]
    want = a.train(g, h)
    a.close()
    held = torch.empty(torch.cuda.mem_get_info()[0] - used + (96 << 20), dtype=torch.uint8, device="cuda")
    b = GpuTreeLearner(ds, cfg)
    left = torch.cuda.mem_get_info()[0]
    del held
    torch.cuda.empty_cache()
    assert left < used
    got = b.train(g, h)
    assert len(got[0]) == len(want[0])
    if quant:
        assert got[0].tobytes() == want[0].tobytes() and np.array_equal(got[1], want[1])
    else:
        np.testing.assert_allclose(got[0]["gain"], want[0]["gain"], rtol=1e-6)
    b.close()


@pytest.mark.parametrize("timed", [False, True])
def test_root_that_is_not_searched_has_no_histogram(timed):
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig
    ds, g, h = _data(500, 4, 8)
    L = GpuTreeLearner(ds, LearnerConfig(num_leaves=31, use_quantized_grad=1, min_data_in_leaf=60))
    L.set_timing(timed)
    for rows, searched in ((None, True), (np.arange(0, 110, dtype=np.int32), False), (None, True)):
        assert len(L.train(g, h, rows)[1]) == 1 or searched
        assert (L.leaf_histogram(0) is not None) == searched
    L.close()
