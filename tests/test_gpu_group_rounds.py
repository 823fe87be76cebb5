"""A learner group's launch policy is timed on whole iterations: members whose trees need more rounds
than the captured iteration holds have them grown to the end.
"""
import pytest

from test_gpu_rounds import _data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_group_autotune_finishes_its_trial_trees():
    import torch
    from lgbm_gb300 import GpuTreeLearner, LearnerConfig, LearnerGroup
    members, grads = [], []
    for i, (F, chain) in enumerate(((4, True), (10, False))):
        ds, g, h = _data(40000, F, i, chain=chain, nan=0.0)
        members.append(GpuTreeLearner(ds, LearnerConfig(num_leaves=255, min_data_in_leaf=1, seed=3)))
        grads.append((torch.from_numpy(g).cuda(), torch.from_numpy(h).cuda()))
    torch.cuda.synchronize()
    group = LearnerGroup(members)
    group.autotune([g.data_ptr() for g, _ in grads], [h.data_ptr() for _, h in grads], trials=1)
    # a trial tree that was left unfinished has no leaf with a histogram yet
    assert all(L.leaf_histogram(0) is not None for L in members)
    group.close()
    for L in members:
        L.close()


def test_batch_calls_run_side_by_side():
    """The learners of a batch call share all of the device's queues: sixteen small ones take less than three
    times as long as four (3.4 times when only half of the queues are in use)."""
    import time

    import numpy as np
    import torch
    from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig, train_batch
    n = 2000
    rng = np.random.default_rng(1)
    X = rng.standard_normal((n, 10))
    ds = BinnedDataset.from_dense(X)
    g = torch.from_numpy((X[:, 0] + 0.3 * rng.standard_normal(n)).astype(np.float32)).cuda()
    h = torch.from_numpy((0.1 + rng.random(n)).astype(np.float32)).cuda()
    members = [GpuTreeLearner(ds, LearnerConfig(num_leaves=15, use_quantized_grad=1, seed=1)) for _ in range(32)]
    torch.cuda.synchronize()

    def run(count):
        t = []
        for _ in range(25):
            a = time.perf_counter()
            outs = train_batch(members[:count], [g.data_ptr()] * count, [h.data_ptr()] * count, on_device=True)
            t.append(time.perf_counter() - a)
        assert all(int(o[3][0]) == 15 for o in outs)
        return float(np.median(t))

    run(32)  # every learner's graph, and its place in the queues
    assert run(16) < 2.9 * run(4)
    for L in members:
        L.close()
