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
