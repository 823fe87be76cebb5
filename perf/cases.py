"""What the learner's performance is measured on: boosting iterations over the range of datasets,
options and execution forms that a user of the framework runs, plus the two row-wise passes beside
training (device bin construction and held-out prediction).

A training pass is one boosting iteration as ``bench.py`` runs it: the objective's gradients on
the device from the current score, one tree (or the K class trees) through ``GpuTreeLearner``, and
the score update with the shrunk leaf values. The gradients of every pass come from the same
mid-training score, as a random forest's do, so that a pass repeated many times keeps growing the
trees that a training run grows; the updated score is an array of its own. The learner's
stochastic-rounding engine advances from pass to pass as it does in training.

Kinds: ``train`` (one dataset, one tree a pass), ``multiclass`` (K class trees a pass),
``group`` (independent jobs, one CUDA graph a pass), ``bin`` (device bin construction of a value
matrix) and ``predict`` (held-out rows through trained trees).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bankai-lightgbm_gb300"))
from lgbm_gb300 import BinnedDataset, GpuTreeLearner, LearnerConfig  # noqa: E402
from lgbm_gb300.learner import LearnerGroup  # noqa: E402
from lgbm_gb300.tree import Tree  # noqa: E402

LR = 0.1
MIN_DATA = 20
ZERO = float(np.float32(1e-35))
FIELDS = ("leaf", "right_leaf", "inner_feature", "threshold", "default_left", "left_count", "right_count",
          "left_output", "right_output", "left_sum_gradient", "left_sum_hessian", "right_sum_gradient",
          "right_sum_hessian", "gain", "left_int_sum", "right_int_sum", "cat_bins")


def listed():
    return [
        # the smallest of the independent jobs that users train by the hundred: launches and latency
        dict(name="job_5k_x20", kind="train", rows=5000, features=20, max_bin=255, leaves=31, objective="binary",
             quant=True, form="graph", nan=0.01),
        # an everyday table in the default full-precision graph form, hessians that vary
        dict(name="float_100k_x28", kind="train", rows=100000, features=28, max_bin=255, leaves=31,
             objective="binary", quant=False, form="graph", nan=0.0),
        # the plain form: one host round trip a split, full precision, an odd feature count. Full-precision
        # cases hold no missing values: where a leaf has none of a column's, both of its missing directions
        # give the same split, and the last bits of sums added in any order pick one (quantized sums are exact)
        dict(name="float_step_1m_x67", kind="train", rows=1000003, features=67, max_bin=255, leaves=63,
             objective="l2", quant=False, form="step", nan=0.0),
        # full precision at scale in one graph
        dict(name="float_4m_x100", kind="train", rows=4000000, features=100, max_bin=255, leaves=255,
             objective="l2", quant=False, form="graph", nan=0.0),
        # the headline workload of the benchmark, with the launch shape autotuned as the benchmark does
        dict(name="l2_10m_x100", kind="train", rows=10000000, features=100, max_bin=255, leaves=255, objective="l2",
             quant=True, form="graph", nan=0.1, autotune=True),
        # the largest: binary with quantized gradients, 200 features
        dict(name="binary_10m_x200", kind="train", rows=10000000, features=200, max_bin=255, leaves=255,
             objective="binary", quant=True, form="graph", nan=0.05),
        # options in earnest: categorical columns, bagged rows and host gradients (a host objective)
        dict(name="cat_bagged_300k_x40", kind="train", rows=300001, features=40, max_bin=255, leaves=63,
             objective="binary", quant=True, form="graph", nan=0.05, categorical=6, bagging=0.7, host_grad=True),
        # quantized training with leaf renewal (the stable partition in the graph form)
        dict(name="renew_500k_x50_bin63", kind="train", rows=500009, features=50, max_bin=63, leaves=63,
             objective="l2", quant=True, form="graph", nan=0.0, renew=True, quant_bins=16),
        # the ten class trees of a softmax iteration
        dict(name="multiclass10_2m_x64", kind="multiclass", rows=2000000, features=64, max_bin=63, leaves=63,
             classes=10),
        # independent jobs of very different sizes, one graph for all of them (few and many bins, 20 to 300
        # features)
        dict(name="group_12_jobs", kind="group", jobs=12, leaves=31),
        # device bin construction of a float table
        dict(name="bin_3m_x100", kind="bin", rows=3000000, features=100, max_bin=255, nan=0.1, wide=False),
        # held-out rows through the trees of a model
        dict(name="predict_2m_x100_10trees", kind="predict", rows=2000000, features=100, max_bin=255, leaves=255,
             trees=10, nan=0.05),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train"] * 6 + ["multiclass", "group", "bin", "predict"])
    if kind == "multiclass":
        return dict(kind=kind, rows=_spread(rng, 20000, 1200000), features=rng.randint(16, 64),
                    max_bin=rng.choice([15, 63, 255]), leaves=rng.choice([15, 31, 63]), classes=rng.randint(3, 10))
    if kind == "group":
        return dict(kind=kind, jobs=rng.randint(4, 12), leaves=rng.choice([15, 31, 63]))
    if kind == "bin":
        return dict(kind=kind, rows=_spread(rng, 2000, 3000000), features=rng.randint(5, 100),
                    max_bin=rng.choice([15, 63, 255]), nan=rng.choice([0.0, 0.1]), wide=rng.random() < 0.3)
    if kind == "predict":
        return dict(kind=kind, rows=_spread(rng, 3000, 2000000), features=rng.randint(20, 100), max_bin=255,
                    leaves=rng.choice([31, 63, 255]), trees=rng.randint(5, 20), nan=0.05)
    quant = rng.random() < 0.65
    form = "graph" if rng.random() < 0.8 else "step"
    rows = _spread(rng, 5000, 4000000)
    c = dict(kind=kind, rows=rows, features=rng.randint(20, 200 if rows < 1500000 else 100),
             max_bin=rng.choice([15, 63, 255, 255]), leaves=rng.choice([15, 31, 63, 127, 255]),
             objective=rng.choice(["l2", "binary"]), quant=quant, form=form, nan=rng.choice([0.0, 0.01, 0.1]) if quant else 0.0)
    if quant:
        c["quant_bins"] = rng.choice([4, 4, 16])
    if rows < 400000 and rng.random() < 0.4:
        c["bagging"] = 0.7
    return c


# ---- inputs ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _values(g, rows, features, nan, integers):
    """Float columns as the benchmark's workloads have them: N(0, 1) and, with ``integers``, 30% of
    whole numbers 0..15, else uniform(-1, 1) for the second half; NaNs at random."""
    X = torch.empty((rows, features), dtype=torch.float32, device="cuda")
    k = max(1, (features * 7) // 10 if integers else features // 2)
    X[:, :k].normal_(generator=g)
    if k < features:
        if integers:
            X[:, k:] = torch.randint(0, 16, (rows, features - k), generator=g, device="cuda").float()
        else:
            X[:, k:].uniform_(-1.0, 1.0, generator=g)
    return X


def _add_nan(g, X, nan):
    if nan > 0:
        for c0 in range(0, X.shape[1], 25):
            blk = X[:, c0:c0 + 25]
            blk[torch.rand(blk.shape, generator=g, device="cuda") < nan] = float("nan")
    return X


def _target(g, X, objective):
    """The label and a score from the middle of training: twenty step functions of features (l2), a
    sparse linear logistic model (binary); the score explains about half of the signal."""
    n, F = X.shape
    if objective == "l2":
        z = torch.zeros(n, device="cuda")
        for f in torch.randint(0, F, (20,), generator=g, device="cuda").tolist():
            thr, a, b = torch.randn(3, generator=g, device="cuda").tolist()
            z += torch.where(X[:, f] > 0.5 * thr, a, b)
        y = z + 0.1 * torch.randn(n, generator=g, device="cuda")
        noise = 0.3
    else:
        w = torch.randn(F, generator=g, device="cuda") * (torch.rand(F, generator=g, device="cuda") < 0.2)
        w[0] = 1.0
        z = X @ w
        y = (torch.rand(n, generator=g, device="cuda") < torch.sigmoid(z)).float()
        noise = 0.3
    score = 0.5 * z.double() + noise * torch.randn(n, generator=g, device="cuda").double()
    return y.contiguous(), score.contiguous()


def _config(case, const_hess):
    return LearnerConfig(num_leaves=case["leaves"], min_data_in_leaf=MIN_DATA,
                         use_quantized_grad=int(case.get("quant", True)),
                         num_grad_quant_bins=case.get("quant_bins", 4), stochastic_rounding=1,
                         quant_train_renew_leaf=int(case.get("renew", False)), seed=0, num_threads=16, fused_madd=1,
                         is_constant_hessian=int(const_hess))


def _dataset(X, case):
    return BinnedDataset.from_dense_device(X, max_bin=case["max_bin"], min_data_in_leaf=MIN_DATA,
                                           bin_construct_sample_cnt=20000)


class _Training:
    """One learner with its score, label and results: what a training program holds."""

    def __init__(self, case, ds, y, score, rows=None):
        self.case, self.ds, self.rows = case, ds, rows
        self.kind = {"l2": 0, "binary": 1, "softmax": 2}[case["objective"]]
        self.label, self.start = y, score
        self.K = case.get("classes", 1)
        self.learner = GpuTreeLearner(ds, _config(case, self.kind == 0), num_jobs=self.K,
                                      loop_mode=0 if case.get("form") == "step" else 1)
        self.score = score.clone()
        self.g, self.h = self.learner.gradient_buffers()
        self.host = None
        torch.cuda.synchronize()
        if case.get("host_grad"):  # a host objective: the gradients of the start score, in host memory
            p = torch.sigmoid(score)
            self.host = ((p - y.double()).float().cpu().numpy(), (p * (1.0 - p)).float().cpu().numpy())
        if case.get("autotune"):
            self.gradients()
            self.learner.autotune(self.g, self.h, on_device=True, trials=2)

    def gradients(self):
        self.learner.objective_gradients(self.kind, self.start.data_ptr(), self.label.data_ptr())

    def step(self):
        if self.host is not None:
            splits, lv, roots, nls = self.learner.train_raw(self.host[0], self.host[1], rows=self.rows)
        else:
            self.gradients()
            splits, lv, roots, nls = self.learner.train_raw(self.g, self.h, rows=self.rows, on_device=True)
        vals = lv * LR
        vals[np.abs(vals) <= ZERO] = 0.0
        self.learner.add_prediction_to_score(vals, self.score.data_ptr(), on_device=True)
        out = {f: splits[f] for f in FIELDS}
        out.update(leaf_values=lv, root_outputs=roots, num_leaves=nls, score=self.score)
        return out


def _categorical_dataset(g, X, case):
    """The last columns become categories (3 to 200 of them, some rows missing); binned on the host,
    as categorical columns are."""
    n, F = X.shape
    cols = list(range(F - case["categorical"], F))
    for j, c in enumerate(cols):
        k = (3, 8, 20, 40, 90, 200)[j % 6]
        X[:, c] = torch.floor(torch.rand(n, generator=g, device="cuda").square() * k)
    return BinnedDataset.from_dense(X.cpu().numpy(), max_bin=case["max_bin"], min_data_in_leaf=MIN_DATA,
                                    bin_construct_sample_cnt=20000, categorical=cols)


def _prepare_train(case, seed):
    g = _gen(seed)
    X = _values(g, case["rows"], case["features"], case["nan"], case["objective"] == "l2")
    y, score = _target(g, X, case["objective"])
    X = _add_nan(g, X, case["nan"])
    ds = _categorical_dataset(g, X, case) if case.get("categorical") else _dataset(X, case)
    rows = None
    if case.get("bagging"):
        keep = torch.rand(case["rows"], generator=g, device="cuda") < case["bagging"]
        rows = torch.nonzero(keep).flatten().int().cpu().numpy()
    return _Training(case, ds, y, score, rows)


def _prepare_multiclass(case, seed):
    g = _gen(seed)
    n, F, K = case["rows"], case["features"], case["classes"]
    means = torch.randn((K, F), generator=g, device="cuda") * (2.0 / math.sqrt(F)) * 4.0
    y = torch.randint(0, K, (n,), generator=g, device="cuda")
    X = torch.randn((n, F), generator=g, device="cuda") + means[y]
    score = 0.5 * torch.randn((K, n), generator=g, device="cuda").double()
    score[y, torch.arange(n, device="cuda")] += 0.7
    c = dict(case, objective="softmax")
    return _Training(c, _dataset(X, c), y.float(), score.contiguous())


class _Group:
    def __init__(self, case, seed):
        g = _gen(seed)
        rng = np.random.RandomState(7 + case["jobs"])  # the jobs' shapes; their values come from the seed
        self.members = []
        for _ in range(case["jobs"]):
            n = int(round(math.exp(rng.uniform(math.log(5000), math.log(500000)))))
            c = dict(case, features=int(rng.randint(20, 301)), max_bin=int(rng.choice([15, 63, 255])),
                     objective="binary")
            X = torch.randn((n, c["features"]), generator=g, device="cuda")
            y, score = _target(g, X, "binary")
            self.members.append(_Training(c, _dataset(_add_nan(g, X, 0.01), c), y, score))
        self.group = LearnerGroup([m.learner for m in self.members])
        self.gp, self.hp = [m.g for m in self.members], [m.h for m in self.members]
        for m in self.members:
            m.gradients()
        self.group.autotune(self.gp, self.hp, trials=2)

    def step(self):
        for m in self.members:
            m.gradients()
        outs = self.group.train(self.gp, self.hp, shrinkage=LR, scores=[m.score.data_ptr() for m in self.members])
        return [{"splits": s.view(np.uint8), "leaf_values": lv, "num_leaves": nls, "score": m.score}
                for (s, lv, _, nls), m in zip(outs, self.members)]


class _Binning:
    def __init__(self, case, seed):
        g = _gen(seed)
        X = _add_nan(g, _values(g, case["rows"], case["features"], case["nan"], True), case["nan"])
        self.X = X.double() if case["wide"] else X
        self.ds = _dataset(self.X[:min(len(X), 50000)], case)

    def step(self):
        return self.ds.bin_like_device(self.X)


class _Prediction:
    """Held-out rows through trees grown on a training sample of the same distribution."""

    def __init__(self, case, seed):
        g = _gen(seed)
        fit = dict(case, objective="l2", quant=True, rows=20000)
        X = _values(g, 20000 + case["rows"], case["features"], case["nan"], True)
        y, score = _target(g, X, "l2")
        X = _add_nan(g, X, case["nan"])
        t = _Training(fit, _dataset(X[:20000].contiguous(), fit), y[:20000].contiguous(), score[:20000].contiguous())
        self.learner, self.trees = t.learner, []
        for _ in range(case["trees"]):
            t.learner.objective_gradients(0, t.score.data_ptr(), t.label.data_ptr())
            out = t.learner.train_raw(t.g, t.h, on_device=True)
            tree = t.learner.trees(*out)[0]
            tree.apply_shrinkage(LR)
            t.learner.add_prediction_to_score(out[1] * LR, t.score.data_ptr(), on_device=True)
            self.trees.append(tree)
        self.bins = t.ds.bin_like_device(X[20000:].contiguous())
        self.features = t.ds.features
        self.score = score[20000:].contiguous()

    def step(self):
        for tree in self.trees:
            self.learner.predict_add(tree, self.bins.data_ptr(), self.bins.shape[1], self.score.data_ptr())
        return self.score


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind == "multiclass":
        return _prepare_multiclass(case, seed)
    return {"group": _Group, "bin": _Binning, "predict": _Prediction}[kind](case, seed)


def run(state):
    return state.step()


def work(case):
    """Each stored bin, label and score read once and the new score and records written once; an
    addition to the gradient and the hessian sum for every stored bin (of the root histogram)."""
    kind = case["kind"]
    if kind == "bin":
        size = 8 if case["wide"] else 4
        return {"bytes": case["rows"] * case["features"] * (size + 1.0), "flops": 0.0}
    if kind == "predict":
        depth = math.log2(case["leaves"]) + 2.0
        return {"bytes": case["rows"] * (min(case["features"], depth * case["trees"]) + 16.0),
                "flops": case["rows"] * float(case["trees"])}
    if kind == "group":
        rng = np.random.RandomState(7 + case["jobs"])
        total = [0.0, 0.0]
        for _ in range(case["jobs"]):
            n = int(round(math.exp(rng.uniform(math.log(5000), math.log(500000)))))
            F, b = int(rng.randint(20, 301)), int(rng.choice([15, 63, 255]))
            total[0] += n * (F * (0.5 if b == 15 else 1.0) + 28.0)
            total[1] += 2.0 * n * F
        return {"bytes": total[0], "flops": total[1]}
    n, F, K = case["rows"], case["features"], case.get("classes", 1)
    n *= case.get("bagging", 1.0)
    width = 0.5 if case["max_bin"] <= 15 else 1.0
    return {"bytes": n * (F * width + 4.0 + 24.0 * K) + K * case["leaves"] * 168.0, "flops": 2.0 * n * F * K}


# ---- the same in 64 bits, in plain torch ----

def _bins_of(ds):
    """The bin-mapper bin of every (feature, row) from the stored bins (the most frequent bin is
    stored as 0, the others shifted past it)."""
    b = ds.bins.to(torch.int64)
    for j, fi in enumerate(ds.features):
        mfb, off = fi.most_freq_bin, 1 if fi.most_freq_bin == 0 else 0
        b[j] = torch.where(b[j] == 0, mfb, b[j] - 1 + off)
    return b


def _exact_bin(case, seed):
    return None  # bytes: they have to be equal


def _exact_predict(s):
    bins, score = _bins_of(type("D", (), {"bins": s.bins, "features": s.features})), s.score.clone()
    nb = torch.tensor([fi.num_bin for fi in s.features], device="cuda")
    miss = torch.tensor([fi.missing_type for fi in s.features], device="cuda")
    rows = torch.arange(bins.shape[1], device="cuda")
    for t in s.trees:
        ni = t.num_leaves - 1
        arr = {k: torch.tensor(np.asarray(getattr(t, k)[:ni]).astype(np.int64), device="cuda")
               for k in ("left_child", "right_child", "split_feature_inner", "threshold_in_bin", "decision_type")}
        node = torch.zeros(bins.shape[1], dtype=torch.int64, device="cuda")
        while ni and bool((node >= 0).any()):
            at = node.clamp(min=0)
            f = arr["split_feature_inner"][at]
            b = bins[f, rows]
            missing = (miss[f] == 2) & (b == nb[f] - 1)
            left = torch.where(missing, (arr["decision_type"][at] & 2) != 0, b <= arr["threshold_in_bin"][at])
            node = torch.where(node < 0, node, torch.where(left, arr["left_child"][at], arr["right_child"][at]))
        score += torch.tensor(np.asarray(t.leaf_value), device="cuda")[(~node).clamp(min=0)]
    return score


def _exact_float(case, s):
    """Leaf-wise growth on f64 histograms: the smaller child's by summation, its sibling's by
    subtraction; both missing directions of every threshold; the best leaf first."""
    bins, feats = _bins_of(s.ds), s.ds.features
    F, n, L = len(feats), bins.shape[1], case["leaves"]
    B = max(fi.num_bin for fi in feats)
    nb = torch.tensor([fi.num_bin for fi in feats], device="cuda")
    na = (torch.tensor([fi.missing_type for fi in feats], device="cuda") == 2) & (nb > 2)
    y = s.label.double()
    if s.kind == 0:
        g, h = (s.start - y).float().double(), torch.ones(n, dtype=torch.float64, device="cuda")
    else:
        p = torch.sigmoid(s.start)
        g, h = (p - y).float().double(), (p * (1.0 - p)).float().double()
    base = torch.arange(F, device="cuda")[:, None] * B
    col = torch.arange(B, device="cuda")[None, :]

    def hist(rows):
        out = torch.zeros(2, F * B, dtype=torch.float64, device="cuda")
        for part in rows.split(1 << 20):
            idx = (bins[:, part] + base).flatten()
            for k, w in enumerate((g, h)):
                out[k] += torch.bincount(idx, weights=w[part].expand(F, -1).flatten(), minlength=F * B)
        return out.view(2, F, B)

    def search(H, G0, H0, count, used):
        cnt = torch.floor(H[1] * (count / H0) + 0.5)
        shift = G0 * G0 / H0
        is_na = na[:, None] & (col == nb[:, None] - 1)
        v = torch.stack([H[0], H[1], cnt])
        low = v.masked_fill(is_na, 0.0)
        right = low.flip(2).cumsum(2).flip(2) - low  # bins past the threshold, without the missing one
        left = v.cumsum(2)                           # bins up to it
        best = None
        for d, side in ((0, right), (1, left)):
            og, oh, oc = G0 - side[0], H0 - side[1], count - side[2]
            last = nb[:, None] - (2 if d == 1 else torch.where(na[:, None], 3, 2))
            ok = (col <= last) & used[:, None] & (side[2] >= MIN_DATA) & (oc >= MIN_DATA) & (side[1] >= 1e-3) & (oh >= 1e-3)
            if d == 1:
                ok &= na[:, None]
            gain = side[0] ** 2 / side[1] + og ** 2 / oh
            gain = torch.where(ok & (gain > shift), gain, torch.full_like(gain, -math.inf))
            top = gain.max(1).values
            near = gain >= (top - 1e-12 * top.abs())[:, None]
            t = torch.where(near, col, -1).max(1).values if d == 0 else torch.where(near, col, B).min(1).values
            if best is None:
                best = (top, t, torch.zeros_like(t))
            else:
                take = top > best[0]
                best = tuple(torch.where(take, a, b) for a, b in ((top, best[0]), (t, best[1]), (torch.ones_like(t), best[2])))
        top = best[0] - shift
        can = torch.isfinite(best[0])
        f = int(torch.where(can, top, torch.full_like(top, -math.inf)).argmax())
        if not bool(can[f]):
            return None, can
        t, d = int(best[1][f]), int(best[2][f])
        sd = (right if d == 0 else left)[:, f, t]
        lg, lh = (G0 - sd[0], H0 - sd[1]) if d == 0 else (sd[0], sd[1])
        return (float(top[f]), f, t, d, float(lg), float(lh)), can

    rows = torch.arange(n, device="cuda") if s.rows is None else torch.from_numpy(s.rows).long().cuda()
    G0, H0 = float(g[rows].sum()), float(h[rows].sum())
    leaves = [dict(rows=rows, hist=hist(rows), G=G0, H=H0, used=torch.ones(F, dtype=torch.bool, device="cuda"))]
    leaves[0]["best"], leaves[0]["can"] = search(leaves[0]["hist"], G0, H0, len(rows), leaves[0]["used"])
    rec = {k: np.zeros((1, L - 1)) for k in ("left_output", "right_output", "left_sum_gradient", "left_sum_hessian",
                                             "right_sum_gradient", "right_sum_hessian", "gain")}
    for i in range(L - 1):
        gains = [-math.inf if x["best"] is None else x["best"][0] for x in leaves]
        at = int(np.argmax(gains))
        if gains[at] <= 0.0:
            break
        P = leaves[at]
        gain, f, t, d, lg, lh = P["best"]
        b = bins[f, P["rows"]]
        go = b <= t
        if bool(na[f]):
            go = torch.where(b == int(nb[f]) - 1, torch.tensor(d == 0, device="cuda"), go)
        sides = [dict(rows=P["rows"][go], G=lg, H=lh), dict(rows=P["rows"][~go], G=P["G"] - lg, H=P["H"] - lh)]
        for k, c in zip(("left", "right"), sides):
            rec[k + "_output"][0, i] = -c["G"] / c["H"]
            rec[k + "_sum_gradient"][0, i], rec[k + "_sum_hessian"][0, i] = c["G"], c["H"]
        rec["gain"][0, i] = gain
        small = 0 if len(sides[0]["rows"]) < len(sides[1]["rows"]) else 1
        if max(len(c["rows"]) for c in sides) >= 2 * MIN_DATA:
            sides[small]["hist"] = hist(sides[small]["rows"])
            sides[1 - small]["hist"] = P["hist"] - sides[small]["hist"]
            for c in sides:
                c["used"] = P["can"]
                c["best"], c["can"] = search(c["hist"], c["G"], c["H"], len(c["rows"]), c["used"])
        else:
            sides[0]["best"] = sides[1]["best"] = None
        leaves[at] = sides[0]
        leaves.append(sides[1])
    lv = np.zeros((1, L))
    score = s.start.clone()
    for k, x in enumerate(leaves):
        lv[0, k] = -x["G"] / x["H"]
        score[x["rows"]] += LR * lv[0, k]
    out = {k: rec.get(k) for k in FIELDS}
    out.update(leaf_values=lv, root_outputs=np.array([-G0 / H0]), num_leaves=None, score=score)
    return out


def exact(case, seed):
    """Full-precision trees and predictions; quantized trees follow the reference's random rounding
    bit for bit, which has no value in 64 bits, and stored bins are bytes."""
    if case["kind"] == "predict":
        return _exact_predict(prepare(case, seed))
    if case["kind"] == "train" and not case["quant"] and not case.get("categorical"):
        return _exact_float(case, prepare(case, seed))
    return None
