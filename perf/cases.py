"""Workloads that stand for what programs ask of this framework on one GPU.

Three kinds of work, each through the public entry points:

* ``train``   - ``fb.train`` on a constructed ``Dataset`` (the bins are in place, as when one data set serves many runs):
  booster set-up, every boosting round, the metrics of the validation set where there is one. The answer is the raw
  training scores, to which every tree has contributed, the features' gains and the recorded metrics.
* ``ingest``  - a feature matrix in GPU memory becomes a ``Dataset`` (bin boundaries, binning) and a few rounds are
  trained on it: the refit of a model on fresh data.
* ``predict`` - ``Booster.predict`` of a CUDA tensor with a loaded model: scores, probabilities or leaf indices.

The inputs have the shapes of the project's benchmark configurations (``falcata_b200.utils.synthetic``) or are plain
normal data; the models of the ``predict`` cases are written as model text, best-first trees whose thresholds lie on
each feature's bin boundaries, so that they do not depend on the training code.
"""
from __future__ import annotations

import heapq
import math
from typing import Any, Dict, List

import numpy as np
import torch

import falcata_b200 as fb
from falcata_b200.utils import synthetic

_TRAIN = {"kind": "train", "task": "binary", "features": 28, "max_bin": 255, "leaves": 31, "rounds": 100, "quant": "none", "levels": 0, "grow": "level",
          "feature_fraction": 1.0, "bagging": 1.0, "weighted": False, "classes": 1, "valid_rows": 0}
_PREDICT = {"kind": "predict", "features": 28, "trees": 100, "leaves": 255, "classes": 1, "dtype": "float32", "output": "raw", "missing": False}


def listed() -> List[Dict[str, Any]]:
    return [
        # A small table with every parameter at its default: 100 rounds of 31 leaves, launches and host steps count.
        dict(_TRAIN, name="train_small_defaults", rows=10_000),
        # The headline benchmark configuration: 11M x 28, 255 leaves, 63 bins, 4 gradient levels.
        dict(_TRAIN, name="train_binary_11m", rows=11_000_000, max_bin=63, leaves=255, rounds=30, quant="stochastic", levels=4),
        # Exact best-first trees on one eighth of it (the shard of one GPU of eight), a row count that divides by nothing.
        dict(_TRAIN, name="train_binary_leafwise", rows=1_375_003, max_bin=63, leaves=255, rounds=30, quant="stochastic", levels=4, grow="leaf"),
        # The usual development loop: 255 bins, full precision, a bag per round, AUC and log loss of a validation set every round.
        dict(_TRAIN, name="train_with_validation", rows=1_000_000, leaves=63, rounds=40, bagging=0.8, valid_rows=200_000),
        # A mid-sized weighted regression table (515k x 90) on fixed-point gradients.
        dict(_TRAIN, name="train_regression_weighted", task="regression", rows=515_345, features=90, leaves=255, rounds=40, quant="fixedpoint", levels=64, weighted=True),
        # Wide, low-cardinality integer data; a tenth of the columns per tree.
        dict(_TRAIN, name="train_wide_sampled", task="wide", rows=1_000_000, features=2000, max_bin=16, leaves=255, rounds=20, quant="fixedpoint", levels=64, feature_fraction=0.1),
        # Ten classes, full precision: ten trees per round.
        dict(_TRAIN, name="train_multiclass", task="multiclass", rows=1_000_000, features=100, leaves=127, rounds=4, classes=10),
        # Learning to rank on queries of 1 to 200 documents, full precision.
        dict(_TRAIN, name="train_ranking", task="ranking", rows=2_000_000, features=136, leaves=255, rounds=4),
        # Fresh data in GPU memory to a trained model.
        dict(_TRAIN, name="ingest_fresh_data", kind="ingest", rows=5_000_000, max_bin=63, leaves=255, rounds=5, quant="stochastic", levels=4),
        # One request of an online service: a handful of rows.
        dict(_PREDICT, name="predict_request", rows=16, trees=200, leaves=31, output="probability"),
        # Class probabilities of a mid-sized batch of double-precision rows, some values missing.
        dict(_PREDICT, name="predict_multiclass_f64", rows=200_003, features=100, trees=500, leaves=127, classes=10, dtype="float64", output="probability", missing=True),
        # Batch scoring with a large forest: the ranking shape.
        dict(_PREDICT, name="predict_batch", rows=4_000_000, features=136, trees=500),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> Dict[str, Any]:
    """One more case of the ranges above; the sizes are spread over their logarithms and shrunk until the work is in range."""
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "train", "predict", "predict", "ingest"])
        if kind == "predict":
            classes = rng.choice([1, 1, 1, 3, 10])
            case = dict(_PREDICT, rows=_log_int(rng, 1, 6_000_000), features=_log_int(rng, 4, 200), trees=classes * _log_int(rng, 10, 600 // classes),
                        leaves=rng.choice([7, 31, 63, 127, 255, 400]), classes=classes, dtype=rng.choice(["float32", "float32", "float64", "float16"]),
                        output=rng.choice(["raw", "probability", "raw", "leaf"]), missing=rng.random() < 0.3)
        else:
            task = rng.choice(["binary", "binary", "binary", "regression", "regression", "multiclass", "ranking", "wide"]) if kind == "train" else "binary"
            case = dict(_TRAIN, kind=kind, task=task, rows=_log_int(rng, 2_000, 6_000_000), leaves=rng.choice([15, 31, 63, 127, 255]), rounds=_log_int(rng, 3, 40))
            case["quant"] = rng.choice(["none", "stochastic", "fixedpoint"])
            case["levels"] = 0 if case["quant"] == "none" else rng.choice([4, 16, 64])
            case["max_bin"] = rng.choice([15, 63, 127, 255])
            case["grow"] = rng.choice(["level", "level", "leaf"])
            if task == "regression":
                case["features"] = _log_int(rng, 4, 200)
                case["weighted"] = rng.random() < 0.5
            elif task == "multiclass":
                case.update(features=_log_int(rng, 8, 120), classes=rng.choice([3, 5, 10]), rounds=_log_int(rng, 2, 10))
            elif task == "ranking":
                case.update(features=136, rows=max(20_000, case["rows"] // 3), rounds=rng.randint(2, 4))
            elif task == "wide":
                case.update(features=_log_int(rng, 300, 2000), max_bin=16, feature_fraction=rng.choice([0.1, 0.3, 1.0]))
            if kind == "train" and task in ("binary", "regression"):
                case["bagging"] = rng.choice([1.0, 1.0, 0.8, 0.5])
                case["valid_rows"] = rng.choice([0, 0, max(1000, case["rows"] // 5)])
        largest = case["rows"] * (case["features"] if case.get("output") != "leaf" else case["trees"])   # values of the matrix, or of the answer
        if largest <= 2_000_000_000 and _cost(case) <= most:
            return case


# ---------------------------------------------------------------------------------------------------- inputs ----
def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _data(case: Dict[str, Any], rows: int, seed: int):
    """(X on the GPU, y, weight, group) of the task."""
    task, f = case["task"], case["features"]
    if task == "wide":
        x, y = synthetic.regression_wide(rows, f, seed=seed)
        return x, y.cpu().numpy(), None, None
    if task == "multiclass":
        x, y = synthetic.multiclass(rows, f, case["classes"], seed=seed)
        return x, y.cpu().numpy(), None, None
    if task == "ranking":
        x, y, _ = synthetic.ranking(-(-rows // 100), f=f, seed=seed)
        group = []
        r = np.random.RandomState(seed % (1 << 31))
        left = rows
        while left > 0:
            group.append(min(left, int(r.randint(1, 201))))
            left -= group[-1]
        return x[:rows], y[:rows].cpu().numpy(), None, np.asarray(group, dtype=np.int32)
    if task == "regression":
        g = _generator(seed)
        x = torch.randn(rows, f, generator=g, device="cuda")
        w = torch.randn(f, generator=g, device="cuda")
        y = x @ w + 2.0 * torch.sin(3.0 * x[:, 0]) * x[:, 1] + torch.randn(rows, generator=g, device="cuda")
        weight = (0.5 + torch.rand(rows, generator=g, device="cuda")).cpu().numpy() if case["weighted"] else None
        return x, y.cpu().numpy(), weight, None
    x, y = synthetic.binary_higgs_like(rows, seed=seed)
    return x, y.cpu().numpy(), None, None


def _params(case: Dict[str, Any]) -> Dict[str, Any]:
    objective = {"wide": "regression", "ranking": "lambdarank"}.get(case["task"], case["task"])
    p = {"objective": objective, "num_leaves": case["leaves"], "max_bin": case["max_bin"], "grow_policy": case["grow"], "device_type": "cuda", "verbosity": -1}
    if case["quant"] != "none":
        p.update(quant_mode=case["quant"], quant_bins=case["levels"])
    if case["classes"] > 1:
        p["num_class"] = case["classes"]
    if case["feature_fraction"] < 1.0:
        p["feature_fraction"] = case["feature_fraction"]
    if case["bagging"] < 1.0:
        p.update(bagging_fraction=case["bagging"], bagging_freq=1)
    if case["valid_rows"]:
        p["metric"] = "auc,binary_logloss" if objective == "binary" else "l2"
    return p


def _tree_text(index: int, rng: np.random.RandomState, leaves: int, features: int, boundaries: np.ndarray, missing: bool) -> str:
    """A best-first tree: the leaf that holds the most rows (times a random factor) splits next, at a random bin boundary."""
    n = leaves - 1
    feature = rng.randint(0, features, n)
    cut = 0.15 + 0.7 * rng.rand(n)
    threshold = boundaries[(cut * len(boundaries)).astype(np.int64)]
    pick = rng.rand(2 * leaves)
    left, right = [0] * n, [0] * n
    heap = [(-1.0, 0, 1.0, -1, False)]   # (-priority, leaf, mass, parent, is the parent's right child)
    for s in range(n):
        _, leaf, mass, parent, is_right = heapq.heappop(heap)
        if parent >= 0:
            (right if is_right else left)[parent] = s
        left[s], right[s] = ~leaf, ~(s + 1)
        a = mass * float(cut[s])
        b = mass - a
        heapq.heappush(heap, (-a * float(pick[2 * s]), leaf, a, s, False))
        heapq.heappush(heap, (-b * float(pick[2 * s + 1]), s + 1, b, s, True))
    kind = 10 if missing else 2   # 10: missing values are NaN, to the left; 2: the feature has none
    value = 0.05 * rng.randn(leaves)
    words = lambda v: " ".join(map(repr, v.tolist() if isinstance(v, np.ndarray) else v))  # noqa: E731
    return (f"Tree={index}\nnum_leaves={leaves}\nnum_cat=0\nsplit_feature={words(feature)}\nthreshold={words(threshold)}\n"
            f"decision_type={' '.join([str(kind)] * n)}\nleft_child={words(left)}\nright_child={words(right)}\nleaf_value={words(value)}\nis_linear=0\nshrinkage=0.1\n\n\n")


def _model(case: Dict[str, Any], seed: int) -> str:
    rng = np.random.RandomState(seed % (1 << 31))
    k, f = case["classes"], case["features"]
    boundaries = np.sort(rng.randn(254))
    objective = f"multiclass num_class:{k}" if k > 1 else "binary sigmoid:1"
    names = " ".join(f"Column_{j}" for j in range(f))
    head = (f"tree\nversion=v4\nnum_class={k}\nnum_tree_per_iteration={k}\nlabel_index=0\nmax_feature_idx={f - 1}\nobjective={objective}\n"
            f"feature_names={names}\nfeature_infos={' '.join(['[-5:5]'] * f)}\n\n")
    return head + "".join(_tree_text(i, rng, case["leaves"], f, boundaries, case["missing"]) for i in range(case["trees"])) + "end of trees\n"


def prepare(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    state: Dict[str, Any] = {"case": case, "kind": case["kind"], "booster": None}
    if case["kind"] == "predict":
        g = _generator(seed)
        x = torch.randn(case["rows"], case["features"], generator=g, device="cuda")
        if case["missing"]:
            x[torch.rand(x.shape, generator=g, device="cuda") < 0.02] = float("nan")
        state["x"] = x.to(getattr(torch, case["dtype"]))
        state["booster"] = fb.Booster(model_str=_model(case, seed))
        return state
    state["params"] = _params(case)
    x, y, weight, group = _data(case, case["rows"] + case["valid_rows"], seed)
    n = case["rows"]
    if case["kind"] == "ingest":
        state.update(x=x, y=y)
        return state
    dataset_params = {"max_bin": case["max_bin"], "device_type": "cuda", "verbosity": -1}
    state["train"] = fb.Dataset(x[:n], y[:n], weight=None if weight is None else weight[:n], group=group, params=dataset_params).construct()
    state["valid"] = None
    if case["valid_rows"]:
        state["valid"] = state["train"].create_valid(x[n:], y[n:], weight=None if weight is None else weight[n:]).construct()
    return state


# ------------------------------------------------------------------------------------------------------ work ----
def run(state: Dict[str, Any]) -> Dict[str, Any]:
    case = state["case"]
    if state["kind"] == "predict":
        if case["output"] == "leaf":
            return {"leaf": state["booster"].predict(state["x"], pred_leaf=True)}
        return {"score": state["booster"].predict(state["x"], raw_score=case["output"] == "raw")}
    state["booster"] = None   # the previous model makes room
    if state["kind"] == "ingest":
        train = fb.Dataset(state["x"], state["y"], params={"max_bin": case["max_bin"], "device_type": "cuda", "verbosity": -1})
        valid = None
    else:
        train, valid = state["train"], state["valid"]
    history: Dict[str, Any] = {}
    callbacks = [fb.record_evaluation(history)] if valid is not None else None
    booster = fb.train(state["params"], train, case["rounds"], valid_sets=None if valid is None else [valid], callbacks=callbacks, keep_training_booster=True)
    state["booster"] = booster
    # the tensor is a view of the booster's memory: the answer is a copy that outlives it
    return {"score": booster.train_score_tensor().clone(), "gain": booster.feature_importance("gain"),
            "metrics": {name: np.asarray(values) for name, values in history.get("valid_0", {}).items()}}


def work(case: Dict[str, Any]) -> Dict[str, float]:
    rows, f, k = case["rows"], case["features"], case["classes"]
    if case["kind"] == "predict":
        size = {"float32": 4, "float64": 8, "float16": 2}[case["dtype"]]
        out = case["trees"] if case["output"] == "leaf" else k
        depth = math.log2(case["leaves"])
        return {"bytes": rows * (f * size + out * 4) + case["trees"] * case["leaves"] * 12, "flops": rows * case["trees"] * depth}
    # A tree of depth d reads every row's sampled bins once for the root and half of them for each further level (the
    # sibling follows by subtraction), the split column of every row at each level, and per round the labels and scores.
    trees, depth = case["rounds"] * k, math.ceil(math.log2(case["leaves"]))
    sampled, bagged = f * case["feature_fraction"], rows * case["bagging"]
    bin_bytes = 0.5 if case["max_bin"] <= 16 else 1.0
    passes = 1.0 + 0.5 * (depth - 1)
    per_tree = bagged * (passes * sampled * bin_bytes + depth) + rows * 8
    total = trees * per_tree + case["rounds"] * rows * 4
    total += trees * case["valid_rows"] * (depth + 8)
    if case["kind"] == "ingest":
        total += rows * f * 5
    return {"bytes": total, "flops": trees * bagged * passes * sampled * 2}


def _cost(case: Dict[str, Any]) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case: Dict[str, Any]) -> Any:
    if case["kind"] == "predict":
        # against sums in double: 7e-8 and 3e-7
        return "exact" if case["output"] == "leaf" else {"rel": 1e-6, "max": 1e-5}
    if case["task"] == "ranking":
        # sums in another order turn near-ties between splits around, and a row that changes leaves changes its query's
        # order and with it other rows' gradients: up to 7e-4 after 4 rounds, 5e-2 to 1e-1 after 8
        return {"rel": 3e-3, "max": 0.9}
    if case["quant"] != "none":
        # integer histograms: only the fp32 gradients, scores and outputs are rounded (2e-6 and 1e-4 with the gradients in double)
        return {"rel": 1e-5, "max": 1e-3}
    # fp32 histograms: sums in another order turn an occasional near-tie around (6e-5 with one turned split in 40 trees of
    # 63 leaves, 2e-3 on the small table)
    return {"rel": 1e-2, "max": 0.9}
