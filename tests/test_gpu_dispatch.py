"""Kernel variants that a rule on sizes selects, at the edges of the rule: the lane construct's block flush, the one-launch row
partition, the split search, the per-row kernels of a round's set-up and the tile shapes of prediction."""
import ctypes

import numpy as np
import pytest
import torch

import falcata_b200 as fb
from util import make_binary, model_body

pytestmark = pytest.mark.gpu


def _rows(n, groups, nb, gen):
    stride = ((groups + 4 + 15) // 16) * 16
    rows = torch.full((n, stride), 255, dtype=torch.uint8, device="cuda")   # bytes past the last group are no bins
    rows[:, :groups] = torch.randint(0, nb, (n, groups), generator=gen, device="cuda", dtype=torch.int32).to(torch.uint8)
    rows[: n // 2, 0] = nb - 1   # runs of one bin: equal cells inside a step are forwarded in registers
    return rows


def _reference(rows, groups, nb, value, idx=None):
    sel = rows if idx is None else rows[idx.long()]
    v = (value if idx is None else value[idx.long()]).double()
    out = torch.zeros(groups * nb, dtype=torch.float64, device="cuda")
    for k in range(groups):
        out.index_add_(0, sel[:, k].long() + k * nb, v)
    return out


@pytest.mark.parametrize("nb", [16, 17, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("n,groups,rpb", [(1, 1, 512), (31, 16, 512), (33, 17, 64), (2049, 28, 512), (20011, 32, 4096), (9001, 33, 1024), (5003, 49, 96)])
def test_lane_construct(n, groups, nb, rpb):
    from falcata_b200 import ops
    gen = torch.Generator(device="cuda"); gen.manual_seed(n * 1000 + groups + nb)
    rows = _rows(n, groups, nb, gen)
    idx = torch.randperm(n, generator=gen, device="cuda")[: max(1, (2 * n) // 3)].int()
    for qbins in (4, 64):
        gi = torch.randint(-(qbins // 2), qbins // 2 + 1, (n,), generator=gen, device="cuda", dtype=torch.int32)
        hi = torch.randint(0, qbins + 1, (n,), generator=gen, device="cuda", dtype=torch.int32)
        packed = (gi << 16) | (hi & 0xFFFF)
        for mode in (1, 2):
            for sub in (None, idx):
                out = ops.histogram(rows, packed, [nb] * groups, idx=sub, quant=True, quant_bins=qbins, rows_per_block=rpb, lane_mode=mode)
                assert torch.equal(out[:, 0], _reference(rows, groups, nb, gi, sub).long()) and torch.equal(out[:, 1], _reference(rows, groups, nb, hi, sub).long())
    gh = torch.randn(n, 2, device="cuda", generator=gen); gh[:, 1].abs_()
    for mode in (1, 2):   # load-add-store, reduction adds
        for sub in (None, idx):
            out = ops.histogram(rows, gh, [nb] * groups, idx=sub, quant=False, rows_per_block=rpb, lane_mode=mode)
            count = _reference(rows, groups, nb, torch.ones(n, device="cuda"), sub)
            for k in range(2):
                # fp32 sums of a cell's rows: at most `count` roundings of a running sum of at most sum |v|
                bound = count * 2.0 ** -24 * _reference(rows, groups, nb, gh[:, k].abs(), sub) + 1e-12
                assert bool(((out[:, k] - _reference(rows, groups, nb, gh[:, k], sub)).abs() <= bound).all())


@pytest.mark.parametrize("warps,quant,nb", [(6, False, 256), (9, False, 200), (12, True, 256), (6, True, 256)])
def test_lane_construct_with_few_warps(monkeypatch, warps, quant, nb):
    """Few warps stage little: the block's flush, which takes the stages' place, then decides how many tiles fit."""
    from falcata_b200 import ops
    monkeypatch.setenv("FALCATA_LANE_WARPS", str(warps))
    gen = torch.Generator(device="cuda"); gen.manual_seed(warps)
    n, groups = 5003, 33
    rows = _rows(n, groups, nb, gen)
    if quant:
        gi = torch.randint(-32, 33, (n,), generator=gen, device="cuda", dtype=torch.int32)
        hi = torch.randint(0, 65, (n,), generator=gen, device="cuda", dtype=torch.int32)
        out = ops.histogram(rows, (gi << 16) | hi, [nb] * groups, quant=True, quant_bins=64, rows_per_block=512, lane_mode=1)
        assert torch.equal(out[:, 0], _reference(rows, groups, nb, gi).long()) and torch.equal(out[:, 1], _reference(rows, groups, nb, hi).long())
    else:
        gh = torch.randint(-8, 9, (n, 2), generator=gen, device="cuda").float() / 8   # sums of a coarse grid: exact in fp32
        out = ops.histogram(rows, gh, [nb] * groups, quant=False, rows_per_block=512, lane_mode=2)
        for k in range(2):
            assert torch.equal(out[:, k], _reference(rows, groups, nb, gh[:, k]))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 148 * 8 * 256 * 4 + 3])
def test_quantize_walks_every_row(n):
    from falcata_b200 import ops
    g = torch.randn(n, device="cuda"); h = torch.rand(n, device="cuda")
    packed, scales, sums = ops.quantize(g, h, 64, False, seed=7, iter_key=3)
    assert torch.equal(scales, torch.stack([g.abs().max() / 32, h.max() / 64]))
    assert torch.equal(sums, torch.stack([(packed >> 16).long().sum(), (packed & 0xFFFF).long().sum()]))
    # rounding to the nearest level: half a level, and one unit in the last place of a product of at most 64
    assert float(((packed >> 16) * scales[0] - g).abs().max()) <= float(scales[0]) * (0.5 + 1e-5)
    # the same words from buffers that allow no 16-byte access
    if n > 4:
        g1 = torch.empty(n + 1, device="cuda")[1:]; g1.copy_(g); h1 = torch.empty(n + 1, device="cuda")[1:]; h1.copy_(h)
        assert torch.equal(ops.quantize(g1, h1, 64, False, seed=7, iter_key=3)[0], packed)


@pytest.mark.parametrize("extra", [{}, {"bagging_fraction": 0.7, "bagging_freq": 1}, {"grow_policy": "leaf"}, {"use_missing": True, "nan": 0.2}])
@pytest.mark.parametrize("n", [2047, 2049, 150001])
def test_one_launch_partition_gives_the_same_model(n, extra):
    """More chunks of a split than one look-back window (32 x 2048 rows), a window that is one chunk, and one row more."""
    X, y = make_binary(n, 12)
    extra = dict(extra)
    X[np.random.RandomState(0).rand(*X.shape) < extra.pop("nan", 0.0)] = np.nan
    p = dict({"objective": "binary", "num_leaves": 63, "max_bin": 63, "verbosity": -1, "quant_mode": "stochastic", "quant_bins": 4, "device_type": "cuda", "min_data_in_leaf": 3}, **extra)
    models = [model_body(fb.train(dict(p, cuda_plan=plan), fb.Dataset(X, y), 5).model_to_string()) for plan in ("auto", "auto,fused_scan:off")]
    assert models[0] == models[1]


@pytest.mark.parametrize("polls", [0, 1, 4096])
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 32 * 2048, 33 * 2048 + 1, 65 * 2048 + 5, 400001])
def test_one_launch_partition(n, polls):
    """Windows of one chunk, of a whole look-back window (32 chunks before the last) and of several. Without polls every chunk
    counts the rows of all chunks before it: the way out of a wait for a predecessor that does not publish."""
    from falcata_b200 import ops
    gen = torch.Generator(device="cuda"); gen.manual_seed(n)
    rows = torch.randint(0, 64, (n, 16), generator=gen, device="cuda", dtype=torch.int32).to(torch.uint8)
    perm = torch.randperm(n, generator=gen, device="cuda").int()
    for idx in (None, perm):
        order = torch.arange(n, device="cuda", dtype=torch.int32) if idx is None else idx
        for threshold in (-1, 20, 63):
            out, left = ops.partition_one_launch(rows, idx, 5, threshold, num_bin=64, polls=polls)
            go_left = rows[order.long(), 5].int() <= threshold
            assert left == int(go_left.sum()) and torch.equal(out, torch.cat([order[go_left], order[~go_left].flip(0)]))


def test_partition_of_no_rows_sets_up_the_children():
    """A rank of several may hold none of a split's rows: there is nothing to move, but the left count (zero) is due."""
    from falcata_b200 import ops
    rows = torch.zeros(4, 16, dtype=torch.uint8, device="cuda")
    out, left = ops.partition(rows, torch.empty(0, dtype=torch.int32, device="cuda"), 0, 3)
    assert out.numel() == 0 and left == 0


@pytest.mark.parametrize("flip", ["fused_scan:off", "fused_tail:off,fused_scan:off", "device_controller:off"])
@pytest.mark.parametrize("max_bin", [15, 63])
@pytest.mark.parametrize("n", [2049, 30000, 150001])
def test_fp32_sums_do_not_depend_on_the_partition_form(n, max_bin, flip):
    """fp32 histograms of at most 64 bins are sums in the order of a leaf's rows: every form of the partition leaves the same
    order, and every level loop ends its blocks at the same rows."""
    X, y = make_binary(n, 20)
    p = {"objective": "binary", "num_leaves": 63, "max_bin": max_bin, "verbosity": -1, "quant_mode": "none", "device_type": "cuda", "min_data_in_leaf": 5}
    models = [model_body(fb.train(dict(p, cuda_plan=plan), fb.Dataset(X, y), 8).model_to_string()) for plan in ("auto", "auto," + flip)]
    assert models[0] == models[1]


@pytest.mark.parametrize("grow", ["level", "leaf"])
@pytest.mark.parametrize("rate", [1e-39, 3e-38, 2.0 ** -100, 1e-20])
def test_leaf_outputs_of_any_size_reach_the_scores(rate, grow):
    """Subnormal leaf outputs and scores, and outputs on both sides of the size from which reduction adds are used."""
    X, y = make_binary(3000, 5)
    p = {"objective": "binary", "num_leaves": 15, "verbosity": -1, "quant_mode": "stochastic", "device_type": "cuda", "learning_rate": rate, "boost_from_average": False, "grow_policy": grow}
    bst = fb.train(p, fb.Dataset(X, y), 1, keep_training_booster=True)
    expected = bst.predict(X, raw_score=True).astype(np.float32)   # one tree on scores of zero: its outputs, rounded once
    assert np.count_nonzero(expected) == len(expected) and np.array_equal(bst.train_score_tensor().cpu().numpy().reshape(-1), expected)


@pytest.mark.parametrize("features", [1, 8, 9, 16, 17, 40])
@pytest.mark.parametrize("max_bin", [7, 31, 32, 33, 64, 65, 127, 255])
def test_split_search_agrees_with_the_host(features, max_bin):
    rng = np.random.RandomState(features * 1000 + max_bin)
    X = rng.randn(3000, features).astype(np.float32)
    X[rng.rand(*X.shape) < 0.1] = np.nan
    # gradients of a custom L2 objective on a coarse grid are exact, so host and device quantize alike
    y = (np.nan_to_num(X).sum(axis=1) + rng.randn(3000) > 0).astype(np.float32)
    p = {"objective": "none", "num_leaves": 31, "max_bin": max_bin, "verbosity": -1, "quant_mode": "fixedpoint", "quant_bins": 16, "min_data_in_leaf": 5, "grow_policy": "level"}

    def fobj(preds, ds):
        raw = preds.cpu().numpy() if isinstance(preds, torch.Tensor) else np.asarray(preds)
        return (np.round((raw - y) * 8) / 8).astype(np.float32), np.ones_like(y)

    def trained(**kw):
        bst = fb.Booster(dict(p, **kw), fb.Dataset(X, y, params={"max_bin": max_bin}))
        bst.update(fobj=fobj)
        return model_body(bst.model_to_string())

    device = trained(device_type="cuda")
    assert device == trained(device_type="cuda", cuda_plan="auto,fused_tail:off")
    assert device == trained(device_type="cpu")


@pytest.mark.parametrize("missing", ["none", "nan", "zero"])
@pytest.mark.parametrize("features", [1, 9, 17])
@pytest.mark.parametrize("max_bin", [7, 32, 33, 64, 65, 128, 129, 255])
def test_fp32_split_search_agrees_with_the_host(max_bin, features, missing):
    """fp64 prefix sums over staged fp32 histograms: runs of 1 to 8 bins per lane, with the bin of missing values at the end
    (NaN) or inside (zero). The gradients lie on a coarse grid, so all sums are exact and both learners see the same ones."""
    rng = np.random.RandomState(features * 1000 + max_bin)
    X = rng.randn(3000, features).astype(np.float32)
    if missing != "none":
        X[rng.rand(*X.shape) < 0.1] = np.nan if missing == "nan" else 0.0
    y = (np.round((np.nan_to_num(X).sum(axis=1) + np.isnan(X[:, 0]) + rng.randn(3000)) * 8) / 8).astype(np.float32)
    p = {"objective": "none", "num_leaves": 31, "max_bin": max_bin, "verbosity": -1, "quant_mode": "none", "min_data_in_leaf": 5, "grow_policy": "level"}

    def trained(**kw):
        bst = fb.Booster(dict(p, **kw), fb.Dataset(X, y, params={"max_bin": max_bin, "zero_as_missing": missing == "zero"}))
        bst.update(fobj=lambda preds, ds: (-y, np.ones_like(y)))
        return model_body(bst.model_to_string())

    device = trained(device_type="cuda")
    assert device == trained(device_type="cuda", cuda_plan="auto,fused_tail:off")
    assert device == trained(device_type="cpu")


@pytest.mark.parametrize("zero_as_missing", [False, True])
@pytest.mark.parametrize("quant", ["fixedpoint", "none"])
@pytest.mark.parametrize("levels", [20, 33, 66, 130, 200])
def test_search_of_bundled_features_agrees_with_the_host(levels, quant, zero_as_missing):
    """Exclusive sparse columns share a byte column; the bin of zero, which lies between the negative and the positive values, is
    not stored there and the search reconstructs it: in runs of 1, 2, 4 and 8 bins per lane."""
    rng = np.random.RandomState(levels)
    n, columns = 6000, [levels, 24, 12, 12]
    which = rng.randint(0, len(columns), size=n)
    X = np.zeros((n, len(columns) + 1), dtype=np.float32)
    for j, k in enumerate(columns):
        rows = np.flatnonzero(which == j)
        v = rng.randint(1, k + 1, size=len(rows)).astype(np.float32) - k // 3   # a third of the values is negative
        X[rows, j] = np.where(v <= 0, v - 1, v)
    X[:, -1] = rng.randn(n)
    # gradients of a custom L2 objective on a coarse grid: sums of 6000 of them are exact in fp32, so both learners see the same sums
    y = (np.round((X.sum(axis=1) % 7 + which + rng.randn(n)) * 8) / 8).astype(np.float32)
    p = {"objective": "none", "num_leaves": 31, "max_bin": 255, "verbosity": -1, "quant_mode": quant, "quant_bins": 16, "min_data_in_leaf": 5, "grow_policy": "level"}
    bodies = []
    for device in ("cuda", "cpu"):
        data = fb.Dataset(X, y, params={"max_bin": 255, "min_data_in_bin": 1, "zero_as_missing": zero_as_missing})
        bst = fb.Booster(dict(p, device_type=device), data)
        assert data.info()["num_groups"] < X.shape[1]
        bst.update(fobj=lambda preds, ds: (-y, np.ones_like(y)))
        bodies.append(model_body(bst.model_to_string()))
    assert bodies[0] == bodies[1]
    assert any(int(t) < len(columns) for line in bodies[0].splitlines() if line.startswith("split_feature=") for t in line.split("=")[1].split())


@pytest.mark.parametrize("missing", [False, True])
def test_nan_leaf_outputs(missing):
    """Rows that reach a NaN leaf get NaN, all others the same bits as without it: the same kernel adds them in the same order."""
    rng = np.random.RandomState(9)
    X = rng.randn(4000, 12).astype(np.float32)
    if missing:
        X[rng.rand(*X.shape) < 0.1] = np.nan
    bst = _forest(300, 31, 12, 2, X)
    x = torch.from_numpy(X[:1500]).cuda()
    before = bst.predict(x, raw_score=True).cpu().numpy().reshape(-1)
    leaf = np.asarray(bst.predict(X[:1500], pred_leaf=True)).reshape(1500, -1)
    hit = np.zeros(1500, dtype=bool)
    for tree in (0, 7, 299):
        bst.set_leaf_output(tree, int(leaf[tree, tree]), float("nan"))
        hit |= leaf[:, tree] == leaf[tree, tree]
    after = bst.predict(x, raw_score=True).cpu().numpy().reshape(-1)
    assert 0 < hit.sum() < 1500 and np.isnan(after[hit]).all() and np.array_equal(after[~hit], before[~hit])
    assert np.array_equal(bst.predict(x, pred_leaf=True).cpu().numpy().reshape(1500, -1), leaf)


def test_several_threads_predict_at_once():
    """Forests large enough to be packed by a team of threads, predicted by several threads at a time: each gets its own answer."""
    import threading
    rng = np.random.RandomState(3)
    X = rng.randn(4000, 30).astype(np.float32)
    boosters = [_forest(150 + 20 * k, 127, 30, k, X) for k in range(3)]   # about 38k nodes and more
    x = torch.from_numpy(X[:500]).cuda()
    alone = [(b.predict(x, raw_score=True).clone(), b.predict(x, pred_leaf=True).clone()) for b in boosters]
    same = [False] * 6

    def work(i):
        b, (score, leaf) = boosters[i % 3], alone[i % 3]
        same[i] = all(torch.equal(b.predict(x, raw_score=True), score) and torch.equal(b.predict(x, pred_leaf=True), leaf) for _ in range(5))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(same)


def _forest(trees, leaves, features, seed, X):
    rng = np.random.RandomState(seed)
    y = (X[:, 0] + rng.randn(len(X)) > 0).astype(np.float32)
    # random labels and one feature per split from all of them: every feature is used by some tree
    return fb.train({"objective": "binary", "num_leaves": leaves, "verbosity": -1, "min_data_in_leaf": 1, "min_sum_hessian_in_leaf": 0, "feature_fraction": 0.05 if features > 60 else 0.5,
                     "seed": seed}, fb.Dataset(X, y), trees)


@pytest.mark.parametrize("rows,features,trees,leaves", [(1, 5, 3, 7), (31, 40, 70, 31), (33, 152, 60, 63), (148 * 32 + 1, 152, 40, 255), (40001, 155, 40, 63), (3001, 320, 40, 127), (257, 12, 9, 1500)])
def test_predict_tiles_match_the_host(rows, features, trees, leaves):
    rng = np.random.RandomState(rows)
    X = rng.randn(max(rows, 4000), features).astype(np.float32)
    bst = _forest(trees, leaves, features, 1, X)
    x = X[:rows]
    # leaf values and the sums are rounded to fp32 once each: 2^-23 of the largest partial sum, far below 1e-5
    for t in (torch.from_numpy(x).cuda(), torch.from_numpy(x.astype(np.float64)).cuda()):
        np.testing.assert_allclose(bst.predict(t, raw_score=True).cpu().numpy().reshape(-1), np.asarray(bst.predict(x, raw_score=True)).reshape(-1), rtol=1e-5, atol=1e-5)
    host = np.asarray(bst.predict(x, pred_leaf=True)).reshape(rows, -1)
    rc, leaf = _device_leaves(bst, torch.from_numpy(x).cuda(), trees)
    assert rc == 0 and np.array_equal(leaf, host)


def _device_leaves(bst, x, trees):
    """Leaf indices by the device entry point itself: ``Booster.predict`` would take what the device refuses to the host."""
    from falcata_b200.basic import _lib
    out = torch.full((x.shape[0], trees), -1, dtype=torch.int32, device="cuda")
    code = {torch.float32: 0, torch.float64: 1, torch.float16: 6}[x.dtype]
    rc = _lib().FB_BoosterPredictForDeviceMat(bst._handle, ctypes.c_void_p(x.data_ptr()), code, ctypes.c_int32(x.shape[0]), ctypes.c_int32(x.shape[1]), 1, 2, 0, -1,
                                              ctypes.c_void_p(out.data_ptr()))
    return rc, out.cpu().numpy()


@pytest.mark.parametrize("features", [156, 157, 330, 1215, 1216])
def test_leaf_indices_of_wide_forests(features):
    """Up to 1215 used features (32 rows a tile) the device gives the host's leaves for fp32 and half rows; double rows, which the
    host compares in double, are the device's up to 156 and the host's beyond."""
    rng = np.random.RandomState(features)
    X = rng.randn(1000, features).astype(np.float16).astype(np.float32)
    # two halves of one feature each round: a round per feature, and every feature is used
    trees = features
    body = "".join(f"Tree={j}\nnum_leaves=3\nnum_cat=0\nsplit_feature={j} {(j * 7 + 3) % features}\nthreshold={float(np.median(X[:, j]))!r} 0.25\ndecision_type=2 2\n"
                   f"left_child=1 -1\nright_child=-2 -3\nleaf_value=0.5 -0.25 0.125\nis_linear=0\nshrinkage=1\n\n\n" for j in range(trees))
    bst = fb.Booster(model_str=f"tree\nversion=v4\nnum_class=1\nnum_tree_per_iteration=1\nlabel_index=0\nmax_feature_idx={features - 1}\nobjective=regression\n"
                               f"feature_names={' '.join(f'Column_{j}' for j in range(features))}\nfeature_infos={' '.join(['[-5:5]'] * features)}\n\n{body}end of trees\n")
    host = np.asarray(bst.predict(X, pred_leaf=True)).reshape(len(X), -1)
    for dtype in (torch.float32, torch.float16, torch.float64):
        x = torch.from_numpy(X).cuda().to(dtype)
        rc, leaf = _device_leaves(bst, x, trees)
        assert (rc == 0) == (features <= (156 if dtype is torch.float64 else 1215))
        if rc == 0:
            assert np.array_equal(leaf, host)
        assert np.array_equal(bst.predict(x, pred_leaf=True).cpu().numpy().reshape(len(X), -1), host)


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("sizes,levels", [([1, 2, 29, 30, 31, 33, 64], 5), ([128, 1, 90], 5), ([600, 3], 5), ([40, 65], 70)])
@pytest.mark.parametrize("truncation", [1, 30, 31, 64, 1000])
def test_lambdarank_pairs_agree_with_the_host(truncation, sizes, levels, norm, monkeypatch):
    """Gradients of single documents at truncations below, at and above the query lengths: the tree puts every document into a
    leaf of its own, so the new scores are -g / (h + 1) of that document. (600 documents: blocks of 256 threads; 70 label levels:
    the scan instead of the counts.)"""
    rng = np.random.RandomState(truncation + len(sizes))
    n = sum(sizes)
    X = np.column_stack([np.arange(n) // 25, np.arange(n) % 25]).astype(np.float32)
    y = rng.randint(0, levels, size=n).astype(np.float32)
    start = rng.randn(n)
    p = {"objective": "lambdarank", "num_leaves": 1000, "max_bin": 255, "min_data_in_leaf": 1, "min_sum_hessian_in_leaf": 0, "lambda_l2": 1.0, "learning_rate": 1.0, "verbosity": -1,
         "quant_mode": "none", "device_type": "cuda", "grow_policy": "level", "lambdarank_truncation_level": truncation, "lambdarank_norm": norm, "boost_from_average": False,
         "label_gain": ",".join(str(2 ** k - 1 if levels <= 31 else k) for k in range(levels))}

    def scores():
        data = fb.Dataset(X, y, group=np.asarray(sizes, dtype=np.int32), init_score=start, params={"min_data_in_bin": 1, "max_bin": 255})
        bst = fb.train(p, data, 1, keep_training_booster=True)
        return bst.train_score_tensor().cpu().numpy().reshape(-1) - start.astype(np.float32)

    device = scores()
    monkeypatch.setenv("FALCATA_HOST_GRADIENTS", "1")
    host = scores()
    assert np.count_nonzero(host) > 0
    # a document's sums run over up to 600 fp32 pairs on the device, and the step is the difference of two fp32 scores of up to 10:
    # 600 x 2^-24 of the step and 2^-20. A truncation off by one moves a hundred documents or more, most by 1e-3 and up
    np.testing.assert_allclose(device, host, rtol=1e-4, atol=1e-5)
