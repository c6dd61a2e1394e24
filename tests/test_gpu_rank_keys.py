"""Rank keys (forests of at most 8 levels) at the edges of their kernels:
unit and batch sizes of the walks, rows in pairs, one by one and in tiles, groups of mixed depth, classes that
share a group of trees, more thresholds than the half-precision comparison holds, and the direct
and the shared-memory ranking of rows."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _forest(trees, levels, features, classes=0, p=0.2, seed=5, whole=False):
    marg = synth.Marginal("int16" if whole else "normal", features)
    f = synth.generate_forest(seed, trees, levels, features, p, 0.1, marg, num_classes=classes)
    if classes:   # uneven classes, one of them empty: several class boundaries fall into one group
        rng = np.random.Generator(np.random.PCG64(seed))
        f.class_id[:] = np.minimum(rng.integers(0, classes, trees), rng.integers(0, classes, trees))
        f.class_id[f.class_id == 1] = 2
    return f, marg


def _rows(f, marg, n, seed=9):
    rng = np.random.Generator(np.random.PCG64(seed))
    X = marg.sample_rows(rng, n)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(400, 4 * n)):   # values equal to thresholds, and their neighbours
        g = split[(i * 37) % len(split)]
        X[(i * 13) % n, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    if n > 6:
        X[3, :], X[4, 0], X[5, f.num_features - 1] = np.nan, np.inf, -np.inf
    return X


@pytest.mark.parametrize("trees,levels,features,classes,rows", [
    (1, 1, 1, 0, 1), (31, 2, 32, 0, 79), (33, 3, 33, 0, 81), (100, 6, 8, 0, 320), (97, 8, 64, 0, 321),
    (300, 7, 20, 0, 148 * 80 * 4 + 77), (64, 8, 28, 3, 5), (45, 5, 16, 7, 12003), (400, 8, 40, 26, 2500),
    (140, 8, 1, 0, 4000), (1, 3, 65, 0, 1), (33, 8, 90, 0, 129), (90, 7, 111, 0, 148 * 128 * 3 + 5),
    (70, 6, 511, 0, 2000), (40, 8, 300, 0, 30011)])
def test_rank_key_walk_is_exact(trees, levels, features, classes, rows):
    f, marg = _forest(trees, levels, features, classes, p=0.0 if features == 1 and trees > 1 else 0.2)
    X = _rows(f, marg, rows)
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    assert df.info().schedule.feature_bits == 16
    dX = torch.from_numpy(X).cuda()
    ids = df.predict_leaf_ids(dX).cpu().numpy()
    df.check_status()
    assert np.array_equal(ids, want_ids)
    got, part = df.predict(dX), df.predict_partial(dX)
    df.check_status()
    if classes:
        _, sums = oracle.predict(f, X, class_sums=True)
        sums[:, np.bincount(f.class_id, minlength=classes) == 0] = f.initial_value   # classes without trees
        best = sums.max(axis=1)
        cls = got.cpu().numpy().astype(int)
        assert (sums[np.arange(rows), cls] >= best - 1e-5 * np.abs(best) - 1e-5).all()
        assert np.allclose(part.cpu().numpy() + f.initial_value, sums, rtol=1e-5, atol=1e-5)
        assert np.array_equal(df.predict(dX, int8=True).cpu().numpy(), cls.astype(np.int8))
    else:
        assert_predictions_close(got.cpu().numpy(), want)
        assert_predictions_close(df.finalize(part).cpu().numpy(), want)


def test_rank_keys_on_several_streams_and_in_a_graph():
    """Every stream has its own key memory; a captured call keeps the memory it was captured with."""
    f, marg = _forest(200, 8, 28)
    batches = [torch.from_numpy(_rows(f, marg, 3000 + 500 * i, seed=i)).cuda() for i in range(6)]
    df = kernels.DeviceForest(f, representation="auto", batch_hint=3000)
    want = [df.predict(b).clone() for b in batches]
    streams = [torch.cuda.Stream() for _ in batches]
    torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for b, s in zip(batches, streams):
            with torch.cuda.stream(s):
                got.append(df.predict(b))
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    out = torch.empty_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        df.predict(batches[0], out=out)
    out.zero_()
    graph.replay()
    other = df.predict(batches[1])
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and torch.equal(other, want[1])
    df.check_status()


@pytest.mark.parametrize("trees,levels,features,classes,rows", [
    (33, 6, 20, 0, 1), (97, 8, 64, 0, 70001), (140, 8, 300, 0, 9003), (60, 6, 16, 5, 30011), (40, 6, 700, 0, 1005)])
def test_the_call_that_may_not_allocate(trees, levels, features, classes, rows):
    f, marg = _forest(trees, levels, features, classes)
    dX = torch.from_numpy(_rows(f, marg, rows)).cuda()
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    want, out = df.predict(dX), torch.empty(rows, device="cuda")
    for _ in range(2):
        kernels._check(kernels.lib().tbk_predict_noalloc(df._h, dX.data_ptr(), rows, features, out.data_ptr(), kernels.OUT_F32,
                                                         torch.cuda.current_stream().cuda_stream))
        df.check_status()
        if classes:
            assert (out == want).float().mean() > 0.999   # (other tree chunks: near-ties may fall either way)
        else:
            assert_predictions_close(out.cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("rows", [1, 1005, 9601])
def test_the_call_that_may_not_allocate_on_rounded_keys(rows):
    """Wide rows whose keys are asked for, or whose batches are not announced, stay on rounded keys."""
    f, marg = _forest(40, 6, 700)
    dX = torch.from_numpy(_rows(f, marg, rows)).cuda()
    for options in (dict(batch_hint=rows, feature_bits=16), {}):
        df = kernels.DeviceForest(f, representation="auto", **options)
        assert df.info().layout == kernels.LAYOUT_ROUNDED_KEYS
        want, out = df.predict(dX), torch.empty(rows, device="cuda")
        kernels._check(kernels.lib().tbk_predict_noalloc(df._h, dX.data_ptr(), rows, 700, out.data_ptr(), kernels.OUT_F32,
                                                         torch.cuda.current_stream().cuda_stream))
        df.check_status()
        assert_predictions_close(out.cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("features", [490, 491, 506, 507, 511])
@pytest.mark.parametrize("rows", [300, 20011])
def test_widest_rank_key_rows_under_the_deepest_trees(features, rows):
    """One quad of tiles of 491 features and a ring of three 32 KB planes leave room for 8 walker warps,
    from 507 on for 4."""
    f, marg = _forest(40, 8, features)
    X = _rows(f, marg, rows)
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    assert df.info().schedule.feature_bits == 16
    dX = torch.from_numpy(X).cuda()
    assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
    got = df.predict(dX)
    df.check_status()
    assert_predictions_close(got.cpu().numpy(), want)


@pytest.mark.parametrize("features,rows,threads,rows_per_block", [
    (28, 1, 32 * 3, 4), (28, 5, 32 * 5, 12), (28, 80, 32 * 22, 80), (28, 148 * 320, 32 * 22, 320), (90, 300, None, None),
    (90, 50003, None, None), (511, 2000, 32 * 6, 128)])
def test_the_launch_that_is_reported_is_the_one_that_ran(features, rows, threads, rows_per_block):
    """A walker warp per four rows of a unit (one chunk asked for: the units then come from the rows alone)
    or per share of a quad, and two warps that copy."""
    f, marg = _forest(64, 8, features)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=70000, tree_chunks=1)
    df.predict(torch.from_numpy(_rows(f, marg, rows)).cuda())
    df.check_status()
    info = df.info()
    s = info.schedule
    assert info.layout == kernels.LAYOUT_RANK_KEYS and s.tree_chunks == 1
    if threads:
        assert (info.threads_per_block, s.rows_per_block) == (threads, rows_per_block)
    if features > 64:
        assert s.rows_per_block % 128 == 0 and info.threads_per_block == 32 * (s.rows_per_block // 128 * s.tree_threads + 2)
    else:
        assert s.tree_threads == 1


@pytest.mark.parametrize("features,rows", [(28, 1), (28, 9), (28, 10), (64, 4), (3, 79), (3, 80), (3, 81), (3, 85), (2, 128),
                                           (1, 161), (1, 256), (1, 257), (5, 300), (33, 640)])
def test_small_host_batches_on_either_side_of_what_travels_with_the_launch(features, rows):
    """Up to 256 values in the launch parameters, over one block of rows or several; beyond that rows in mapped
    memory.  A row stride that is wider than the row."""
    f, marg = _forest(70, 6, features, p=0.0 if features == 1 else 0.2)
    X = _rows(f, marg, rows)
    X[np.isnan(X)] = 0.5
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    wide = np.full((rows, features + 3), 7.5, np.float32)
    wide[:, :features] = X
    want = oracle.predict(f, X)
    for _ in range(2):
        assert_predictions_close(df.predict_host(X), want)
        assert_predictions_close(df.predict_host(wide[:, :features]), want)
    df.check_status()


@pytest.mark.parametrize("trees,levels,features,hint,tiles", [
    (30, 8, 400, 3000, True), (30, 8, 400, 300, False), (100, 6, 400, 5999, True), (101, 6, 400, 5999, False), (64, 8, 400, 10000, True),
    (64, 8, 400, 20000, False), (30, 8, 400, 0, False), (30, 8, 325, 3000, False), (30, 8, 326, 3000, True), (30, 8, 330, 3000, True), (30, 8, 330, 7000, False)])
def test_few_trees_over_several_hundred_features(trees, levels, features, hint, tiles):
    """Where ranking a row costs more than it saves the batches that are announced go through fp32 tiles: the
    same leaves as on rank keys, for whatever batch comes."""
    f, marg = _forest(trees, levels, features)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=hint)
    keys = kernels.DeviceForest(f, representation="auto", feature_bits=16, batch_hint=hint)
    assert df.info().layout == (kernels.LAYOUT_TILES if tiles else kernels.LAYOUT_RANK_KEYS)
    assert keys.info().layout == kernels.LAYOUT_RANK_KEYS
    for rows in (1, 700, 3001):
        X = _rows(f, marg, rows, seed=rows)
        want, want_ids = oracle.predict(f, X, leaf_ids=True)
        dX = torch.from_numpy(X).cuda()
        assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
        got = df.predict(dX)
        df.check_status()
        assert_predictions_close(got.cpu().numpy(), want)
        assert_predictions_close(keys.predict(dX).cpu().numpy(), want)
