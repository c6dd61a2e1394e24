"""The lane walk (trees that no other layout of the library's choice takes) and tree groups that fit
a shared-memory stage only once, at their edges: one row, ragged tiles, tree ranges split over warps
and blocks, fewer classes than warps, a class without trees."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _case(trees, levels, features, classes, rows, p):
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(11, trees, levels, features, p, 0.1, marg, num_classes=classes)
    if classes > 2:
        f.class_id[f.class_id == 1] = 2
    rng = np.random.Generator(np.random.PCG64(3))
    X = marg.sample_rows(rng, rows)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(300, 3 * rows)):
        g = split[(i * 37) % len(split)]
        X[(i * 13) % rows, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    if rows > 4:
        X[3, :], X[4, 0] = np.nan, np.inf
    return f, X


def _check(df, f, X):
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    dX = torch.from_numpy(X).cuda()
    assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
    got, part = df.predict(dX).cpu().numpy(), df.predict_partial(dX)
    df.check_status()
    if f.num_classes:
        _, sums = oracle.predict(f, X, class_sums=True)
        sums[:, np.bincount(f.class_id, minlength=f.num_classes) == 0] = f.initial_value
        best, cls = sums.max(axis=1), got.astype(int)
        assert (sums[np.arange(len(X)), cls] >= best - 1e-5 * np.abs(best) - 1e-5).all()
        assert np.allclose(part.cpu().numpy() + f.initial_value, sums, rtol=1e-5, atol=1e-5)
        assert np.array_equal(df.predict(dX, int8=True).cpu().numpy(), cls.astype(np.int8))
    else:
        assert_predictions_close(got, want)
        assert_predictions_close(df.finalize(part).cpu().numpy(), want)


@pytest.mark.parametrize("trees,levels,features,classes,rows", [
    (1, 14, 3, 0, 1), (7, 13, 33, 0, 33), (200, 16, 32, 0, 5000), (60, 13, 200, 0, 70001), (30, 10, 9, 3, 777),
    (120, 14, 20, 12, 40001)])
def test_lane_walk(trees, levels, features, classes, rows):
    f, X = _case(trees, levels, features, classes, rows, 0.25)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    assert df.info().staged == 0 and df.info().schedule.feature_bits == 32
    _check(df, f, X)
    out = torch.empty(1, device="cuda")
    dX = torch.from_numpy(X[:1]).cuda()   # the variant that may not allocate
    kernels._check(kernels.lib().tbk_predict_noalloc(df._h, dX.data_ptr(), 1, features, out.data_ptr(), kernels.OUT_F32,
                                                     torch.cuda.current_stream().cuda_stream))
    assert abs(float(out[0] - df.predict(dX)[0])) < 1e-5


@pytest.mark.parametrize("trees,classes,rows", [(1000, 0, 65536), (2000, 0, 65536), (4000, 0, 2048), (60, 0, 65536), (1200, 3, 40000)])
def test_long_lane_walks_round_their_sums_once(trees, classes, rows):
    f, X = _case(trees, 14, 16, classes, rows, 0.25)
    X = np.nan_to_num(X, nan=0.0, posinf=3.0)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    part = df.predict_partial(torch.from_numpy(X).cuda())[-3000:].double().cpu().numpy()
    df.check_status()
    info = df.info()
    assert info.layout == kernels.LAYOUT_LANES
    _, ids = oracle.predict(f, X[-3000:], leaf_ids=True)
    leaves = f.thr[f.tree_off[:-1][None, :] + ids].astype(np.float64)
    groups = [f.class_id == c for c in range(classes)] if classes else [np.ones(trees, bool)]
    for c, g in enumerate(groups):
        exact, got = leaves[:, g].sum(axis=1), part[:, c]
        # half an ulp for every rounding, of a sum about as large as the result: a share's or a chunk's and
        # the result's for long chains; one per leaf, of random sign, for chains of up to 64 leaves in fp32
        chain = g.sum() / (info.schedule.tree_chunks * (1 if classes else info.schedule.tree_threads))
        roundings = 3 if chain > 64 else 3 + np.sqrt(64)
        assert np.linalg.norm(got - exact) <= roundings * 2.0 ** -24 * np.linalg.norm(exact)


@pytest.mark.parametrize("tile,rows", [(2, 3001), (2, 20000)])
def test_groups_that_fit_one_stage(tile, rows):
    f, X = _case(70, 8, 20, 0, rows, 0.1)
    df = kernels.DeviceForest(f, representation="sparse", tile_size=tile, batch_hint=rows)
    assert df.info().staged == 1 and df.info().smem_bytes > 100 * 1024
    _check(df, f, X)
