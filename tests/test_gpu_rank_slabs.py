"""Rows ranked with lane = feature (slabs of 32 features), and one-byte rank keys over wide rows: row widths on both
sides of a slab, of a line of keys and of the widths where four tiles of keys fit; batches ranked through either kernel;
values that equal thresholds, NaN, infinities, whole numbers.  Leaf ids are exact."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _forest(trees, levels, features, seed=3):
    return synth.generate_forest(seed, trees, levels, features, 0.05, 0.1, synth.Marginal("normal", features), synth.IDENTITY, 0)


def _rows(f, n, features, whole=False, seed=1):
    X = np.random.default_rng(seed).standard_normal((n, features)).astype(np.float32)
    if whole:
        X = np.round(X * 3).astype(np.float32)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(2000, 4 * n)):
        g = split[(i * 37) % len(split)]
        X[(i * 11) % n, f.feat[g]] = f.thr[g]
    X[1 % n, :] = np.nan
    X[2 % n, ::2] = np.inf
    X[3 % n, ::3] = -np.inf
    return X


def _check(f, X, rows=None, **options):
    from treebeard_b200 import kernels
    n = len(X)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=n, **options)
    assert df.info().layout == kernels.LAYOUT_RANK_KEYS
    rows = torch.from_numpy(X).cuda() if rows is None else rows
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    ids = df.predict_leaf_ids(rows).cpu().numpy()
    df.check_status()
    assert bool(df.info().reserved[2] & kernels.RAN_SLABS) == (n * f.num_features > 148 * 2048 and f.num_features > 64)
    assert np.array_equal(ids, want_ids)
    got = df.predict(rows).cpu().numpy()
    part = df.finalize(df.predict_partial(rows)).cpu().numpy()
    df.check_status()
    assert_predictions_close(got, want)
    assert_predictions_close(part, want)
    return df


# 148 SMs x 2048 values is the least that is ranked in slabs
@pytest.mark.parametrize("features,trees,levels", [(65, 40, 7), (95, 40, 7), (96, 33, 7), (97, 200, 8), (130, 300, 6), (511, 100, 8)])
@pytest.mark.parametrize("whole", [False, True])
def test_slabs(features, trees, levels, whole):
    f = _forest(trees, levels, features)
    if whole:
        f.thr = np.where(f.left >= 0, np.round(f.thr * 3), f.thr).astype(np.float32)
    _check(f, _rows(f, 148 * 2048 // features + 45, features, whole))


@pytest.mark.parametrize("features", [512, 513, 543, 545, 960, 1100, 1501, 2000, 2018])
@pytest.mark.parametrize("rows", [1, 33, 5003])
def test_one_byte_keys(features, rows):
    f = _forest(200, 8 if features != 960 else 6, features)
    _check(f, _rows(f, rows, features))


def test_one_byte_keys_whole_numbers_strides_and_chunks():
    f = _forest(250, 7, 700)
    f.thr = np.where(f.left >= 0, np.round(f.thr * 3), f.thr).astype(np.float32)
    X = _rows(f, 3001, 700, True)
    flat = torch.full((5 + 3001 * 703,), float("nan"), device="cuda")
    rows = flat[5:].view(3001, 703)[:, :700]
    rows.copy_(torch.from_numpy(X))
    df = _check(f, X, rows)
    again = _check(f, X, rows, tree_chunks=3)
    assert_predictions_close(again.predict(rows).cpu().numpy(), df.predict(rows).cpu().numpy())


def test_one_byte_keys_in_several_passes():
    """More rows than the keys of one pass hold; the last pass is short."""
    from treebeard_b200 import kernels
    f = _forest(200, 6, 2000)
    n = 60001
    X = _rows(f, n, 2000)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=n)
    got = df.predict(torch.from_numpy(X).cuda()).cpu().numpy()
    df.check_status()
    some = np.r_[0:300, 47000:47700, n - 300:n]
    assert_predictions_close(got[some], oracle.predict(f, X[some]))


def test_more_thresholds_than_a_byte_holds_keep_rounded_keys():
    from treebeard_b200 import kernels
    f = _forest(200, 6, 600)
    split = f.left >= 0
    f.feat = np.where(split, f.feat % 7, f.feat).astype(f.feat.dtype)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=5000)
    assert df.info().layout == kernels.LAYOUT_ROUNDED_KEYS
    X = _rows(f, 500, 600)
    assert np.array_equal(df.predict_leaf_ids(torch.from_numpy(X).cuda()).cpu().numpy(), oracle.predict(f, X, leaf_ids=True)[1])


def test_one_byte_keys_without_allocation():
    """tbk_predict_noalloc takes the widths that it took on rounded keys: rows that an fp32 tile could hold."""
    from treebeard_b200 import kernels
    f = _forest(200, 6, 700)
    X = _rows(f, 9001, 700)
    rows = torch.from_numpy(X).cuda()
    df = kernels.DeviceForest(f, representation="auto", batch_hint=len(X))
    out = torch.empty(len(X), device="cuda")
    kernels._check(kernels.lib().tbk_predict_noalloc(df._h, rows.data_ptr(), len(X), 700, out.data_ptr(), kernels.OUT_F32, None))
    torch.cuda.synchronize()
    df.check_status()
    assert_predictions_close(out.cpu().numpy(), oracle.predict(f, X))
    f = _forest(100, 6, 2000)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=100)
    rows = torch.zeros((100, 2000), device="cuda")
    with pytest.raises(kernels.TbkError, match="16-bit key"):
        kernels._check(kernels.lib().tbk_predict_noalloc(df._h, rows.data_ptr(), 100, 2000, out.data_ptr(), kernels.OUT_F32, None))


@pytest.mark.parametrize("features,stride", [(130, 480000), (600, 1 << 20)])
def test_slabs_take_rows_of_a_wide_table(features, stride):
    """A column range of a table so wide that the rows lie further apart than 32 bits of bytes reach."""
    from treebeard_b200 import kernels
    f = _forest(60, 6, features)
    n = 148 * 2048 // features + 45
    assert 4 * stride * n > 1 << 31
    X = _rows(f, n, features)
    table = torch.empty(7 + n * stride, device="cuda")
    rows = table[7:].view(n, stride)[:, :features]
    rows.copy_(torch.from_numpy(X))
    df = _check(f, X, rows)
    assert df.info().reserved[2] & kernels.RAN_SLABS


def _crowded(f, seed):
    """Thresholds of every feature that crowd in one bucket of its table, whatever the number of buckets (up to eight for
    each threshold), by kind of feature: within a unit around 1, with one far off; within a unit below one far off; over a range
    that fp32 cannot divide; between two neighbouring numbers; all over the range (not crowded)."""
    g = np.random.default_rng(seed)
    split = np.nonzero(f.left >= 0)[0]
    thr = f.thr.copy()
    far = {}
    for k in split:
        i = int(f.feat[k])
        kind = i % 5
        if kind == 0:
            thr[k] = 1 + g.random(dtype=np.float32)
        elif kind == 1:
            thr[k] = 5e6 + np.float32(g.integers(0, 200) / 2)
        elif kind == 2:
            thr[k] = np.float32(g.random() * 10)
        elif kind == 3:
            thr[k] = np.nextafter(np.float32(1), np.float32(1 + g.integers(0, 2)))
        far.setdefault(i, k)
    for i, k in far.items():
        thr[k] = {0: -1e7, 1: -3e6, 2: -3.2e38, 3: thr[k], 4: thr[k]}[i % 5]
    far2 = {}
    for k in split[::-1]:
        i = int(f.feat[k])
        if i % 5 == 2 and i not in far2 and far[i] != k:
            far2[i] = k
            thr[k] = 3.2e38
    f.thr = thr
    return f


@pytest.mark.parametrize("features,trees,levels", [(65, 40, 7), (100, 60, 8), (511, 100, 8), (512, 100, 8), (700, 150, 8), (2000, 300, 8)])
def test_crowded_thresholds(features, trees, levels):
    """Buckets that take more search steps than the variants with a number of steps of their own have."""
    f = _crowded(_forest(trees, levels, features), features)
    split = f.left >= 0
    crowd = max(len(np.unique(f.thr[split & (f.feat == i)])) for i in range(0, features, 5))
    assert 8 < crowd - 1 <= 255   # thresholds in one bucket: four search steps and more
    n = 148 * 2048 // features + 45
    X = _rows(f, n, features)
    g = np.random.default_rng(2)
    at = np.nonzero(split)[0]
    for i in range(features):     # both sides of the feature's thresholds
        mine = f.thr[at[f.feat[at] == i]]
        if len(mine):
            pick = mine[g.integers(0, len(mine), n - 4)]
            X[4:, i] = np.nextafter(pick, np.float32([-np.inf, np.inf])[g.integers(0, 2, n - 4)])
            X[4::3, i] = pick[::3]
    _check(f, X)


@pytest.mark.parametrize("features,hint", [(1500, 32768), (1750, 70000), (2000, 262144)])
def test_one_byte_keys_whatever_the_announced_batch(features, hint):
    from treebeard_b200 import kernels
    f = _forest(800, 3, features)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=hint)
    assert df.info().layout == kernels.LAYOUT_RANK_KEYS
    X = _rows(f, 300, features)
    assert np.array_equal(df.predict_leaf_ids(torch.from_numpy(X).cuda()).cpu().numpy(), oracle.predict(f, X, leaf_ids=True)[1])


@pytest.mark.parametrize("most,ranks", [(255, True), (256, False)])
@pytest.mark.parametrize("used", [0, 300, 599])
def test_the_most_thresholds_that_a_byte_holds(most, ranks, used):
    """One feature with `most` distinct thresholds, each of them several times, and all others with fewer."""
    from treebeard_b200 import kernels
    f = _forest(40, 7, 600)
    split = np.nonzero(f.left >= 0)[0]
    mine = split[::5]
    assert len(mine) > 3 * most
    f.feat = np.where(f.left >= 0, np.where(f.feat == used, (used + 1) % 600, f.feat), f.feat).astype(f.feat.dtype)
    f.feat[mine] = used
    f.thr[mine] = (np.arange(len(mine)) % most / 64).astype(np.float32)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=500)
    assert df.info().layout == (kernels.LAYOUT_RANK_KEYS if ranks else kernels.LAYOUT_ROUNDED_KEYS)
    X = _rows(f, 500, 600)
    X[4:, used] = np.random.default_rng(1).integers(-20, 300, 496) / np.float32(64)
    assert np.array_equal(df.predict_leaf_ids(torch.from_numpy(X).cuda()).cpu().numpy(), oracle.predict(f, X, leaf_ids=True)[1])


@pytest.mark.parametrize("features,levels,fits", [(2019, 8, True), (2024, 8, True), (2025, 8, False), (2044, 7, True), (2045, 7, False)])
def test_widest_one_byte_keys(features, levels, fits):
    from treebeard_b200 import kernels
    f = _forest(70, levels, features)
    for n in (1, 33, 3001):
        X = _rows(f, n, features)
        if fits:
            _check(f, X)
            _check(f, X, tree_chunks=2)
        else:
            df = kernels.DeviceForest(f, representation="auto", batch_hint=n)
            assert df.info().layout == kernels.LAYOUT_TILES   # (too wide for rounded keys too)
            ids = df.predict_leaf_ids(torch.from_numpy(X).cuda()).cpu().numpy()
            assert np.array_equal(ids, oracle.predict(f, X, leaf_ids=True)[1])
