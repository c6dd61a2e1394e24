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
