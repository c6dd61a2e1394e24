"""Deep trees of one depth, whose leaf values are staged beside the nodes: every depth the kernel is made for, odd and
single trees, a shallower tree padded to the others' depth, ragged rows, the widest and narrowest blocks, ranges of trees."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _staged(df):
    return bool(df.info().reserved[2] & kernels.RAN_STAGED_LEAVES)


@pytest.mark.parametrize("levels", [9, 10, 11, 12])
@pytest.mark.parametrize("trees,features,rows,chunks", [
    (1, 3, 1, 0), (7, 16, 33, 0), (40, 128, 1000, 1), (41, 60, 5003, 3), (33, 140, 700, 1), (35, 24, 150001, 0)])
def test_staged_leaves(levels, trees, features, rows, chunks):
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(7, trees, levels, features, 0.03, 0.1, marg)
    if trees > 34:  # one tree of a single split among many deep ones
        a, b = f.tree_off[5], f.tree_off[6]
        keep = [a, a + f.left[a], a + f.right[a]]
        size = int(b - a)
        for name in ("left", "right", "feat", "thr"):
            v = getattr(f, name)
            setattr(f, name, np.concatenate([v[:a], v[keep], v[b:]]))
        f.left[a:a + 3], f.right[a:a + 3] = [1, -1, -1], [2, -1, -1]
        f.tree_off = f.tree_off.copy()
        f.tree_off[6:] -= size - 3
    X = marg.sample_rows(np.random.Generator(np.random.PCG64(5)), rows)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(3 * rows, 600)):
        g = split[(i * 37) % len(split)]
        X[(i * 13) % rows, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    if rows > 4:
        X[3, :], X[4, 0] = np.nan, np.inf
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows, tree_chunks=chunks)
    assert df.info().layout == kernels.LAYOUT_DEEP_KEYS
    dX = torch.from_numpy(X).cuda()
    some = slice(0, 3000)
    got = df.predict(dX)
    assert _staged(df)
    part = df.predict_partial(dX)
    assert _staged(df)
    df.check_status()
    want, want_ids = oracle.predict(f, X[some], leaf_ids=True)
    assert_predictions_close(got.cpu().numpy()[some], want)
    assert_predictions_close(df.finalize(part).cpu().numpy()[some], want)
    assert np.array_equal(df.predict_leaf_ids(dX[some]).cpu().numpy(), want_ids)
    # the same sums from the oracle's leaves, for the rest of a large batch
    if rows > 3000:
        tail = oracle.predict(f, X[-500:])
        assert_predictions_close(got.cpu().numpy()[-500:], tail)


@pytest.mark.parametrize("trees,features,rows,chunks", [(7, 90, 33, 0), (40, 200, 5003, 3), (41, 90, 20011, 1), (40, 83, 1000, 0)])
def test_gathered_leaves(trees, features, rows, chunks):
    """12 levels over widths at which a ring with leaf values would cost row warps: leaf values are gathered, by the kernel
    for 12 levels over narrow rows."""
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(8, trees, 12, features, 0.02, 0.1, marg)
    X = marg.sample_rows(np.random.Generator(np.random.PCG64(6)), rows)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(3 * rows, 600)):
        g = split[(i * 37) % len(split)]
        X[(i * 13) % rows, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    X[3, :], X[4, 0] = np.nan, np.inf
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows, tree_chunks=chunks)
    assert df.info().layout == kernels.LAYOUT_DEEP_KEYS
    dX = torch.from_numpy(X).cuda()
    got, part, ids = df.predict(dX), df.predict_partial(dX), df.predict_leaf_ids(dX)
    assert not _staged(df)
    df.predict(dX)
    assert not _staged(df)
    df.check_status()
    some = np.r_[0:min(rows, 3000), max(0, rows - 500):rows]
    want, want_ids = oracle.predict(f, X[some], leaf_ids=True)
    assert_predictions_close(got.cpu().numpy()[some], want)
    assert_predictions_close(df.finalize(part).cpu().numpy()[some], want)
    assert np.array_equal(ids.cpu().numpy()[some], want_ids)


@pytest.mark.parametrize("trees,features,rows,staged", [
    (80, 24, 90001, True), (80, 92, 60001, True), (60, 128, 40001, True), (66, 128, 80001, False), (80, 96, 80033, False),
    (80, 160, 50001, False), (300, 128, 2001, True), (1501, 128, 50001, False), (1501, 128, 100001, True)])
def test_twelve_levels(trees, features, rows, staged):
    """Leaf values of 12 levels are gathered where rows are wide and blocks walk many pairs, unless many trees meet a large
    batch; the last block has warps without rows."""
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(9, trees, 12, features, 0.02 if trees < 1000 else 0.12, 0.1, marg)
    X = np.tile(marg.sample_rows(np.random.Generator(np.random.PCG64(7)), 5003), (rows // 5003 + 1, 1))[:rows]
    split = np.nonzero(f.left >= 0)[0]
    some = np.r_[0:300, rows - 300:rows]
    for i, r in enumerate(np.repeat(some, 3)):
        g = split[(i * 37) % len(split)]
        X[r, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    X[3, :], X[4, 0] = np.nan, np.inf
    df = kernels.DeviceForest(f, representation="auto")
    assert df.info().layout == kernels.LAYOUT_DEEP_KEYS
    dX = torch.from_numpy(X).cuda()
    got = df.predict(dX)
    assert _staged(df) == staged
    part = df.predict_partial(dX)
    assert _staged(df) == staged
    ids = df.predict_leaf_ids(dX[-5000:]) if trees < 1000 else None
    df.check_status()
    want, want_ids = oracle.predict(f, X[some], leaf_ids=True)
    assert_predictions_close(got.cpu().numpy()[some], want)
    assert_predictions_close(df.finalize(part).cpu().numpy()[some], want)
    if ids is not None:
        assert np.array_equal(ids[-300:].cpu().numpy(), want_ids[-300:])


@pytest.mark.parametrize("features,twice", [(30, True), (600, False)])
def test_resident_bytes_count_both_orders_of_the_planes(features, twice):
    f = synth.generate_forest(2, 5, 10, features, 0.0, 0.1, synth.Marginal("normal", features))
    words = lambda levels: ((2 ** levels - 1) + (2 ** levels - 1) // 32 + (2 ** levels - 1) // 1024 + 4) // 4 * 4
    df = kernels.DeviceForest(f, representation="auto")
    df.predict(torch.zeros((100, features), device="cuda"))
    assert _staged(df) == twice
    assert df.info().packed_bytes == 6 * (8 * words(10) + (16 * words(9) if twice else 0))
