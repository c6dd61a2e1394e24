"""The general walk's rows turned around in shared memory (large batches, one block per SM): widths
on both sides of a piece of 8 features, batches that end inside a warp's rows, tiles of every size,
strided and unaligned rows, one and two tree threads.  Leaf ids are exact, so a value in the wrong
place shows."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _forest(trees, levels, features):
    return synth.generate_forest(9, trees, levels, features, 0.02, 0.1, synth.Marginal("normal", features), synth.IDENTITY, 0)


@pytest.mark.parametrize("features", [8, 9, 15, 16, 17, 63, 90])
@pytest.mark.parametrize("layout,tile,trees", [("sparse", 1, 40), ("sparse", 2, 33), ("array", 1, 20), ("reorg", 1, 20), ("sparse", 4, 40), ("sparse", 3, 40)])
def test_widths(features, layout, tile, trees):
    from treebeard_b200 import kernels
    f = _forest(trees, 8, features)
    n = 148 * 32 * 8 + 33
    X = np.random.default_rng(features).standard_normal((n, features)).astype(np.float32)
    # (as many row warps as fit, one tree thread: the block takes more than half of the shared memory)
    df = kernels.DeviceForest(f, batch_hint=n, representation=layout, tile_size=tile, rows_per_block=1024, tree_threads=1)
    ids = df.predict_leaf_ids(torch.from_numpy(X).cuda()).cpu().numpy()
    some = np.r_[0:97, n - 97:n]
    _, want_ids = oracle.predict(f, X[some], leaf_ids=True)[:2]
    assert np.array_equal(ids[some], want_ids)
    # (nodes of tiles of three and four are read from global memory here: narrow rows leave a block too small)
    turned = tile <= 2 or features >= 63
    assert bool(df.info().reserved[2] & kernels.RAN_ROWS_TURNED) == turned
    got = df.predict(torch.from_numpy(X).cuda()).cpu().numpy()
    df.check_status()
    assert bool(df.info().reserved[2] & kernels.RAN_ROWS_TURNED) == turned
    assert_predictions_close(got, oracle.predict(f, X), f)


@pytest.mark.parametrize("threads", [1, 2])
@pytest.mark.parametrize("offset,stride", [(0, 61), (1, 61), (3, 64), (0, 58)])
def test_strides_and_tree_threads(threads, offset, stride):
    from treebeard_b200 import kernels
    features, n = 58, 7001
    f = _forest(50, 8, features)
    X = np.random.default_rng(3).standard_normal((n, features)).astype(np.float32)
    flat = torch.full((offset + n * stride,), float("nan"), device="cuda")
    rows = flat[offset:].view(n, stride)[:, :features]
    rows.copy_(torch.from_numpy(X))
    df = kernels.DeviceForest(f, batch_hint=n, representation="sparse", tile_size=2, rows_per_block=256, tree_threads=threads)
    ids = df.predict_leaf_ids(rows).cpu().numpy()
    df.check_status()
    assert df.info().reserved[2] & kernels.RAN_ROWS_TURNED
    assert np.array_equal(ids, oracle.predict(f, X, leaf_ids=True)[1])


@pytest.mark.parametrize("tile", [1, 2, 3])
def test_partial_sums_and_classes(tile):
    """Partial sums, and a multiclass forest whose sums stay in registers (predictions) or in shared memory (partial sums)."""
    from treebeard_b200 import kernels
    features, n = 30, 148 * 32 * 64 + 33
    f = synth.generate_forest(4, 34, 7, features, 0.02, 0.1, synth.Marginal("normal", features), synth.SOFTMAX, 3)
    X = np.random.default_rng(4).standard_normal((n, features)).astype(np.float32)
    dX = torch.from_numpy(X).cuda()
    some = np.r_[0:1100, n - 1100:n]
    want, sums = oracle.predict(f, X[some], class_sums=True)
    for options in (dict(), dict(rows_per_block=512, tree_threads=2)):
        df = kernels.DeviceForest(f, batch_hint=n, representation="sparse", tile_size=tile, **options)
        got = df.predict(dX).cpu().numpy()
        assert df.info().reserved[2] & kernels.RAN_ROWS_TURNED
        part = df.predict_partial(dX)
        assert df.info().reserved[2] & kernels.RAN_ROWS_TURNED
        df.check_status()
        assert_predictions_close(got[some], want, f, sums)
        assert_predictions_close(df.finalize(part).cpu().numpy()[some], want, f, sums)
    f = _forest(40, 8, features)
    df = kernels.DeviceForest(f, batch_hint=n, representation="sparse", tile_size=tile)
    part = df.predict_partial(dX)
    assert df.info().reserved[2] & kernels.RAN_ROWS_TURNED
    df.check_status()
    assert_predictions_close(df.finalize(part).cpu().numpy()[some], oracle.predict(f, X[some]))
