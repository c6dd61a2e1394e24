"""The count of row values that rank keys had to compare with thresholds (tbk_forest_info.reserved) is a property of the
batch: the kernel that ranks it makes no difference, nor do the rows and features that fill up a tile."""
import numpy as np
import pytest

from treebeard_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("trees,features,rows", [
    (40, 20, 3), (40, 20, 3001), (40, 20, 20001),       # inside the walk; pairs of rows, tables in global and in shared memory
    (40, 50, 3001), (40, 50, 20001),                    # row by row
    (40, 90, 501), (40, 90, 4001), (900, 90, 4001),     # tiles: tables in global memory, slabs, too many thresholds for slabs
    (60, 600, 101), (60, 600, 3001)])                   # one-byte keys
def test_compared_values_are_counted_alike(trees, features, rows):
    from treebeard_b200 import kernels
    f = synth.generate_forest(3, trees, 7 if trees > 100 else 5, features, 0.05, 0.1, synth.Marginal("normal", features), synth.IDENTITY, 0)
    split = f.left >= 0
    f.feat = np.where(split & (f.feat % 7 == 5), 0, f.feat).astype(f.feat.dtype)   # features without splits
    f.thr = np.where(split & (f.feat % 3 == 1), np.round(f.thr * 5), f.thr).astype(np.float32)
    X = np.random.default_rng(1).standard_normal((rows, features)).astype(np.float32) * 5
    X[:, ::2] = np.round(X[:, ::2])
    X[1, :], X[2, :5] = np.nan, np.inf
    compared = 0
    for i in range(features):
        thr = np.unique(f.thr[split & (f.feat == i)])
        if len(thr) == 0:
            continue
        lattice = bool((thr == np.floor(thr)).all())    # (these lie close together)
        compared += int((X[:, i] != np.floor(X[:, i])).sum()) if lattice else rows
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    assert df.info().layout == kernels.LAYOUT_RANK_KEYS
    for calls in (1, 2):
        df.predict(torch.from_numpy(X).cuda())
        df.check_status()
        info = df.info()
        assert info.reserved[0] + (info.reserved[1] << 31) == calls * compared
