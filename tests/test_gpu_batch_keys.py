"""Rounded keys over rows narrow enough to be staged several tiles at a time: what the library lays out
so by itself is multiclass forests over more than 64 features, and features with more distinct
thresholds than ranks reach."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# (complete trees of 8 or 6 levels have kernels of their own; 100 features: many tiles to a batch, 320: four)
@pytest.mark.parametrize("trees,levels,features,classes,p,rows", [
    (33, 8, 65, 2, 0.0, 1), (70, 8, 100, 3, 0.0, 40003), (21, 6, 320, 7, 0.2, 5000), (60, 5, 200, 5, 0.2, 77),
    (64, 6, 128, 4, 0.0, 148 * 32 * 3 + 1), (300, 8, 1, 0, 0.0, 6001), (1100, 6, 1, 0, 0.0, 999), (1000, 7, 1, 0, 0.1, 2500),
    (700, 8, 2, 0, 0.0, 33)])
def test_batches_of_rounded_key_tiles_are_exact(trees, levels, features, classes, p, rows):
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(8, trees, levels, features, p, 0.1, marg, num_classes=classes)
    X = marg.sample_rows(np.random.Generator(np.random.PCG64(9)), rows)
    split = np.nonzero(f.left >= 0)[0]
    for i in range(min(600, 2 * rows)):   # values equal to thresholds, and their neighbours
        g = split[(i * 37) % len(split)]
        X[(i * 13) % rows, f.feat[g]] = np.nextafter(f.thr[g], np.float32([-np.inf, np.inf, f.thr[g]][i % 3]))
    if rows > 6:
        X[3, :], X[4, 0], X[5, features - 1] = np.nan, np.inf, -np.inf
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    dX = torch.from_numpy(X).cuda()
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
    got, part = df.predict(dX), df.predict_partial(dX)
    df.check_status()
    info = df.info()
    assert info.layout == kernels.LAYOUT_ROUNDED_KEYS and info.threads_per_block == 704
    assert info.reserved[0] > 0   # key ties were hit and resolved exactly
    if classes:
        _, sums = oracle.predict(f, X, class_sums=True)
        assert_predictions_close(got.cpu().numpy(), want, f, sums)
        assert np.allclose(part.cpu().numpy() + f.initial_value, sums, rtol=1e-5, atol=1e-5)
        assert np.array_equal(df.predict(dX, int8=True).cpu().numpy(), got.cpu().numpy().astype(np.int8))
    else:
        assert_predictions_close(got.cpu().numpy(), want)
        assert_predictions_close(df.finalize(part).cpu().numpy(), want)
