"""Deep-tree forests that L2 does not hold: walked in ranges of their trees, the rows' sums carried over in
64 bits."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _chains(trees, levels, features, seed=3):
    """Trees that are one path of `levels` decisions: few nodes, whole planes once they are laid out."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, d = 2 * levels + 1, np.arange(levels)
    right = rng.integers(0, 2, (trees, levels)).astype(bool)   # the side on which the path goes on
    left_of, right_of = np.full((trees, n), -1, np.int32), np.full((trees, n), -1, np.int32)
    on, off = 2 * d + 1, 2 * d + 2   # node 0 is the root; the path goes on at 1, 3, 5, ...
    path = np.concatenate([[0], on[:-1]])
    left_of[:, path] = np.where(right, off, on)
    right_of[:, path] = np.where(right, on, off)
    thr = (rng.standard_normal((trees, n)) * 0.05).astype(np.float32)
    thr[:, path] = rng.standard_normal((trees, levels)) * 0.3 + np.where(right, -1.0, 1.0)
    feat = np.zeros((trees, n), np.int32)
    feat[:, path] = rng.integers(0, features, (trees, levels))
    return synth.ForestArrays(np.arange(trees + 1, dtype=np.int64) * n, left_of.ravel(), right_of.ravel(), feat.ravel(),
                              thr.ravel(), np.zeros(trees, np.int32), 0, synth.IDENTITY, 0.25, features)


@pytest.mark.parametrize("trees,rows", [(7001, 300001), (12500, 400000)])
def test_ranges_of_a_forest_larger_than_l2(trees, rows):
    f = _chains(trees, 12, 12)
    X = np.random.Generator(np.random.PCG64(5)).standard_normal((rows, 12)).astype(np.float32)
    X[7, 3], X[rows - 1, 0] = np.nan, np.inf
    split = np.nonzero(f.left >= 0)[0]
    for i in range(2000):   # values equal to thresholds: trees behind a key tie
        g = split[(i * 977) % len(split)]
        X[(i * 151) % rows, f.feat[g]] = f.thr[g]
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    assert df.info().layout == kernels.LAYOUT_DEEP_KEYS and df.info().packed_bytes > 1.5 * l2
    dX = torch.from_numpy(X).cuda()
    before = df.launch_count()
    got = df.predict(dX)
    assert df.launch_count() - before >= round(df.info().packed_bytes / l2)
    df.check_status()
    again = df.finalize(df.predict_partial(dX))
    whole = kernels.DeviceForest(f, representation="auto", batch_hint=rows, tree_chunks=2)
    assert torch.allclose(got, whole.predict(dX), rtol=1e-5, atol=1e-6, equal_nan=True)
    for first in (0, rows // 2, rows - 1500):
        part = slice(first, first + 1500)
        want, want_ids = oracle.predict(f, X[part], leaf_ids=True)
        assert_predictions_close(got[part].cpu().numpy(), want)
        assert_predictions_close(again[part].cpu().numpy(), want)
        assert np.array_equal(df.predict_leaf_ids(dX[part]).cpu().numpy(), want_ids)
    df.check_status()


def test_leaf_ids_and_captured_calls_in_ranges():
    f = _chains(6100, 12, 4)
    rows = 2 * 148 * 30 * 32 + 1
    X = torch.randn((rows, 4), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows)
    want = df.predict(X).clone()
    out = torch.empty_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        df.predict(X, out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    ids = df.predict_leaf_ids(X)
    df.check_status()
    sample = slice(rows - 1000, rows)
    assert np.array_equal(ids[sample].cpu().numpy(), oracle.predict(f, X[sample].cpu().numpy(), leaf_ids=True)[1])
