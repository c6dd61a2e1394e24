"""Deep trees whose rows meet thresholds exactly: a few key ties per row (walked after all other
trees), more than a thread remembers, and trees numbered beyond what it can remember."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("trees,levels,features,rows,leaf_p,chunks,meet", [
    (1, 9, 3, 1, 0.1, 0, 1.0), (65, 12, 128, 700, 0.05, 1, 0.02), (65, 12, 128, 700, 0.05, 1, 1.0),
    (40, 10, 600, 100, 0.1, 3, 0.3), (70000, 9, 20, 40, 0.7, 1, 0.5)])
def test_rows_on_thresholds(trees, levels, features, rows, leaf_p, chunks, meet):
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(3, trees, levels, features, leaf_p, 0.1, marg)
    rng = np.random.Generator(np.random.PCG64(5))
    X = marg.sample_rows(rng, rows)
    split = np.nonzero(f.left >= 0)[0]
    for g in rng.choice(split, int(meet * rows * features) + 1):
        X[rng.integers(rows), f.feat[g]] = f.thr[g]
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows, tree_chunks=chunks)
    assert df.info().schedule.feature_bits == 16
    dX = torch.from_numpy(X).cuda()
    assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
    got, part = df.predict(dX), df.predict_partial(dX)
    df.check_status()
    assert_predictions_close(got.cpu().numpy(), want)
    assert_predictions_close(df.finalize(part).cpu().numpy(), want)


@pytest.mark.parametrize("trees,rows", [(8, 500), (24, 500), (60, 300), (400, 100)])
def test_more_ties_than_a_thread_keeps_at_hand(trees, rows):
    """Thresholds and row values from one coarse set of numbers that is no lattice: about one comparison in ten
    ties, from a few trees per row to far more than can be put off."""
    marg = synth.Marginal("normal", 16)
    f = synth.generate_forest(4, trees, 11, 16, 0.05, 0.1, marg)
    rng = np.random.Generator(np.random.PCG64(6))
    X = marg.sample_rows(rng, rows)
    split = f.left >= 0
    f.thr[split] = (np.round(f.thr[split] / 0.37) * 0.37).astype(np.float32)
    X = (np.round(X / 0.37) * 0.37).astype(np.float32)
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    df = kernels.DeviceForest(f, representation="auto", batch_hint=rows, tree_chunks=1)
    assert df.info().layout == kernels.LAYOUT_DEEP_KEYS
    dX = torch.from_numpy(X).cuda()
    before = df.info().reserved[0]
    got = df.predict(dX)
    assert df.info().reserved[0] - before > rows * min(3, trees // 8)
    part = df.predict_partial(dX)
    assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy(), want_ids)
    df.check_status()
    assert_predictions_close(got.cpu().numpy(), want)
    assert_predictions_close(df.finalize(part).cpu().numpy(), want)
