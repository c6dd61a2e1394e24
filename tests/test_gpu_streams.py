"""Forests of every layout and the streams that calls come on: what creation has uploaded is there
for a stream that nothing orders behind it."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import kernels, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# layout: trees, levels, features, classes, creation options
LAYOUTS = {
    "rank": (200, 8, 28, 0, {}),
    "rank_tiles": (100, 7, 90, 0, {}),
    "rank_classes": (60, 6, 16, 5, {}),
    "rounded_wide": (48, 8, 700, 0, {}),
    "rounded_classes": (48, 6, 100, 3, {}),
    "deep": (24, 11, 40, 0, {}),
    "lanes": (50, 14, 16, 0, {}),
    "tiles": (300, 8, 28, 0, dict(representation="sparse", tree_chunks=3)),
}


def _case(layout, rows, seed=5):
    trees, levels, features, classes, options = LAYOUTS[layout]
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(seed, trees, levels, features, 0.1, 0.1, marg, num_classes=classes)
    X = marg.sample_rows(np.random.Generator(np.random.PCG64(seed + 1)), rows)
    return f, X, dict(dict(representation="auto"), **options)


@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_a_new_forest_is_ready_for_every_stream(layout):
    """Creation leaves no copy and no memset of its own running, and a call on a non-blocking stream
    right behind it (leaf ids first: the general layout uploads their table then) is right."""
    f, X, options = _case(layout, 3000)
    want, want_ids = oracle.predict(f, X, leaf_ids=True)
    dX = torch.from_numpy(X).cuda()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        df = kernels.DeviceForest(f, batch_hint=len(X), **options)
        assert torch.cuda.default_stream().query()
        with torch.cuda.stream(side):
            ids, got = df.predict_leaf_ids(dX), df.predict(dX)
        side.synchronize()
        df.check_status()
        assert np.array_equal(ids.cpu().numpy(), want_ids)
        if f.num_classes:
            _, sums = oracle.predict(f, X, class_sums=True)
            assert_predictions_close(got.cpu().numpy(), want, f, sums)
        else:
            assert_predictions_close(got.cpu().numpy(), want)
        df.close()
