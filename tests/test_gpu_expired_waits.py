"""Bounded waits that run out, one case per kernel that has them: the first bulk copy of a launch is never issued (the
host's doing), the kernel gives up, waits for the copies that it did start and ends by itself; the status says so, and the
next call is correct."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import assert_predictions_close
from treebeard_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = {
    # name: trees, levels, features, classes, rows, ids, options, layout
    "fp32 tiles, two stages": (60, 5, 12, 0, 3000, False, dict(representation="sparse"), "TILES"),
    "fp32 tiles, one stage, rows turned around": (60, 8, 54, 0, 40000, False, dict(representation="sparse", tile_size=2), "TILES"),
    "rounded keys, wide rows": (70, 6, 600, 0, 500, False, dict(representation="auto", feature_bits=16), "ROUNDED_KEYS"),
    "rounded keys, wide rows, several tiles per block": (70, 8, 600, 0, 9601, False, dict(representation="auto", feature_bits=16), "ROUNDED_KEYS"),
    "rounded keys, batches of tiles": (200, 6, 100, 3, 3000, False, dict(representation="auto"), "ROUNDED_KEYS"),
    "rank keys": (100, 6, 20, 0, 70000, False, dict(representation="auto"), "RANK_KEYS"),
    "rank keys, leaf ids": (100, 6, 40, 0, 500, True, dict(representation="auto"), "RANK_KEYS"),
    "rank keys in tiles": (100, 6, 90, 0, 500, False, dict(representation="auto"), "RANK_KEYS"),
    "rank keys in tiles, leaf ids": (100, 6, 90, 0, 500, True, dict(representation="auto"), "RANK_KEYS"),
    "ranking in slabs": (100, 6, 90, 0, 4000, False, dict(representation="auto"), "RANK_KEYS"),
    "ranking in slabs, several passes, one-byte keys": (60, 6, 2000, 0, 48000, False, dict(representation="auto"), "RANK_KEYS"),
    "one-byte rank keys, pairs of tiles": (100, 8, 2000, 0, 70, False, dict(representation="auto"), "RANK_KEYS"),
    "deep trees, leaf values staged": (40, 11, 60, 0, 3000, False, dict(representation="auto"), "DEEP_KEYS"),
    "deep trees, leaf ids": (40, 11, 60, 0, 3000, True, dict(representation="auto"), "DEEP_KEYS"),
    "deep trees, many features": (20, 10, 600, 0, 500, False, dict(representation="auto"), "DEEP_KEYS"),
}


@pytest.mark.parametrize("name", CASES)
def test_a_wait_that_runs_out_ends_the_launch(name):
    from treebeard_b200 import kernels
    trees, levels, features, classes, rows, ids, options, layout = CASES[name]
    marg = synth.Marginal("normal", features)
    f = synth.generate_forest(5, trees, levels, features, 0.02, 0.1, marg, synth.SOFTMAX if classes else synth.IDENTITY, classes)
    X = marg.sample_rows(np.random.Generator(np.random.PCG64(2)), rows)
    dX = torch.from_numpy(X).cuda()
    df = kernels.DeviceForest(f, batch_hint=rows, **options)
    assert df.info().layout == getattr(kernels, "LAYOUT_" + layout)
    some = slice(0, 2000)
    want, want_ids = oracle.predict(f, X[some], leaf_ids=True)
    sums = oracle.predict(f, X[some], class_sums=True)[1] if classes else None

    def right():
        if ids:
            assert np.array_equal(df.predict_leaf_ids(dX).cpu().numpy()[some], want_ids)
        else:
            assert_predictions_close(df.predict(dX).cpu().numpy()[some], want, f, sums)
        df.check_status()

    right()
    df.expire_next_wait()
    df.predict_leaf_ids(dX) if ids else df.predict(dX)   # undefined results
    torch.cuda.synchronize()
    with pytest.raises(kernels.TbkError) as err:
        df.check_status()
    assert err.value.status == 4
    assert ("ranking kernel" if "slabs" in name else "walk kernel") in str(err.value)
    right()
