"""Forests of every layout and the streams that calls come on: what creation has uploaded is there
for a stream that nothing orders behind it, and calls that may run at the same time have memory of
their own."""
import ctypes
import threading

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
    "rank_bytes": (48, 8, 700, 0, {}),   # (where batches are announced)
    "rounded_wide": (48, 8, 700, 0, dict(feature_bits=16)),
    "rounded_classes": (48, 6, 100, 3, {}),
    "deep": (24, 11, 40, 0, {}),
    "lanes": (50, 14, 16, 0, {}),
    "tiles": (300, 8, 28, 0, dict(representation="sparse", tree_chunks=3)),
}

EXPECTED = {"rank": kernels.LAYOUT_RANK_KEYS, "rank_tiles": kernels.LAYOUT_RANK_KEYS, "rank_classes": kernels.LAYOUT_RANK_KEYS,
            "rank_bytes": kernels.LAYOUT_RANK_KEYS, "rounded_wide": kernels.LAYOUT_ROUNDED_KEYS, "rounded_classes": kernels.LAYOUT_ROUNDED_KEYS,
            "deep": kernels.LAYOUT_DEEP_KEYS, "lanes": kernels.LAYOUT_LANES, "tiles": kernels.LAYOUT_TILES}

SINGLE = [name for name, shape in LAYOUTS.items() if not shape[3]]


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
        assert df.info().layout == EXPECTED[layout]
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


def _predict_on(df, rows, out, stream_handle):
    kernels._check(kernels.lib().tbk_predict(df._h, rows.data_ptr(), rows.shape[0], rows.stride(0), out.data_ptr(),
                                             kernels.OUT_F32, stream_handle))


PER_THREAD = 2   # cudaStreamPerThread: one handle, another stream in every thread


@pytest.mark.parametrize("layout", SINGLE)
def test_per_thread_streams_do_not_share_call_memory(layout):
    f, X, options = _case(layout, 24000)
    dX = torch.from_numpy(X).cuda()
    parts = [dX[i * 6000:(i + 1) * 6000] for i in range(4)]
    df = kernels.DeviceForest(f, batch_hint=6000, **options)
    assert df.info().layout == EXPECTED[layout]
    want = [df.predict(p).clone() for p in parts]
    outs = [torch.empty_like(w) for w in want]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(len(parts))

    def work(i):
        mine = torch.cuda.ExternalStream(PER_THREAD)
        for _ in range(200):
            start.wait()
            _predict_on(df, parts[i], outs[i], PER_THREAD)
            mine.synchronize()
            if not torch.equal(outs[i].cpu(), want[i].cpu()):
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(parts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    df.check_status()


@pytest.mark.parametrize("layout", SINGLE)
@pytest.mark.parametrize("alive", [1, 3, 11])
def test_streams_that_come_and_go(layout, alive):
    """Streams are destroyed with a prediction pending and new ones, often under the same handle, take
    their place; `alive` of them at a time (more than the forest has workspaces for, at eleven)."""
    f, X, options = _case(layout, 40000)
    dX = torch.from_numpy(X).cuda()
    df = kernels.DeviceForest(f, batch_hint=5000, **options)
    assert df.info().layout == EXPECTED[layout]
    sizes = [5000 + 307 * i for i in range(12)]
    batches = [dX[1000 * i:1000 * i + n] for i, n in enumerate(sizes)]
    want = [df.predict(b).clone() for b in batches]
    torch.cuda.synchronize()
    rt, handles, outs = torch.cuda.cudart(), [], []
    for i in range(60):
        handle = ctypes.c_void_p()
        assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
        out = torch.empty(sizes[i % 12], device="cuda")
        torch.cuda.current_stream().synchronize()
        _predict_on(df, batches[i % 12], out, handle.value)
        outs.append(out)
        handles.append(handle.value)
        if len(handles) == alive:
            assert int(rt.cudaStreamDestroy(handles.pop(0))) == 0
    for h in handles:
        assert int(rt.cudaStreamDestroy(h)) == 0
    torch.cuda.synchronize()
    df.check_status()
    for i, out in enumerate(outs):
        assert torch.equal(out, want[i % 12]), i


def _captured(df, rows, out):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        df.predict(rows, out=out)
    return graph


@pytest.mark.parametrize("layout", SINGLE)
def test_memory_of_captured_calls_lives_as_long_as_their_graphs(layout):
    f, X, options = _case(layout, 60000)
    dX = torch.from_numpy(X).cuda()
    df = kernels.DeviceForest(f, batch_hint=60000 if layout == "rank_bytes" else 0, **options)
    assert df.info().layout == EXPECTED[layout]
    sizes = [60000 - 1000 * i for i in range(24)]
    want = [df.predict(dX[:n]).clone() for n in sizes]
    outs = [torch.empty(n, device="cuda") for n in sizes]
    torch.cuda.synchronize()
    # two graphs at a time: replayed side by side, each with its own memory
    side = torch.cuda.Stream()
    for i in (0, 1):
        graphs = [_captured(df, dX[:sizes[j]], outs[j]) for j in (i, i + 2)]
        for _ in range(20):
            for g, s in zip(graphs, (side, torch.cuda.Stream())):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
        for j in (i, i + 2):
            assert torch.equal(outs[j], want[j])
        del graphs, g
    # one after another, a new shape each: the memory of those that are gone serves the next
    free = []
    for k in range(48):
        n, out = sizes[k % 24], outs[k % 24]
        out.zero_()
        graph = _captured(df, dX[:n], out)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[k % 24])
        del graph
        free.append(torch.cuda.mem_get_info()[0])
    keys = {"rank": 4, "rank_tiles": 16, "rank_bytes": 64}.get(layout, 1) << 20   # the most that one call takes, to a power of two
    assert min(free[8:]) >= free[0] - 8 * keys
    assert torch.equal(df.predict(dX[:sizes[0]]), want[0])
    df.check_status()


def test_forests_of_one_kernel_and_different_sizes_in_two_threads():
    """The same kernels, launched by two threads with different amounts of shared memory."""
    forests = []
    for layout, rows, features in (("tiles", 64, 28), ("tiles", 64, 90), ("rounded_wide", 64, 700), ("rounded_wide", 64, 1500),
                                   ("deep", 64, 20), ("deep", 64, 60)):
        trees, levels, _, _, options = LAYOUTS[layout]
        marg = synth.Marginal("normal", features)
        f = synth.generate_forest(features, 16, levels, features, 0.1, 0.1, marg)
        X = torch.from_numpy(marg.sample_rows(np.random.Generator(np.random.PCG64(1)), rows)).cuda()
        df = kernels.DeviceForest(f, **dict(dict(representation="auto"), **options))
        assert df.info().layout == EXPECTED[layout]
        forests.append((df, X, df.predict(X).clone()))
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(2)

    def work(mine):
        stream = torch.cuda.Stream()
        outs = [torch.zeros_like(want) for _, _, want in mine]
        torch.cuda.synchronize()
        start.wait()
        try:
            for i in range(9000):
                df, X, _ = mine[i % len(mine)]
                _predict_on(df, X, outs[i % len(mine)], stream.cuda_stream)
        except kernels.TbkError as e:
            wrong.append(str(e))
        stream.synchronize()
        wrong.extend("values" for out, (_, _, want) in zip(outs, mine) if not torch.equal(out, want))

    threads = [threading.Thread(target=work, args=(forests[i::2],)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[0]
