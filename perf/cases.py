"""The cases that the speed of this framework is judged by: forests and batches as its users
have them, each taken through the public entry points.

A case is a forest shape (trees, decision levels, features, the chance that a node ends early,
classes), a batch (rows, how the values are distributed) and the call that is made:

  "host"      TreebeardInferenceRunner.RunInference on a numpy batch (copies in and out included)
  "bulk"      TreebeardInferenceRunner.RunInferenceOnMultipleBatches on a numpy table
  "device"    TreebeardInferenceRunner.RunInference on a CUDA tensor
  "predict"   DeviceForest.predict on a CUDA tensor (stream-ordered)
  "shard"     DeviceForest.predict_partial + finalize: what a tree-sharded rank runs
  "leaf_ids"  DeviceForest.predict_leaf_ids: the leaf of every (row, tree)

``layout`` is "auto" (the library's choice, the default of a runner whose context names none) or
one of the representations that a user of the reference names, with its tile size.
"""
import math

import torch

from treebeard_b200 import kernels, synth
from treebeard_b200.treebeard import CompilerOptions, TreebeardInferenceRunner

_TRANSFORM = {"identity": synth.IDENTITY, "sigmoid": synth.SIGMOID, "softmax": synth.SOFTMAX}


def _case(call, rows, features, trees, levels, leaf_p=0.0, values="normal", transform="identity", classes=0,
          layout="auto", tile=1):
    return dict(call=call, rows=rows, features=features, trees=trees, levels=levels, leaf_p=leaf_p, values=values,
                transform=transform, classes=classes, layout=layout, tile=tile)


def listed():
    return [
        # one row scored while its requester waits: nothing but latency
        dict(name="one_row_request", **_case("host", 1, 28, 500, 6, 0.1, transform="sigmoid")),
        # the small regression configuration (100 complete trees of 6 levels) on its own batch,
        # in host memory as the reference's API takes it
        dict(name="regression_1k_host", **_case("host", 1024, 8, 100, 6, values="uniform01")),
        # the binary-classifier configuration at its smallest batch, rows already on the GPU
        dict(name="binary_4k", **_case("predict", 4096, 28, 1000, 8, 0.15, transform="sigmoid")),
        # the same forest at its largest batch
        dict(name="binary_1m", **_case("predict", 1048576, 28, 1000, 8, 0.15, transform="sigmoid")),
        # a table of the same kind scored from host memory in one call of the batch API
        dict(name="binary_bulk_host", **_case("bulk", 524288, 28, 1000, 8, 0.15, transform="sigmoid")),
        # an ordinary regression forest over more columns; ragged row and tree counts
        dict(name="regression_50k_90col", **_case("device", 50003, 90, 467, 7, 0.1)),
        # the wide dense regressor: rows of 8 KB, the streaming-bound configuration, full batch
        dict(name="wide_2000col", **_case("predict", 262144, 2000, 1000, 8)),
        # the 26-class configuration over small whole-number features, class ids out, full batch
        dict(name="multiclass_26", **_case("device", 1048576, 16, 2600, 8, 0.1, "int16", "softmax", 26)),
        # one rank's share of the large forest when eight ranks split its trees (a quarter of
        # its batch): partial sums, then the second pass
        dict(name="deep_tree_shard", **_case("shard", 1048576, 128, 2000, 12, 0.05, "mix")),
        # leaf indices as features of a second model
        dict(name="leaf_indices_20k", **_case("leaf_ids", 20011, 28, 1000, 8, 0.15)),
        # a runner whose user names the sparse representation and tiles of two nodes
        dict(name="sparse_tile2_100k", **_case("device", 100000, 54, 300, 8, 0.1, layout="gpu_sparse", tile=2)),
        # trees grown until their leaves are pure, a few hundred of them: deeper than the
        # whole-tree stages reach
        dict(name="pure_leaves_64k", **_case("predict", 65536, 32, 200, 16, 0.25)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["narrow", "narrow", "host", "host", "wide", "multiclass", "deep", "named", "pure", "leaves"])
    p = rng.choice([0.0, 0.1, 0.15])
    transform = rng.choice(["identity", "sigmoid"])
    values = rng.choice(["normal", "uniform01", "mix", "normal"])
    if family == "narrow":
        return _case(rng.choice(["predict", "device"]), _log(rng, 256, 1048576), _log(rng, 4, 400), _log(rng, 30, 1000),
                     rng.randint(4, 8), p, values, transform)
    if family == "host":
        return _case(rng.choice(["host", "host", "bulk"]), _log(rng, 1, 524288), _log(rng, 4, 128), _log(rng, 30, 1000),
                     rng.randint(4, 8), p, values, transform)
    if family == "wide":
        return _case(rng.choice(["predict", "device"]), _log(rng, 1024, 131072), _log(rng, 500, 2000), _log(rng, 100, 1000),
                     rng.randint(6, 8), p, values, transform)
    if family == "multiclass":
        classes = rng.randint(3, 26)
        return _case(rng.choice(["predict", "device"]), _log(rng, 512, 524288), _log(rng, 6, 64),
                     classes * _log(rng, 10, 100), rng.randint(4, 8), p, rng.choice(["int16", "normal"]), "softmax", classes)
    if family == "deep":
        return _case(rng.choice(["predict", "shard"]), _log(rng, 1024, 262144), _log(rng, 16, 200), _log(rng, 50, 1000),
                     rng.randint(9, 12), 0.05, values, transform)
    if family == "named":
        layout = rng.choice(["gpu_sparse", "gpu_array", "gpu_reorg"])
        return _case("device", _log(rng, 1024, 131072), _log(rng, 4, 128), _log(rng, 50, 500), rng.randint(4, 8), 0.1, values,
                     transform, layout=layout, tile=1 if layout == "gpu_reorg" else rng.randint(1, 4))
    if family == "pure":
        return _case("predict", _log(rng, 1024, 131072), _log(rng, 8, 64), _log(rng, 20, 200), rng.randint(13, 16), 0.25, values,
                     transform)
    return _case("leaf_ids", _log(rng, 256, 32768), _log(rng, 4, 128), _log(rng, 30, 1000), rng.randint(4, 8), p, values)


def _rows(case, marginal, seed):
    """The batch as a CUDA tensor, with the distributions of synth.Marginal."""
    n, F = case["rows"], case["features"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["values"] == "uniform01":
        return torch.rand((n, F), generator=gen, device="cuda")
    if case["values"] == "int16":
        return torch.randint(0, 16, (n, F), generator=gen, device="cuda").to(torch.float32)
    x = torch.randn((n, F), generator=gen, device="cuda")
    if case["values"] == "mix":
        cols = torch.from_numpy(marginal.uniform_cols).cuda()
        x[:, cols] = torch.rand((n, int(cols.sum())), generator=gen, device="cuda") * 10.0 - 5.0
    return x


def prepare(case, seed):
    """A packed forest (or a runner) and a batch for it, both drawn from the seed."""
    marginal = synth.Marginal(case["values"], case["features"], seed=seed)
    forest = synth.generate_forest(seed, case["trees"], case["levels"], case["features"], case["leaf_p"], 0.05, marginal,
                                   _TRANSFORM[case["transform"]], case["classes"])
    rows = _rows(case, marginal, seed + 1)
    state = dict(call=case["call"], int8=case["classes"] > 0)
    if case["call"] in ("host", "bulk", "device"):
        # a bulk call goes through a runner for batches of a quarter of the table
        batch = max(1, case["rows"] // 4) if case["call"] == "bulk" else case["rows"]
        opts = CompilerOptions(batch, case["tile"])
        if state["int8"]:
            opts.SetReturnTypeWidth(8)
            opts.SetReturnTypeIsFloatType(False)
        layout = "gpu_auto" if case["layout"] == "auto" else case["layout"]
        state["runner"] = TreebeardInferenceRunner.FromForestArrays(forest, opts, representation=layout)
        if case["call"] == "bulk":
            rows = rows[:batch * (case["rows"] // batch)]
        state["rows"] = rows if case["call"] == "device" else rows.cpu().numpy()
    else:
        state["forest"] = kernels.DeviceForest(forest, device=0, batch_hint=case["rows"], representation=case["layout"],
                                               tile_size=case["tile"])
        state["rows"] = rows
    return state


def run(state):
    call = state["call"]
    if call == "predict":
        return state["forest"].predict(state["rows"], int8=state["int8"])
    if call in ("host", "device"):
        # (the result type of a runner that returns class ids is stated for numpy batches only)
        return state["runner"].RunInference(state["rows"])
    if call == "bulk":
        return state["runner"].RunInferenceOnMultipleBatches(state["rows"])
    if call == "shard":
        partial = state["forest"].predict_partial(state["rows"])
        return partial, state["forest"].finalize(partial)
    return state["forest"].predict_leaf_ids(state["rows"])


def work(case):
    """Every row value read once, every result written once, the forest (a threshold and a
    feature index per split, a value per leaf) read once; a comparison per decision on a row's
    path through a tree and an addition per tree."""
    n, T, D, keep = case["rows"], case["trees"], case["levels"], 1.0 - case["leaf_p"]
    splits = 1.0 + sum(2 ** d * keep ** d for d in range(1, D))        # per tree (the root never ends early)
    path = sum(keep ** d for d in range(D))                            # decisions from root to leaf
    out = {"shard": 8, "leaf_ids": 4 * T}.get(case["call"], 1 if case["classes"] else 4)
    return {"bytes": n * (4 * case["features"] + out) + T * (splits * 6 + (splits + 1) * 4), "flops": n * T * (path + 1)}


def tolerance(case):
    if case["call"] == "leaf_ids":
        return "exact"                       # node ids
    if case["classes"]:
        return {"rel": 0.0, "differ": 5e-4}  # the best of several fp32 class sums: near-ties may fall either way
    # fp32 sums in another order; the sum of a single row may cancel, that of a batch does not
    return {"rel": 1e-5, "max": 1e-4} if case["rows"] >= 64 else {"rel": 5e-5, "max": 1e-4}
