"""Packed images whose sections fit each other and whose checksum is right, but which no packer of this library makes: they
are refused when they are read, before a kernel could be launched over them.  Host only."""
import struct

import pytest

from treebeard_b200 import kernels, synth

MASK, PRIME, SEED = (1 << 64) - 1, 1099511628211, 14695981039346656037


def _fnv(h, data):
    for b in data:
        h = (h ^ b) * PRIME & MASK
    return h


def _checksum(data):
    """csrc/checksum.h"""
    if len(data) < 4096:
        return _fnv(SEED, data)
    h = SEED
    for at in range(0, len(data), 1 << 20):
        block = data[at:at + (1 << 20)]
        lanes = [SEED, SEED ^ 0x9e3779b97f4a7c15, SEED ^ 0xc2b2ae3d27d4eb4f, SEED ^ 0x165667b19e3779f9]
        whole = len(block) // 32 * 32
        for i, w in enumerate(struct.unpack(f"<{whole // 8}Q", block[:whole])):
            lanes[i % 4] = (lanes[i % 4] ^ w) * 0x9e3779b97f4a7c15 & MASK
        part = SEED
        for lane in lanes:
            part = (part ^ lane ^ lane >> 29) * PRIME & MASK
        h = (h ^ _fnv(part, block[whole:])) * PRIME & MASK
    return h


HEAD = 8 + 4 + 4 * 4 + 4 + 12 * 4 + 2 * 4   # magic, version, kind and request, limit, schedule, deep shape
FOREST = HEAD + 4 + 4 + 8 + 8 + 8 + 4       # features, transform, initial value, trees, nodes, levels


def _signed(body):
    return bytes(body) + struct.pack("<Q", _checksum(bytes(body)))


def _image(trees, levels, features):
    forest = synth.generate_forest(3, trees, levels, features, 0.0, 0.1, synth.Marginal("normal", features), synth.IDENTITY, 0)
    data = bytearray(kernels.PackedImage.pack(forest, representation="auto").to_bytes())
    assert _signed(data[:-8]) == bytes(data) and struct.unpack_from("<i", data, HEAD)[0] == features
    return data[:-8]


def _rank_image(features, levels):
    """An image over `features` columns, of which the trees use the first 100."""
    body = _image(3, 2, 100)
    at = FOREST + 3 * 4                                        # classes, lattice, comparison
    for element in (16, 4, 4, 4, 4, 4):                        # groups, three planes, trees, classes
        at += 8 + element * struct.unpack_from("<Q", body, at)[0]
    assert struct.unpack_from("<Q", body, at)[0] == 100
    last = body[at + 8 + 99 * 32:at + 8 + 100 * 32]
    body[at + 8 + 100 * 32:at + 8 + 100 * 32] = last * (features - 100)
    struct.pack_into("<Q", body, at, features)
    struct.pack_into("<i", body, HEAD, features)
    struct.pack_into("<i", body, FOREST - 4, levels)
    return _signed(body)


@pytest.mark.parametrize("features,levels,fits", [
    (100, 8, True), (511, 8, True), (512, 8, True), (2024, 8, True), (2025, 8, False), (2040, 8, False), (2044, 8, False),
    (2044, 7, True), (2045, 7, False)])
def test_rank_images_without_a_launch_shape(features, levels, fits):
    data = _rank_image(features, levels)
    if fits:
        assert kernels.PackedImage.from_bytes(data).to_bytes() == data
    else:
        with pytest.raises(kernels.TbkError):
            kernels.PackedImage.from_bytes(data)


def _deep_image(pairs, levels):
    """An image whose table of pairs is `pairs` (elements, levels each; None: as packed) and whose forest has `levels` levels."""
    body = _image(5, 9, 30)
    at, n = FOREST + 8, struct.unpack_from("<Q", body, FOREST)[0]
    table = [struct.unpack_from("<QII", body, at + 16 * i) for i in range(n)]
    assert [t[1] for t in table] == [9] * n == [9] * 3
    for i, elements in enumerate(pairs or []):
        struct.pack_into("<Q", body, at + 16 * i, elements * 2 * table[0][2])
    struct.pack_into("<i", body, FOREST - 4, levels)
    return _signed(body)


@pytest.mark.parametrize("pairs,levels,whole", [(None, 9, True), ([0, 1, 2], 9, True), ([0, 0, 0], 9, False), ([1, 0, 2], 9, False),
                                                ([0, 1, 1], 9, False), (None, 12, False), (None, 8, False), (None, -1, False)])
def test_deep_images_whose_pairs_do_not_lie_one_behind_the_other(pairs, levels, whole):
    """The re-ordering of a forest's planes and the kernels for one depth count on it."""
    data = _deep_image(pairs, levels)
    if whole:
        assert kernels.PackedImage.from_bytes(data).to_bytes() == data
    else:
        with pytest.raises(kernels.TbkError):
            kernels.PackedImage.from_bytes(data)


def test_deep_images_without_all_their_planes():
    """Two of three pairs' planes, their sizes alike."""
    body = _image(5, 9, 30)
    at = FOREST + 8 + 16 * 3
    for _ in range(4):                                          # nodes, leaves, exact thresholds, original leaves
        n = struct.unpack_from("<Q", body, at)[0]
        keep = n // 3 * 2
        struct.pack_into("<Q", body, at, keep)
        del body[at + 8 + 4 * keep:at + 8 + 4 * n]
        at += 8 + 4 * keep
    with pytest.raises(kernels.TbkError):
        kernels.PackedImage.from_bytes(_signed(body))
