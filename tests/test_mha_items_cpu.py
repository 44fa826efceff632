"""The division of the INT8 attention's work into items (csrc/mha_items.h, plain C++) against a model of its launch."""
import ctypes
import random
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tensorrt_b200" / "csrc"
CTAS, TILE, UNKNOWN = 148, 128, 2 ** 63 - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("items")
    (d / "items.cpp").write_text('#include "mha_items.h"\n'
                                 'extern "C" void plan(int32_t B, int32_t N, int32_t S, int64_t missing, int64_t ctas, int32_t* out)'
                                 "{ auto p = b200::planItems(B, N, S, missing, ctas); out[0] = p.tilesPerItem; out[1] = p.chunks; out[2] = p.longestFirst; }\n"
                                 'extern "C" int64_t cut(int32_t B, int32_t N, int32_t S, int64_t tokens, int64_t ctas) { return b200::cutTiles(B, N, S, tokens, ctas); }\n'
                                 'extern "C" int32_t item(int32_t round, int32_t cta, int32_t ctas) { return b200::itemOfRound(round, cta, ctas); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "items.cpp"), "-o", str(d / "items.so")], check=True)
    so = ctypes.CDLL(str(d / "items.so"))
    so.cut.restype = ctypes.c_int64
    return so


def _plan(lib, b, heads, s, missing):
    out = (ctypes.c_int32 * 3)()
    lib.plan(b, heads, s, ctypes.c_int64(missing), ctypes.c_int64(CTAS), out)
    return out[0], out[1], bool(out[2])


def _time(lengths, s, heads, tiles, chunks, padded, item=None):
    """Longest list of a CTA: a tile costs three units per key block, an item one more for the wait for its keys and values."""
    items = len(lengths) * heads * chunks
    ctas = min(CTAS, items)
    if item:
        lengths = sorted(lengths, reverse=True)
    longest = 0
    for cta in range(ctas):
        load = 0
        for r in range(-(-items // ctas)):
            i = item(r, cta, ctas) if item else r * ctas + cta
            if i >= items:
                continue
            pair, c = divmod(i, chunks)
            blocks = -(-lengths[pair // heads] // TILE)
            t = min(-(-s // TILE) if padded else blocks, (c + 1) * tiles) - c * tiles
            load += (3 * t + 1) * blocks if t > 0 else 0
        longest = max(longest, load)
    return longest


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("heads", [12, 16])
def test_ragged_batches_are_not_slower_than_whole_pairs_as_they_come(lib, heads, padded):
    """Packed or padded batches whose lengths the host does not know: hardly ever is a CTA's list longer, and often shorter."""
    rng = random.Random(heads + padded)
    ratio = []
    for _ in range(1500):
        s, b = rng.randint(1, 512), rng.randint(1, 60)
        lengths = [rng.randint(max(1, s // rng.choice([1, 2, 8])), s) for _ in range(b)]
        lengths[rng.randrange(b)] = s
        tiles, chunks, longest_first = _plan(lib, b, heads, s, UNKNOWN if padded else b * s - sum(lengths))
        nq = -(-s // TILE)
        assert 1 <= tiles <= nq and chunks == -(-nq // tiles) and (chunks == 1 or not longest_first)
        ratio.append(_time(lengths, s, heads, tiles, chunks, padded, lib.item if longest_first else None)
                     / _time(lengths, s, heads, nq, 1, padded))
    assert max(ratio) <= 1.13 and sum(r > 1.03 for r in ratio) <= 3, sorted(ratio)[-5:]
    assert sum(ratio) / len(ratio) < 0.9


@pytest.mark.parametrize("heads", [1, 12, 16])
def test_few_ragged_pairs_are_cut_into_tiles_where_that_is_shorter(lib, heads):
    """Tiles dealt longest first against whole pairs: never a longer list, all tiles inside the bound that the launch is made for."""
    rng = random.Random(heads)
    ratio = []
    for _ in range(3000):
        s, b = rng.randint(1, 512), rng.randint(1, CTAS // heads)
        lengths = [rng.randint(s // rng.choice([1, 2, 4, 12]), s) for _ in range(b)]
        lengths[rng.randrange(b)] = s
        most = lib.cut(b, heads, s, ctypes.c_int64(sum(lengths)), ctypes.c_int64(CTAS))
        if most == 0 or _plan(lib, b, heads, s, b * s - sum(lengths))[1] > 1:
            continue
        blocks = sorted((-(-n // TILE) for n in lengths), reverse=True)
        tiles = [4 * n for n in blocks for _ in range(heads * n)]
        assert len(tiles) <= most <= 64 * CTAS
        ctas = min(CTAS, most)
        load = [0] * ctas
        seen = set()
        for r in range(-(-most // ctas)):
            for cta in range(ctas):
                i = lib.item(r, cta, ctas)
                seen.add(i)
                load[cta] += tiles[i] if i < len(tiles) else 0
        assert seen >= set(range(len(tiles)))
        ratio.append(max(load) / max((3 * n + 1) * n for n in blocks))
    assert not ratio or (max(ratio) <= 1.0 and sum(ratio) / len(ratio) < 0.75), max(ratio)
    assert ratio or heads == 1


def test_equal_lengths_are_cut_where_that_is_shorter(lib):
    """Full sequences, or all of the same number of tiles: the shortest of all divisions."""
    for heads in (12, 16):
        for s in (128, 200, 256, 384, 512):
            nq = -(-s // TILE)
            for b in range(1, 80):
                tiles, chunks, longest_first = _plan(lib, b, heads, s, (s - (nq - 1) * TILE - 1) if b % 2 else 0)
                best = min(_time([s] * b, s, heads, t, -(-nq // t), False) for t in range(1, nq + 1))
                assert not longest_first and _time([s] * b, s, heads, tiles, chunks, False) == best, (heads, s, b)


def test_every_item_has_one_turn(lib):
    for items in (149, 148 * 2, 148 * 3 - 1, 148 * 7 + 31):
        rounds = -(-items // CTAS)
        seen = [lib.item(r, c, CTAS) for r in range(rounds) for c in range(CTAS)]
        assert sorted(seen) == list(range(rounds * CTAS))


def test_limits_of_the_order(lib):
    assert _plan(lib, 256, 37, 512, UNKNOWN) == (4, 1, True)      # 256 sequences, 64 rounds of 148 pairs
    assert _plan(lib, 257, 1, 512, UNKNOWN) == (4, 1, False)
    assert _plan(lib, 256, 38, 512, UNKNOWN) == (4, 1, False)
    assert _plan(lib, 65535, 32768, 512, 0) == (4, 1, False)      # chunks would pass 32 bits
    assert not _plan(lib, 9, 16, 512, UNKNOWN)[2]                 # a round is enough
