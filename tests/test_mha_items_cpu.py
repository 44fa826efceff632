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
                                 'extern "C" int32_t shorter(int32_t tiles, int32_t longest, int32_t ctas) { return b200::cutIsShorter(tiles, longest, ctas); }\n'
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


def _cut(lib, heads, s, lengths):
    """Units of the longest CTA's list over those of whole pairs: of the tiles as the CTAs deal them, 1 where they decide on whole pairs, None where the host does."""
    b = len(lengths)
    most = lib.cut(b, heads, s, ctypes.c_int64(sum(lengths)), ctypes.c_int64(CTAS))
    if most == 0 or _plan(lib, b, heads, s, b * s - sum(lengths))[1] > 1:
        return None
    blocks = sorted((-(-n // TILE) for n in lengths), reverse=True)
    tiles = [4 * n for n in blocks for _ in range(heads * n)]
    ctas = min(CTAS, most)
    assert len(tiles) <= most and b * heads <= ctas   # a CTA for each pair, should they stay whole
    if not lib.shorter(len(tiles), blocks[0], ctas):
        return 1.0
    rounds = -(-len(tiles) // ctas)
    assert rounds <= 3 * -(-s // TILE) // 4           # what the launch has room for
    load, seen = [0] * ctas, set()
    for r in range(rounds):
        for cta in range(ctas):
            i = lib.item(r, cta, ctas)
            seen.add(i)
            load[cta] += tiles[i] if i < len(tiles) else 0
    assert seen >= set(range(len(tiles)))
    return max(load) / max((3 * n + 1) * n for n in blocks)


@pytest.mark.parametrize("heads", [1, 12, 16])
@pytest.mark.parametrize("seed", range(4))
def test_few_ragged_pairs_are_cut_into_tiles_where_that_is_shorter(lib, heads, seed):
    """Tiles dealt longest first against whole pairs: never a longer list, all tiles inside the bound that the launch is made for."""
    rng = random.Random(100 * seed + heads)
    ratio = []
    for _ in range(3000):
        s, b = rng.randint(129, 512), rng.randint(1, CTAS // heads)
        lengths = [rng.randint(s // rng.choice([1, 2, 4, 12]), s) for _ in range(b)]
        lengths[rng.randrange(b)] = s
        ratio.append(_cut(lib, heads, s, lengths))
    ratio = [r for r in ratio if r is not None]
    assert len(ratio) > 100 and max(ratio) <= 1.0 and sum(ratio) / len(ratio) < 0.8, (len(ratio), max(ratio), sum(ratio) / len(ratio))


@pytest.mark.parametrize("heads", [1, 12, 16])
def test_lengths_just_beyond_a_tile_are_not_cut_where_that_is_longer(lib, heads):
    """Lengths at the edges of tiles, S up to 512 above them: the host guesses that a cut is shorter, the CTAs count."""
    kept = 0
    for s in (130, 200, 256, 257, 300, 385, 400, 512):
        for b in range(1, CTAS // heads + 1):
            for n in (1, 2, 128, 129, 130, 133, 160, 256, 257, 273, 384, 385):
                for first in {s, n, 1}:
                    if max(n, first) <= s:
                        r = _cut(lib, heads, s, [first] + [n] * (b - 1))
                        assert r is None or r <= 1.0, (s, b, n, first)
                        kept += r == 1.0
    assert kept > 100
    for s, lengths, h in [(160, [160, 153, 160, 133, 160], 16), (130, [130] + [129] * 6, 12), (256, [256] + [129] * 91, 1),
                          (273, [257, 273, 260, 259, 257, 270, 265, 261, 258, 1], 12), (512, [128] + [100] * 11, 12)]:
        assert _cut(lib, h, s, lengths) == 1.0   # the guess alone cuts these


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
