"""How the item estimate cuts its work (csrc/item_split.h): compiled for the host, every item of a launch must belong to exactly
one block, whatever the lengths, heads and blocks."""
import ctypes
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WARPS, BLOCKS = 7, 296      # scanning warps of a block; blocks of a launch on 148 SMs

SHIM = """
#include <algorithm>
#include "item_split.h"
using namespace adamas;
extern "C" {
int cache_heads(int h, int group) { return item_cache_heads(h, group); }
int query_heads(int items, int group, int warps) { return item_query_heads(items, group, warps); }
int tiles_of(int n, int t) { return est_tiles(n, t); }
int per_piece(int tiles, int pieces, int blocks) { return item_blocks_per_piece(tiles, pieces, 1, blocks); }
int by_tiles(int heads, int q_heads, int batch, int n, int counts, int rope, int blocks) { return estimate_by_tiles(heads, q_heads, batch, n, counts, rope, blocks); }
int by_tiles_given(int heads, int batch, int n) { return estimate_by_tiles(heads, heads, batch, n, true, false, 296, false); }
void share_one(int tiles, int pieces, int q_part, int blocks, int* out) {
  for (int b = 0; b < blocks; ++b) {
    const ItemShare w = item_share_one(tiles, pieces, q_part, blocks, b);
    out[2 * b] = w.pos; out[2 * b + 1] = w.end;
  }
}
int share_batch(const int* cum, int batch, int pieces, int q_part, int blocks, int* out) {
  const int total = cum[batch] * pieces;
  const int segments = batch * pieces;
  bool apart = item_apart_possible(total, segments, blocks);
  if (apart && !item_apart_simple(total, segments, blocks)) {
    int most = 0;
    for (int s = 0; s < batch; ++s) most = std::max(most, item_apart_most(cum[s + 1] - cum[s], total, blocks - segments));
    apart = q_part > 1 && !item_apart_hopeless(total, segments, q_part, blocks) && item_apart_pays(most, total, q_part, blocks);
  }
  for (int b = 0; b < blocks; ++b) {
    const ItemShare w = apart ? item_share_apart(cum, batch, pieces, blocks, b) : item_share_even(total, blocks, b);
    out[2 * b] = w.pos; out[2 * b + 1] = w.end;
  }
  return apart;
}
int share_columns(const int* cum, int batch, int pieces, int q_part, int blocks, int* out) {   // column shares, piece after piece
  const int columns = item_blocks_per_piece(cum[batch], pieces, q_part, blocks);
  int longest = 0;
  for (int s = 0; s < batch; ++s) longest = std::max(longest, cum[s + 1] - cum[s]);
  const int alike = columns > 0 ? item_columns_alike(cum, batch, columns) : 0;
  const bool apart = columns > 0 && item_columns_apart(cum[batch], longest, batch, q_part, columns);
  for (int b = 0; b < blocks && columns > 0; ++b) {
    const int c = b / pieces;
    ItemShare w{0, 0};
    if (c < columns) w = alike > 0 ? item_share_alike(cum[1], batch, alike, c) : apart ? item_share_apart(cum, batch, 1, columns, c) : item_share_even(cum[batch], columns, c);
    out[2 * b] = w.pos; out[2 * b + 1] = w.end;
  }
  return columns == 0 ? 0 : alike > 0 ? 1 : apart ? 2 : 3;
}
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("split")
    (d / "shim.cpp").write_text(SHIM)
    # (-ftrapv: a product beyond 31 bits ends the test)
    subprocess.run([gxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-ftrapv", "-I", os.path.join(ROOT, "adamas_b200", "csrc"),
                    "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def _one(split, tiles, pieces, q_part, blocks=BLOCKS):
    out = np.full((blocks, 2), -1, dtype=np.int32)
    split.share_one(tiles, pieces, q_part, blocks, out.ctypes.data_as(ctypes.c_void_p))
    return out


def _batch(split, tiles, pieces, q_part, blocks=BLOCKS):
    cum = np.concatenate([[0], np.cumsum(tiles)]).astype(np.int32)
    out = np.full((blocks, 2), -1, dtype=np.int32)
    apart = split.share_batch(cum.ctypes.data_as(ctypes.c_void_p), len(tiles), pieces, q_part, blocks,
                              out.ctypes.data_as(ctypes.c_void_p))
    return out, bool(apart)


def _covers(shares, total):
    busy = sorted((int(a), int(b)) for a, b in shares if a != b)
    assert all(a < b for a, b in busy)
    assert busy[0][0] == 0 and busy[-1][1] == total
    assert all(x[1] == y[0] for x, y in zip(busy, busy[1:]))


GROUPED = [(1, 16), (1, 128), (1, 1024), (2, 32), (4, 7), (8, 4), (8, 8), (8, 12), (5, 3), (128, 8), (301, 3)]


@pytest.mark.parametrize("blocks", [BLOCKS, BLOCKS // 2])
@pytest.mark.parametrize("heads,group", GROUPED)
def test_one_grouped_sequence_every_item_once(split, heads, group, blocks):
    rng = random.Random(heads * group)
    hp = split.cache_heads(heads, group)
    most = 0
    for n in sorted([0, 1, 31, 32, 33, 127, 128, 129, 4095] + [int(2 ** rng.uniform(5, 20)) for _ in range(12)]):
        tiles = split.tiles_of(n, 128 // hp)
        q_part = split.query_heads(tiles * (heads // hp), group, WARPS * blocks)
        pieces = heads // hp * -(-group // q_part)
        _covers(_one(split, tiles, pieces, q_part, blocks), tiles * pieces)
        # a launch has shared memory for the rows of its longest sequence: a shorter one must not need more
        assert q_part >= most
        most = q_part


@pytest.mark.parametrize("blocks", [BLOCKS, BLOCKS // 2])
@pytest.mark.parametrize("heads", [1, 2, 3, 7, 28, 33, 40, 61, 96, 101, 147, 148, 149, 151, 295, 297, 600, 1000, 1024])
def test_one_sequence_every_item_once(split, heads, blocks):
    """No grouped queries: a grid of pieces, or the line; never more blocks than may be resident."""
    rng = random.Random(heads)
    hp = split.cache_heads(heads, 1)
    for n in [1, 31, 32, 33, 127, 128, 129, 4095] + [int(2 ** rng.uniform(5, 20)) for _ in range(12)]:
        tiles, pieces = split.tiles_of(n, 128 // hp), heads // hp
        grid = min(blocks, tiles * pieces)
        per = split.per_piece(tiles, pieces, grid)
        assert per * pieces <= grid and (per > 0 or pieces > grid * 3 // 4 or grid % pieces > grid // 4)
        if per > 0:
            # a long row leaves no more than a quarter of the blocks idle
            assert tiles < 1000 or (grid - per * pieces) * 4 <= grid
        _covers(_one(split, tiles, pieces, 1, grid), tiles * pieces)


@pytest.mark.parametrize("heads,group", [(4, 7), (8, 4), (8, 8), (1, 16), (4, 8)])
def test_short_sequence_in_a_large_cache(split, heads, group):
    """What a block gets follows from the length, which the kernel reads, and not from the capacity: at 3000 tokens half of the
    blocks and more have something, or every tile and query head is on its own."""
    hp = split.cache_heads(heads, group)
    tiles = split.tiles_of(2999, 128 // hp)
    q_part = split.query_heads(tiles * (heads // hp), group, WARPS * BLOCKS)
    shares = _one(split, tiles, heads // hp * -(-group // q_part), q_part)
    assert (shares[:, 1] > shares[:, 0]).sum() >= min(BLOCKS // 2, tiles * heads // hp * group)


@pytest.mark.parametrize("batch,pieces", [(1, 1), (3, 10), (32, 8), (40, 8), (1024, 1)])
def test_batch_without_tokens(split, batch, pieces):
    """Lengths that are all zero (a batch before its lengths are set): no block has anything, and nothing is divided by the total."""
    shares, apart = _batch(split, [0] * batch, pieces, 1)
    assert not apart and (shares[:, 0] == shares[:, 1]).all()


@pytest.mark.parametrize("heads,group", [(4, 1), (40, 1), (32, 1), (7, 1), (8, 4), (4, 7), (8, 8), (1, 16)])
def test_batches_every_item_once(split, heads, group):
    rng = random.Random(heads * 100 + group)
    for case in range(60):
        batch = rng.choice([1, 2, 3, 8, 31, 32, 33, 100, 256, 1024])
        top = rng.choice([1, 40, 700, 5000, 60000])
        lengths = [rng.randrange(0, top + 1) for _ in range(batch)]
        hp = split.cache_heads(heads, group)
        # (a length of 0 tokens besides the newest still has its append; an absent sequence has nothing)
        tiles = [0 if rng.random() < 0.1 else split.tiles_of(n, 128 // hp) for n in lengths]
        if sum(tiles) == 0:
            tiles[-1] = 1
        q_part = split.query_heads(sum(tiles) * (heads // hp), group, WARPS * BLOCKS)
        pieces = heads // hp * -(-group // q_part)
        shares, apart = _batch(split, tiles, pieces, q_part)
        _covers(shares, sum(tiles) * pieces)
        if apart:    # nobody has more than one segment, nor much more than an even share
            ends = np.cumsum(np.repeat(tiles, pieces))
            for a, b in shares:
                if a != b:
                    assert np.searchsorted(ends, a, "right") == np.searchsorted(ends, b - 1, "right")
            total, blocks = sum(tiles) * pieces, BLOCKS
            if batch * pieces * 8 <= blocks:
                assert (shares[:, 1] - shares[:, 0]).max() <= -(-total // blocks) * 1.15 + 1
            elif total * batch * pieces > 4 * blocks * blocks:
                assert ((shares[:, 1] - shares[:, 0]).max() - total // blocks) * q_part <= 24 + q_part


@pytest.mark.parametrize("batch,n,heads,group,want", [(64, 2000, 4, 7, True), (32, 4000, 4, 7, True), (32, 2000, 8, 8, True),
                                                      (24, 1500, 40, 1, False), (20, 16000, 40, 1, False), (12, 8000, 40, 1, False),
                                                      (32, 6000, 32, 1, False), (8, 32768, 32, 1, False), (4, 64000, 32, 1, True)])
def test_batches_that_keep_to_one_segment(split, batch, n, heads, group, want):
    hp = split.cache_heads(heads, group)
    tiles = [split.tiles_of(n - 1, 128 // hp)] * batch
    q_part = split.query_heads(sum(tiles) * (heads // hp), group, WARPS * BLOCKS)
    assert _batch(split, tiles, heads // hp * -(-group // q_part), q_part)[1] is want


@pytest.mark.parametrize("blocks", [BLOCKS, BLOCKS // 2])
@pytest.mark.parametrize("heads,group", [(4, 1), (40, 1), (32, 1), (7, 1), (151, 1), (8, 4), (4, 7), (8, 8), (1, 16)])
def test_columns_of_a_batch_every_item_once(split, heads, group, blocks):
    """Every piece's blocks cover all sequences' tiles; equal lengths get equal shares of one sequence; columns of ragged lengths that
    are kept apart have one sequence each and not much more than an even share."""
    rng = random.Random(heads * 10 + group + blocks)
    for case in range(80):
        batch = rng.choice([1, 2, 3, 8, 16, 31, 37, 100, 256, 1024])
        top = rng.choice([1, 40, 700, 5000, 60000])
        hp = split.cache_heads(heads, group)
        alike = case % 4 == 0
        lengths = [top] * batch if alike else [rng.randrange(0, top + 1) for _ in range(batch)]
        tiles = [0 if not alike and rng.random() < 0.1 else split.tiles_of(n, 128 // hp) for n in lengths]
        if sum(tiles) == 0:
            tiles[-1] = 1
        q_part = split.query_heads(sum(tiles) * (heads // hp), group, WARPS * blocks)
        pieces = heads // hp * -(-group // q_part)
        grid = min(blocks, sum(tiles) * pieces)
        cum = np.concatenate([[0], np.cumsum(tiles)]).astype(np.int32)
        out = np.full((grid, 2), -1, dtype=np.int32)
        mode = split.share_columns(cum.ctypes.data_as(ctypes.c_void_p), batch, pieces, q_part, grid, out.ctypes.data_as(ctypes.c_void_p))
        if mode == 0:
            continue
        columns = split.per_piece(int(cum[-1]), pieces, grid) if q_part == 1 else None
        for piece in range(pieces):
            mine = out[piece::pieces]
            _covers(mine[:columns], int(cum[-1]))
        sizes = out[:, 1] - out[:, 0]
        if mode in (1, 2):
            for a, b in out:
                if a != b:
                    assert np.searchsorted(cum[1:], a, "right") == np.searchsorted(cum[1:], b - 1, "right")
        if mode == 1:
            assert sizes.max() - sizes[sizes > 0].min() <= 1


@pytest.mark.parametrize("batch", [3, 4, 7, 8, 16, 33])
@pytest.mark.parametrize("heads", [4, 32, 40])
def test_an_average_length_in_front_does_not_make_the_others_equal(split, heads, batch):
    """Lengths are equal only if all of them are: otherwise the rule for ragged ones decides."""
    pieces = heads // split.cache_heads(heads, 1)
    tiles = [100] + [100 + (40 if i % 2 else -40) for i in range(batch - 1 - (batch - 1) % 2)] + [100] * ((batch - 1) % 2)
    assert len(tiles) == batch and sum(tiles) == 100 * batch
    cum = np.concatenate([[0], np.cumsum(tiles)]).astype(np.int32)
    out = np.full((BLOCKS, 2), -1, dtype=np.int32)
    assert split.share_columns(cum.ctypes.data_as(ctypes.c_void_p), batch, pieces, 1, BLOCKS, out.ctypes.data_as(ctypes.c_void_p)) in (2, 3)


@pytest.mark.parametrize("heads,batch,n,rope,want", [
    # both sides of every line, with counts
    (16, 1, 3584, False, True), (16, 1, 3585, False, False), (16, 1, 600, True, False), (16, 4, 1856, False, True), (16, 4, 1857, False, False),
    (16, 3, 1536, True, True), (16, 3, 1537, True, False), (32, 1, 3584, False, True), (32, 1, 3585, False, False), (32, 1, 600, True, False),
    (32, 2, 3584, False, True), (32, 3, 2304, False, True), (32, 3, 2305, False, False), (32, 2, 1280, True, True), (32, 2, 1281, True, False),
    (32, 8, 320, True, True), (32, 8, 321, True, False), (32, 10, 204, True, True), (32, 10, 205, True, False), (16, 16, 314, False, True), (16, 16, 315, False, False),
    (64, 1, 600, False, False), (64, 4, 768, False, True), (64, 4, 769, False, False), (64, 2, 300, True, False),
    # short batches that were slower in the item kernel by 4 to 15 % (us a layer beside estimate_by_tiles)
    (32, 2, 600, True, True), (32, 2, 1000, True, True), (32, 2, 1250, True, True), (32, 3, 300, True, True), (32, 3, 450, True, True),
    (32, 3, 300, False, True), (32, 3, 1500, False, True), (32, 4, 600, False, True), (32, 5, 600, False, True), (32, 6, 450, False, True),
    (32, 10, 207, False, True), (16, 3, 1500, True, True), (16, 4, 1800, False, True), (64, 2, 200, False, True),
    # ... and ones that are not
    (32, 6, 1000, False, False), (32, 4, 1500, False, False), (32, 3, 1000, True, False), (16, 8, 1000, False, False), (16, 8, 600, True, False),
    (32, 1024, 3000, False, False), (16, 1024, 2000000, True, False),
    # large batches: more segments of four heads than blocks
    (32, 37, 300, False, False), (32, 38, 300, False, True), (32, 128, 1024, False, True), (32, 128, 1025, False, False), (32, 96, 640, True, True),
    (32, 96, 641, True, False), (64, 18, 300, False, False), (64, 19, 300, False, True), (64, 64, 1025, False, False), (64, 64, 320, True, True),
    (64, 64, 321, True, False), (16, 112, 256, False, True), (16, 112, 257, False, False), (16, 112, 200, True, False),
])
def test_which_kernel_counts(split, heads, batch, n, rope, want):
    assert bool(split.by_tiles(heads, heads, batch, n, 1, rope, BLOCKS)) is want
    for h, q in ((heads // 2, heads), (40, 40), (4, 4)):     # grouped queries and other head counts: the item kernel
        assert not split.by_tiles(h, q, batch, n, 1, rope, BLOCKS)


@pytest.mark.parametrize("heads,n,want", [(16, 65535, True), (16, 65536, False), (32, 1000000, True), (64, 1000000, True), (8, 100, False)])
def test_which_kernel_without_counts(split, heads, n, want):
    assert bool(split.by_tiles(heads, heads, 1, n, 0, 0, BLOCKS)) is want


@pytest.mark.parametrize("heads,n,want", [(16, 5120, True), (16, 5121, False), (32, 12288, True), (32, 12289, False), (64, 4096, False), (64, 4097, True),
                                          (64, 12288, True), (64, 12289, False), (8, 100, False)])
def test_which_kernel_counts_with_given_codes(split, heads, n, want):
    assert bool(split.by_tiles_given(heads, 1, n)) is want
    assert not split.by_tiles_given(heads, 8, n)           # (batches: the rule with the append)
