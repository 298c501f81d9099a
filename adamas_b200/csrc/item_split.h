// How the work of the item estimate (estimate_items.cuh) is cut: what an item is, which of them a block takes; and which launches go
// to it (estimate_by_tiles).  Plain C++ but for the qualifiers, so that both can be checked without a GPU.
//
// An item is 128 / HP tokens (a tile) x HP cache heads; a piece is HP cache heads with a part of their query heads.  The items of
// a launch form a line: sequence after sequence, in it piece after piece, in it tile after tile.  A segment is a piece of a sequence.
#pragma once

#ifdef __CUDACC__
#define ADAMAS_HD __host__ __device__ __forceinline__
#else
#define ADAMAS_HD inline
#endif

namespace adamas {

constexpr int kItemWarps = 7;            // of a block, that scan
constexpr int kItemBlocksPerSm = 2;

// Cache heads of an item, and the query heads of a cache head that a warp takes at a time.  An item has as long a run of a
// token's codes as divides the cache heads, but not more than kItemRows query rows (every row has count tables in every block
// that works on it).  The group of a cache head is halved as long as every part still
// finds a warp of its own (`warps` on the chip; `items` are those of undivided groups): a second round costs more than it saves.
constexpr int kItemRows = 8;
ADAMAS_HD int item_cache_heads(int kv_heads, int q_group) {
  int hp = 4;
  while (hp > 1 && (kv_heads % hp != 0 || (q_group > 1 && hp * q_group > kItemRows))) hp /= 2;
  return hp;
}
ADAMAS_HD int item_query_heads(int items, int q_group, int warps) {
  int heads = q_group;
  for (; heads > 2 * kItemRows; items *= 2) heads = (heads + 1) / 2;
  for (; heads > 1 && items <= warps / 2; items *= 2) heads = (heads + 1) / 2;
  return heads;
}

// Tiles of n tokens.  A sequence whose first token is being appended (n = 0) has an empty one: somebody has to append.
ADAMAS_HD int est_tiles(int n, int tile_tokens) { return n == 0 ? 1 : (n + tile_tokens - 1) / tile_tokens; }

struct ItemShare {
  int pos, end;   // items of the line; none where pos == end
};

// An even cut of the line: block b of `blocks`.
ADAMAS_HD ItemShare item_share_even(int total, int blocks, int b) {
  const int B = blocks < total ? blocks : total;   // (every block that takes part has some)
  if (b >= B) return {0, 0};
  const int q = total / B, r = total - q * B;
  return {b * q + b * r / B, (b + 1) * q + (b + 1) * r / B};   // b * total / B
}

// What keeping to one segment may cost a block of one sequence: this many items (times the query heads of a cache head in them)
// more than an even cut would give it.
constexpr int kItemMore = 16;

// One sequence.  Every piece has the same number of blocks, which share its tiles evenly; a remainder of the blocks stays idle
// (of 296: 11 % with 33 pieces, 18 % with 61, at most a quarter).  0, an even cut of the line instead, with more pieces than blocks, or where more
// than a quarter would stay idle and that costs more than a second segment does (151 heads: 48K tokens 112 us a layer with a block
// per piece, 82 cut evenly, 12K 41 / 35; 61 heads, 48K: 41 with a remainder of 18 %, 49 cut evenly).
ADAMAS_HD int item_blocks_per_piece(int tiles, int pieces, int q_part, int blocks) {
  const int per = blocks / pieces, idle = blocks - per * pieces;
  return idle > blocks / 4 && static_cast<long long>(tiles) * idle * q_part > static_cast<long long>(kItemMore) * per * blocks ? 0 : per;
}
ADAMAS_HD ItemShare item_share_one(int tiles, int pieces, int q_part, int blocks, int b) {
  const int per = item_blocks_per_piece(tiles, pieces, q_part, blocks);
  if (per == 0) return item_share_even(tiles * pieces, blocks, b);
  const int share = (tiles + per - 1) / per;
  // (Long shares: the pieces of a range of tokens in neighbouring blocks, as in a batch's columns, 28 query heads over 4, 100K 24.3 -> 23.6 us a
  // layer.  Short ones: the blocks that have something spread over the launch, 3K 11.8 / 11.0.)
  const int part = share > kItemWarps ? b / pieces : b % per, piece = share > kItemWarps ? b % pieces : b / per, first = part * share;
  if (piece >= pieces || part >= per || first >= tiles) return {0, 0};
  return {piece * tiles + first, piece * tiles + (share < tiles - first ? first + share : tiles)};
}

// A batch: cum[s] tiles lie in front of sequence s.
//
// The blocks form columns of one block per piece (item_blocks_per_piece of them, neighbours in the launch; none, an even cut of the whole
// line, where too many blocks would be left over).  The columns share the line of ONE piece's tiles, so that the pieces of a token's codes,
// which lie side by side, are read at about the same time: with the pieces of a sequence one after the other on the line, blocks read pieces
// of the same tokens far apart (32 heads, us a layer: 8 x 32K 76.0 -> 72.2, 32 x 4-8K 67.9 -> 63.0, 16 x 15-30K 58.4 -> 56.2; 4 x 30K of 64 heads
// 69.7 -> 63.4; all columns of a piece next to one another 72.9, 64.0, 58.1 and 64.0).
//
// Where the sequences are no more than the columns, every column may take a part of ONE, the columns dealt out in proportion to the
// tiles.  A second segment costs a block about 4 us (a query to load and code behind a barrier, counts to add up), a larger share its
// items.  They are kept apart
//  * with equal lengths, where a seventh of the columns at most stays without any: the shares are equal as well (8 x 32K 72.8 a layer, 73.4
//    cut evenly; 20 x 16K of 8 heads 30.7 / 33.1; 10 x 26K of 32 heads, where a fifth would stay idle, 82.2 / 82.0);
//  * where there is little work, or an eighth as many sequences as columns: shares differ by an eighth at most (4 sequences x 64K x 32
//    heads 71.3 us a layer cut evenly, 67.7 apart);
//  * where the largest share cannot be much more than an even one.  It is at most that of the longest sequence with a column of its own, and at
//    most tiles / (columns - sequences): item_columns_apart.
// (Products stay below 2^31.  Lengths that are all zero leave nothing to deal out.)  In what follows a segment is a sequence, a block a
// column, and the kernel's calls have pieces = 1.  item_apart_most is the exact largest share, which takes a look at every length (2.7 us a layer
// on the device): item_columns_apart bounds it instead.  No kernel asks for it, nor for item_apart_hopeless and item_apart_pays, nor cuts several pieces
// apart on one line: the tests of such cuts do.
constexpr int kItemApart = 24;
ADAMAS_HD bool item_apart_possible(int total, int segments, int blocks) { return total > 0 && segments <= blocks && total <= 0x7fffffff / blocks; }
ADAMAS_HD bool item_apart_few(int segments, int blocks) { return segments * 8 <= blocks; }
ADAMAS_HD bool item_apart_simple(int total, int segments, int blocks) {
  return static_cast<long long>(total) * segments <= 4LL * blocks * blocks || item_apart_few(segments, blocks);
}
// (with about one block per segment, and an average one too much for it, there is nothing to ask)
ADAMAS_HD bool item_apart_hopeless(int total, int segments, int q_part, int blocks) {
  return 2 * segments > blocks && static_cast<long long>(total) * (blocks - segments) * q_part > static_cast<long long>(kItemApart) * segments * blocks;
}
// the most that a block gets of the segments of a sequence of `tiles` tiles; spare = blocks - segments
ADAMAS_HD int item_apart_most(int tiles, int total, int spare) {
  const int blocks = 1 + tiles * spare / total;   // of each segment, at least
  return (tiles + blocks - 1) / blocks;
}
ADAMAS_HD bool item_apart_pays(int most, int total, int q_part, int blocks) { return (most - total / blocks) * q_part <= kItemApart; }
ADAMAS_HD ItemShare item_share_apart(const int* cum, int batch, int pieces, int blocks, int b) {
  const int segments = batch * pieces, total = cum[batch] * pieces, spare = blocks - segments;
  auto seg_start = [&](int g) {   // where segment g starts on the line
    const int s = g / pieces;
    return s == batch ? total : cum[s] * pieces + (g - s * pieces) * (cum[s + 1] - cum[s]);
  };
  auto first_block = [&](int g) { return g + seg_start(g) * spare / total; };
  int lo = 0, hi = segments - 1;
  while (lo < hi) {   // the last segment that starts at or before this block
    const int mid = (lo + hi + 1) >> 1;
    if (first_block(mid) <= b) lo = mid; else hi = mid - 1;
  }
  const int start = seg_start(lo), n_items = seg_start(lo + 1) - start, f = first_block(lo), all = first_block(lo + 1) - f;
  const int nblk = all < n_items ? all : n_items;
  if (b - f >= nblk) return {0, 0};
  return {start + n_items * (b - f) / nblk, start + n_items * (b - f + 1) / nblk};
}

constexpr int kItemApartPlain = 40;   // (without grouped queries)
ADAMAS_HD bool item_columns_apart(int total, int longest, int batch, int q_part, int columns) {
  if (!item_apart_possible(total, batch, columns)) return false;
  if (item_apart_simple(total, batch, columns)) return true;
  const int spare = columns - batch, most = static_cast<long long>(longest) * spare <= total ? longest : total / spare + 1;
  return (most - total / columns) * q_part <= (q_part > 1 ? kItemApart : kItemApartPlain);
}
// Equal lengths (the longest is the average): `per` columns a sequence, or 0.
ADAMAS_HD int item_columns_alike(int total, int longest, int batch, int columns) {
  if (batch > columns || static_cast<long long>(longest) * batch != total || columns % batch > columns / 7) return 0;
  return columns / batch;
}
// The same for a host that has the line alone: cum[s] tiles lie in front of sequence s.
inline int item_columns_alike(const int* cum, int batch, int columns) {
  int longest = 0;
  for (int s = 0; s < batch; ++s) longest = cum[s + 1] - cum[s] > longest ? cum[s + 1] - cum[s] : longest;
  return item_columns_alike(cum[batch], longest, batch, columns);
}
ADAMAS_HD ItemShare item_share_alike(int tiles, int batch, int per, int c) {
  const int s = c / per, nblk = per < tiles ? per : tiles, i = c - s * per;
  if (s >= batch || i >= nblk) return {0, 0};
  const int q = tiles / nblk, r = tiles - q * nblk;
  return {s * tiles + i * q + i * r / nblk, s * tiles + (i + 1) * q + (i + 1) * r / nblk};
}

// Which estimate kernel.  n is the length, or the cache's capacity where the length is on the device.
//
// The tile pipeline (estimate.cuh) takes 16, 32 and 64 heads without grouped queries, where a warp keeps the planes of its heads in registers.
// With counts, one L2 atomic per distance in it, it is ahead only where a block of the item kernel has next to nothing to scan and its
// query decides.  us a layer, tiles / items.  One sequence, without rotation: 16 heads, 600 tokens 8.2 / 8.7, 1.5K 8.2 / 8.7, 4K 9.5 / 8.5; 32 heads, 1.5K
// 8.7 / 8.7, 3.6K 9.3 / 9.5, 4.5K 9.9 / 9.7; with it 16 heads, 1.5K 9.0 / 8.7; 32 heads, 1.5K 9.8 / 9.4.  Batches of 16 heads, without rotation 2 x 3.6K
// 10.5 / 11.1, 4 x 1.8K 10.9 / 11.4, 5 x 1.5K 11.8 / 11.6, 6 x 1K 11.3 / 11.8, 8 x 1K 12.4 / 11.8; with it 2 x 2.3K 10.8 / 11.4, 2 x 2.7K 11.8 / 11.4, 4 x 1K
// 11.3 / 11.9, 4 x 1.5K 12.3 / 11.9, 8 x 450 12.1 / 12.3, 8 x 600 12.7 / 12.5.  Batches of 32 heads, where another sequence costs the tiles more, without
// rotation 2 x 3.6K 11.9 / 11.9, 3 x 1.5K 11.3 / 11.8, 3 x 2.5K 12.8 / 12.3, 4 x 1K 11.4 / 11.8, 4 x 1.5K 12.4 / 12.3, 6 x 450 11.8 / 12.3, 6 x 1K 13.8 / 12.8, 8 x 300
// 13.0 / 12.8, 10 x 200 13.4 / 14.2; with it 2 x 600 10.3 / 11.8, 2 x 1.25K 10.7 / 11.9, 2 x 1.8K 12.0 / 11.9, 3 x 450 10.8 / 12.3, 3 x 600 12.3 / 12.3.
// 64 heads: one sequence, 1.5K 10.6 / 9.5; batches without rotation 2 x 300 11.3 / 11.8, 4 x 200 12.4 / 12.8, 4 x 600 13.3 / 13.2, 4 x 1.5K 15.9 / 15.3;
// with it 2 x 300 12.8 / 12.3.  The same with many layers, whose caches do not stay in L2: 32 heads with rotation 3 x 700 12.3 / 12.0 (3 x 350 in caches
// for 700: 8.0 / 9.5), 3 x 1K 12.4 / 12.1, 4 x 450 12.8 / 12.5, 5 x 300 9.0 / 10.5, 8 x 300 10.6 / 11.2, 8 x 450 14.7 / 14.1, 10 x 200 11.2 / 12.3; 64 heads without 3 x 700
// 13.2 / 13.1 (350 in 700: 9.6 / 10.3), 5 x 300 10.3 / 11.8, 10 x 300 15.1 / 17.0, 16 x 200 18.4 / 18.3; 16 heads without 16 x 450 14.8 / 13.9, 10 x 700 13.3 / 12.9.
//
// Where a batch has more segments (of four heads) than the item kernel has blocks, a block codes a query and clears and adds up count
// tables for each of its segments, and short rows go to the tiles again: 32 heads, 36 x 260 (288 segments on 296 blocks) 30.0 / 28.2, 48 x 300
// 38.0 / 42.1, 48 x 1.1K 45.6 / 47.7, 128 x 200 81.1 / 90.4, 160 x 540 116.3 / 117.1; with rotation 48 x 300 39.6 / 43.6, 52 x 1.2K 51.2 / 51.5; 64 heads, 64 x
// 300 81.7 / 90.2, 48 x 1.1K 79.4 / 83.5, with rotation 64 x 260 86.6 / 93.0, 52 x 700 84.6 / 84.0; 16 heads, 112 x 200 45.3 / 47.9, 112 x 420 49.6 / 48.8.
//
// With given codes nobody waits for the query and the tiles keep up longer (us, one sequence, tiles / items): 16 heads, 4.5K 1.86 / 2.05, 6K 2.24 / 2.18; 32
// heads, 4.5K 2.18 / 2.68, 9K 3.06 / 3.52, 14K 3.96 / 3.97; 64 heads, 3.5K 2.95 / 2.75, 4.5K 3.14 / 3.57, 9K 4.47 / 4.88, 14K 7.27 / 7.00.
//
// Without counts there are no atomics: 32 and 64 heads stay with the tiles (one estimate of 32 heads, 64K 11.0 / 11.8, 256K
// 44.2 / 46.9; 64 heads, 32K 10.8 / 12.2), 16 heads do not (128K 17.8 / 11.9).
inline bool tile_heads(int num_heads, int q_heads) { return q_heads == num_heads && (num_heads == 16 || num_heads == 32 || num_heads == 64); }
inline bool estimate_by_tiles(int num_heads, int q_heads, int batch, int n, bool counts, bool rope, int blocks, bool append = true) {
  if (!tile_heads(num_heads, q_heads)) return false;
  const long long tokens = static_cast<long long>(batch) * n;
  if (!counts) return num_heads != 16 || tokens < 65536;
  if (!append && batch == 1) return num_heads == 64 ? n > 4096 && n <= 12288 : n <= (num_heads == 16 ? 5120 : 12288);
  if (n > 3584 || (rope && batch == 1)) return false;
  if (batch * (num_heads / 4) > blocks) return n <= (num_heads == 16 ? (rope ? 0 : 256) : !rope ? 1024 : num_heads == 32 ? 640 : 320);
  if (num_heads == 16) return rope ? tokens <= 4608 : tokens + 200 * batch <= 8224;
  if (num_heads == 32) return batch * tokens <= (rope ? 20480 : 20736) && !(rope && tokens > 2560);
  return !rope && batch > 1 && tokens <= 3072;
}

}  // namespace adamas
