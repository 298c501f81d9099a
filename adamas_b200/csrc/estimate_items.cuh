// The distance estimate (and decode append) for any head count and for grouped queries; the tile pipeline, which takes short rows of 16, 32 and 64
// heads and estimates without counts (estimate_by_tiles), is in estimate.cuh, with the parameters and the distance arithmetic.
//
// Bound: integer issue (logic at half rate and 5 population counts at an eighth, code_distance) for grouped
// queries, HBM for long rows, fill and drain for short ones.  Two blocks of 8 warps per SM.  One warp of a block loads, rotates and codes the
// query while the others' first items are on their way, and appends the new token while they scan (a block that starts late, next
// to the last blocks of the kernel in front, had its query 4.5 us after its start when the scanning warps coded it themselves
// behind their requests).  With grouped queries (up to 16 rows a block) it only loads the rows and all warps code them, one each:
// the last warp alone took 2 us longer for eight (32 query heads over 8, 30K: 20.7 us a layer, 18.2 this way; with one row per warp for the four
// rows of other blocks batches and long rows took 1-3 % longer, for the blocks that start late).  The other seven work alone:
//   * its unit of work is an item of 4 KB of codes: 128 / HP tokens x HP heads (HP = 4, 2 or 1, see item_cache_heads).
//     Its own 16-byte asynchronous copies bring items into its own ring of two or three slots: no
//     producer warp, no barrier between warps.  (A bulk copy with a different address in every lane is issued lane after
//     lane, 45 ns each, which bounded small head counts in a pipeline with producer warps.)
//   * lane = token: a lane reads the two halves of a code (chunk c of row r is stored at c ^ f(r), which makes 32 rows hit
//     different bank groups) and the query's planes from shared memory (all lanes the same address).  With grouped
//     queries the code is read once for all query heads of the cache head, or, with fewer items than warps, once for each
//     of the parts in which several warps take them (item_query_heads).  The 32 lanes store 32 consecutive tokens
//     of one output row.
//   * the distances are counted in shared memory, one table of 32-bit counts per query row and slice, and the tables are added to
//     the global per-slice histograms once per block.  One L2 atomic per distance runs at 90 to 165 per ns on the whole chip, which
//     made 1 M distances 6 to 8 us; additions of the constant 1 in shared memory take 1 to 2 cycles per warp, those of packed
//     16-bit counts 4 to 13 (lanes that meet in a word are taken one after the other).
// A piece is HP cache heads (with a part of their query heads, item_query_heads).  A block works on one piece of a sequence over
// many tokens: it codes 1 to 16 query rows instead of all, its tables are small, and it adds up as many distances as there are before
// a table goes out.  How the items are dealt out is in item_split.h.  The first items are requested before the kernel's dependency
// resolves (the cached codes are final).
// Measured, the whole step, us a layer, against token after token with all heads in it and one block of 16 warps per SM: 40 heads,
// 12K 18.1 -> 15.9; 32 query heads over 8, 30K 24.6 -> 22.9; 4 sequences x 128K x 4 heads 35.6 -> 32.5; 32 heads, 128K 49.1 -> 45.7
// (tile pipeline and a counting launch).  Eight scanning warps and a ninth leave 96 registers: 26.2 against 23.7 for the grouped case.
// Lane = head with four tokens per lane (one 4 KB run of codes per warp) was slower than lane = token.
#pragma once
#include "estimate.cuh"

namespace adamas {

constexpr int kItemThreads = kItemWarps * 32 + 32;   // (one more warp: the query and the append)
constexpr int kItemMaxSlots = 3;         // ring slots per warp at most
constexpr int kItemBytes = 4096;
constexpr int kItemCountWords = 388;     // counts per query row and table (a distance is at most 384)
// A block with up to so many tokens in all counts them in global memory one by one: clearing and adding up tables costs more (16
// heads, 2K tokens in a cache of 64K: 13.8 us a layer with tables, 13.6 without; 32 sequences x 600 x 4 heads 14.6 / 14.3).  Not with
// grouped queries, where a piece has more rows (64 sequences x 2K x 28 over 4: 81.0 / 81.9), nor between a block's other segments (256 x 400
// x 40 heads: 237.4 / 239.2).
// Long rows keep their tables: too many blocks would add to the same few counts (4 heads, 60K 13.35 / 13.7, 8 heads, 16K 12.5 / 12.65).
constexpr int kItemDirect = 256, kItemDirectRow = 8192;

// Count tables of a block: the slices that its tokens may fall into.
__host__ __device__ __forceinline__ constexpr int item_tables(int hp, bool grouped) { return hp == 1 && !grouped ? 4 : 2; }

// A 128-element row spread over a warp, dimensions 4 * lane .. in a lane: the rotation, transform and code of a half-warp
// (hadamard_append.cuh) with the same operations in the same order, so the same bits.
template <typename T>
__device__ __forceinline__ void unpack4(uint2 v, float (&x)[4]) {
  const float2 a = Elem<T>::to_f2(v.x), b = Elem<T>::to_f2(v.y);
  x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}
template <typename T>
__device__ __forceinline__ void rope_warp(float (&x)[4], int lane, const float2* cs_table, bool scaled, float mscale) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // dimension pairs sit in lanes l and l ^ 16
    const float other = __shfl_xor_sync(0xffffffffu, x[i], 16);
    const float2 cs = cs_table[(lane & 15) * 4 + i];
    float r = lane >= 16 ? fmaf(other, cs.y, x[i] * cs.x) : fmaf(-other, cs.y, x[i] * cs.x);
    if (scaled) r *= mscale;
    x[i] = Elem<T>::round(r);
  }
}
// The row's code: lanes 4j .. 4j + 3 get its 32-bit word j.
template <typename T>
__device__ __forceinline__ uint32_t code_word_warp(float (&x)[4], int lane, float scale, const PairThresholds<T>& th) {
#pragma unroll
  for (int s = 1; s < 4; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if ((i & s) == 0) {
        const float a = x[i], b = x[i + s];
        x[i] = __fadd_rn(a, b);
        x[i + s] = __fsub_rn(a, b);
      }
    }
  }
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) {
    const float sgn = (lane & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = __fmaf_rn(x[i], sgn, __shfl_xor_sync(0xffffffffu, x[i], m));
  }
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 2; ++j) w |= buckets2<T>(Elem<T>::from_f2(__fmul_rn(x[2 * j], scale), __fmul_rn(x[2 * j + 1], scale)), th, 4 * j);
  w = (w | (w >> 16)) & 0xffu;
  w <<= 8 * (lane & 3);
  w |= __shfl_xor_sync(0xffffffffu, w, 1);
  return w | __shfl_xor_sync(0xffffffffu, w, 2);
}

struct EstShared {
  int64_t kv_row, code_row;   // GROUPED: the new token's first row of the block's piece in the caches
  float2 cs[kHeadDim / 2];
};

// Dynamic shared memory: rings | planes [seg_rows] | query rows and new key rows [seg_rows + HP][128] (append, GROUPED) | counts [tables][seg_rows][kItemCountWords] (hist) | token tiles of the
// sequences before [batch + 1], the most of one (seqs).  GROUPED: several query heads per cache head (q_group > 1).
// MODE 0: with the append inside (u16 distances); 1: the query codes are given; 2: the same with the XOR metric.
template <typename T, int MODE, int HP, bool GROUPED>
__global__ void __launch_bounds__(kItemThreads, kItemBlocksPerSm) estimate_items_kernel(const EstimateParams p, int slots, int seg_rows) {
  constexpr bool APPEND = MODE == 0;
  constexpr int METRIC = MODE == 2 ? 1 : 0;
  constexpr int TT = 128 / HP;          // tokens of an item
  constexpr int kGroups = TT / 32;      // ... in groups of 32
  constexpr int CPR = 2 * HP;           // 16-byte chunks per token of an item
  constexpr int kTables = item_tables(HP, GROUPED);
  extern __shared__ __align__(128) uint8_t item_smem[];
  __shared__ EstShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int len0 = p.seq_len_dev && !p.seqs ? __ldg(p.seq_len_dev) - 1 : p.n_tokens;   // (on its way while the rest is set up)
  const int q_group = GROUPED ? p.q_group : 1;
  const int rows = p.H * q_group;       // query rows of a sequence
  QPlanes* planes = reinterpret_cast<QPlanes*>(item_smem + kItemWarps * slots * kItemBytes);
  uint4* q_rows = reinterpret_cast<uint4*>(planes + seg_rows);
  uint32_t* counts = reinterpret_cast<uint32_t*>(q_rows + (APPEND && GROUPED ? (seg_rows + HP) * (kHeadDim / 8) : 0));
  int* cum = reinterpret_cast<int*>(counts + (p.hist ? kTables * seg_rows * kItemCountWords : 0));
  uint4* ring = reinterpret_cast<uint4*>(item_smem + warp * (slots * kItemBytes));
  // The last warp codes the query, while the others request the first items, and appends the new token while they scan.
  const bool scanning = warp < kItemWarps;
  // (the position's rotation: two of the other warps)
  const int cs_pair = tid - (kItemWarps - 2) * 32;
  const bool cs_here = APPEND && p.ap.rope_on && scanning && cs_pair >= 0;
  const float cs_freq = cs_here ? rope_inv_freq(cs_pair, p.ap.rp) : 0.f;

  // ---- this block's part of the work ------------------------------------------------------------------------------------
  int tiles_all;
  if (p.seqs) {
    if (warp == 0) est_line<true>(p, TT, lane, cum);
    __syncthreads();
    tiles_all = cum[p.batch];
  } else {
    tiles_all = est_tiles(len0, TT);
  }
  // The group is divided by the length, not by its upper bound: a short sequence in a large cache like one in a small cache (28
  // query heads over 4, 3K tokens in a cache of 128K: 15.8 us a layer, 20.0 with the division for 128K).
  const int q_part = GROUPED ? item_query_heads(tiles_all * (p.H / HP), q_group, p.chip_warps) : 1;
  const int q_split = GROUPED ? (q_group + q_part - 1) / q_part : 1;
  const int pieces = p.H / HP * q_split;
  // One sequence, no grouped queries: blockIdx.x is the piece, blockIdx.y an equal part of its tiles (or, where the grid's rows are not the
  // pieces, an even cut of the line).
  const bool grid_of_pieces = !GROUPED && !p.seqs && static_cast<int>(gridDim.x) == pieces;
  // Several sequences: columns of a block per piece, which share the line of one piece's tiles.
  int pos = 0, line_end = 1, column_piece = -1;
  if (!grid_of_pieces) {
    const int total = tiles_all * pieces;   // (below 2^31: checked on the host)
    if (total == 0) {   // (lengths that are all zero: the kernel behind must not overtake the one in front)
      grid_dependency_wait();
      return;
    }
    ItemShare work;
    const int columns = p.seqs ? item_blocks_per_piece(tiles_all, pieces, q_part, gridDim.x) : 0;
    if (columns > 0) {
      const int column = blockIdx.x / pieces, alike = item_columns_alike(tiles_all, cum[p.batch + 1], p.batch, columns);
      column_piece = blockIdx.x - column * pieces;
      if (column >= columns) work = ItemShare{0, 0};
      else if (alike > 0) work = item_share_alike(cum[p.batch + 1], p.batch, alike, column);
      else if (item_columns_apart(tiles_all, cum[p.batch + 1], p.batch, q_part, columns))
        work = item_share_apart(cum, p.batch, 1, columns, column);
      else work = item_share_even(tiles_all, columns, column);
    } else if (GROUPED && !p.seqs) {
      work = item_share_one(tiles_all, pieces, q_part, gridDim.x, blockIdx.x);
    } else {
      work = item_share_even(total, gridDim.x, blockIdx.x);
    }
    pos = work.pos;
    line_end = work.end;
  }
  bool waited = false;

  while (pos < line_end) {
    // ---- this block's next segment: tiles [first, end) of a piece of a sequence ----------------------------------------
    int s = 0, n = len0, piece, first, end, rest;   // (rest: tiles of the block from here on)
    const uint4* codes = p.codes;
    const int32_t* table = p.page_table;
    if (grid_of_pieces) {
      const int share = (tiles_all + gridDim.y - 1) / gridDim.y;
      piece = blockIdx.x;
      first = blockIdx.y * share;
      end = min(tiles_all, first + share);
      rest = end - first;
      pos = line_end;
      if (first >= end) {
        if (tiles_all == 0) grid_dependency_wait();
        return;
      }
    } else {
      int tiles = tiles_all, at = pos;
      if (p.seqs) {
        const int line_pieces = column_piece >= 0 ? 1 : pieces;
        int lo = 0, hi = p.batch - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (cum[mid] * line_pieces <= pos) lo = mid; else hi = mid - 1;
        }
        s = lo;
        tiles = cum[s + 1] - cum[s];
        at = pos - cum[s] * line_pieces;
        n = __ldg(p.seq_len_dev + s) - 1;
        codes = static_cast<const uint4*>(p.seqs[s].code_data);
        table = p.seqs[s].code_table;
      }
      piece = column_piece >= 0 ? column_piece : at / tiles;
      first = column_piece >= 0 ? at : at - piece * tiles;
      rest = line_end - pos;
      end = min(tiles, first + rest);
      pos += end - first;
    }
    const int head0 = (GROUPED ? piece / q_split : piece) * HP;                   // first cache head
    const int part0 = GROUPED ? (piece - head0 / HP * q_split) * q_part : 0;       // first query head of each of them
    const int heads = GROUPED ? min(q_part, q_group - part0) : 1;                  // query heads of each

    // ---- copies -----------------------------------------------------------------------------------------------
    // the page numbers of an item's tokens (lane = token of each group of 32) are fetched one item ahead of its copies
    auto fetch_entries = [&](int tile, int (&entry)[kGroups]) {
#pragma unroll
      for (int k = 0; k < kGroups; ++k) {
        const unsigned t = static_cast<unsigned>(min(tile * TT + k * 32 + lane, max(n - 1, 0)));   // (absent tokens: the last one's codes)
        entry[k] = __ldg(table + (p.ps_shift >= 0 ? t >> p.ps_shift : t / static_cast<unsigned>(p.page_size)));
      }
    };
    const int64_t stride = 2 * p.H;
    const uint4* base = codes + head0 * 2 + (lane & (CPR - 1));
    auto request = [&](int tile, const int (&entry)[kGroups], uint4* slot) {
      int tok[kGroups];
#pragma unroll
      for (int k = 0; k < kGroups; ++k) {
        const unsigned t = static_cast<unsigned>(min(tile * TT + k * 32 + lane, max(n - 1, 0))), ps = static_cast<unsigned>(p.page_size);
        tok[k] = entry[k] * p.page_size + static_cast<int>(p.ps_shift >= 0 ? t & (ps - 1) : t % ps);
      }
      constexpr int RPI = 32 / CPR;   // tokens per copy instruction
      const int c = lane & (CPR - 1), r0 = lane / CPR;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * RPI + r0;   // r / 32 == i * RPI / 32
        const int slot_of = __shfl_sync(0xffffffffu, tok[i * RPI / 32], r & 31);
        const int f = HP == 4 ? (r & 7) : HP == 2 ? ((r >> 1) & 3) : ((r >> 2) & 1);
        cp_async_16(slot + r * CPR + (c ^ f), base + slot_of * stride);
      }
    };
    // (the page numbers of the first items are on their way together)
    int entry[kGroups], first_entry[kItemMaxSlots][kGroups];
#pragma unroll
    for (int i = 0; i < kItemMaxSlots; ++i)
      if (i < slots && scanning && first + warp + i * kItemWarps < end) fetch_entries(first + warp + i * kItemWarps, first_entry[i]);
    int next = first + warp + slots * kItemWarps;   // the item to be requested next
    if (scanning && next < end) fetch_entries(next, entry);
    // (the new token sits at position n = tokens before it)
    if (cs_here) {
      sh.cs[cs_pair] = rope_cos_sin_at(cs_freq, static_cast<float>(n));
      if (!GROUPED) asm volatile("bar.arrive 1, 96;" ::: "memory");   // (these two warps and the last one)
    }
#pragma unroll
    for (int i = 0; i < kItemMaxSlots; ++i) {
      if (i < slots) {
        if (scanning && first + warp + i * kItemWarps < end) request(first + warp + i * kItemWarps, first_entry[i], ring + i * (kItemBytes / 16));
        cp_async_commit();
      }
    }

    const int64_t seq_row = static_cast<int64_t>(s) * rows;
    // (r / q_part: both are at most 16)
    const unsigned per_part = GROUPED ? 65536u / q_part + 1u : 0u;
    auto head_of = [&](int r) { return GROUPED ? static_cast<int>(r * per_part >> 16) : r; };
    auto query_row = [&](int r) {   // row of the sequence that the segment's row r stands for
      const int h = head_of(r);
      return GROUPED ? (head0 + h) * q_group + part0 + r - h * q_part : head0 + r;
    };
    auto absent = [&](int r) { return GROUPED && r - head_of(r) * q_part >= heads; };   // (of a short last part)
    const int my_rows = HP * q_part;
    // The block with the piece's first tile appends the new token's rows of the piece's cache heads.
    const bool appends = APPEND && first == 0 && part0 == 0;
    const int tab_rows = GROUPED ? my_rows : seg_rows;   // rows of a count table
    const unsigned l8 = lane & 7;
    const bool scaled = p.ap.rp.inv_freq != nullptr;
    const int slice_tokens = p.hist ? 8 * sa_granules_per_block(max(n, 1), p.hist_cl) : 1;
    const int slice0 = p.hist ? first * TT / slice_tokens : 0;
    const bool tables = p.hist && (GROUPED || rest * TT > kItemDirect || n > kItemDirectRow);
    const int used = tables ? min(kTables, (end * TT - 1) / slice_tokens - slice0 + 1) : 0;   // count tables of this segment
    constexpr int kPairs = (HP + 1) / 2;
    uint4 v_row[kPairs];   // (GROUPED, last warp, appending: the new V rows, one in each half)
    if (GROUPED && appends && !scanning && lane == 0) {   // (the page tables are final as well)
      const StepAppend& ap = p.ap;
      const int ps = ap.tgt.page_size;
      const int32_t* kv_table = p.seqs ? p.seqs[s].kv_table : ap.tgt.kv_table;
      const int32_t* code_table = p.seqs ? p.seqs[s].code_table : ap.tgt.code_table;
      int kv_last_page = ap.kv_last_page, kv_entry = ap.kv_entry, code_last_page = ap.code_last_page, code_entry = ap.code_entry;
      if (p.seq_len_dev) {
        kv_last_page = code_last_page = n / ps;
        kv_entry = code_entry = n - kv_last_page * ps;
      }
      const int64_t kv_page = __ldg(kv_table + kv_last_page), code_page = __ldg(code_table + code_last_page);
      sh.kv_row = (kv_page * 2 * ps + kv_entry) * p.H + head0;
      sh.code_row = (code_page * ps + code_entry) * p.H + head0;
    }

    // ---- the sequence's query: codes, planes; the new token's rows ---------------------------------------------
    if (!waited) {
      grid_dependency_wait();   // q, k, v or the query codes are the preceding kernel's output
      grid_launch_dependents();
      waited = true;
    }
    if (scanning) {
      for (int i = tid; i < used * tab_rows * (kItemCountWords / 4); i += kItemWarps * 32) reinterpret_cast<uint4*>(counts)[i] = make_uint4(0, 0, 0, 0);
    } else if (APPEND && GROUPED) {
      const int c = lane & 15;   // (a half-warp per row)
#pragma unroll 2
      for (int r = lane >> 4; r < my_rows; r += 2)
        if (!absent(r)) cp_async_16(q_rows + r * 16 + c, static_cast<const T*>(p.ap.q) + (seq_row + query_row(r)) * kHeadDim + c * 8);
      if (appends) {
#pragma unroll
        for (int i = 0; i < kPairs; ++i) {
          const int h = 2 * i + (lane >> 4);
          if (h >= HP) continue;
          cp_async_16(q_rows + (my_rows + h) * 16 + c, static_cast<const T*>(p.ap.k) + (static_cast<int64_t>(s) * p.H + head0 + h) * kHeadDim + c * 8);
          v_row[i] = ld_16(static_cast<const T*>(p.ap.v) + (static_cast<int64_t>(s) * p.H + head0 + h) * kHeadDim + c * 8);
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
    } else if (APPEND) {
      // eight lanes per row, all (at most four) at a time
      const int row = lane >> 3;
      const int64_t code_row = seq_row + query_row(row < HP ? row : 0);
      const T* src = static_cast<const T*>(p.ap.q) + code_row * kHeadDim + l8 * 8;
      const uint4 q0 = ld_16(src), q1 = ld_16(src + kHeadDim / 2);
      if (p.ap.rope_on) asm volatile("bar.sync 1, 96;" ::: "memory");   // (the rotation is there)
      float2 x[8];
      unpack_pairs<T>(q0, q1, x);
      if (p.ap.rope_on) rope_pairs<T>(x, l8, sh.cs, scaled, p.ap.rp.mscale);
      const uint32_t w = code_pairs<T>(x, l8, p.ap.scale, PairThresholds<T>(p.ap.th));
      // 32-bit words l8 / 2 and 4 + l8 / 2 of the code in the even lanes, and words i and 2 + i, i = l8 / 4, of a plane in every fourth
      const uint32_t next = __shfl_down_sync(0xffffffffu, w, 1);
      const uint32_t c0 = __byte_perm(w, next, 0x5410), c1 = __byte_perm(w, next, 0x7632);
      const uint32_t d0 = __shfl_down_sync(0xffffffffu, c0, 2), d1 = __shfl_down_sync(0xffffffffu, c1, 2);
      if (row < HP) {
        if (first == 0) {   // (the codes may start on any 16-bit word)
          uint16_t* dst = p.ap.q_code_out + code_row * kCodeWords + l8;
          dst[0] = static_cast<uint16_t>(w);
          dst[8] = static_cast<uint16_t>(w >> 16);
        }
        if (!(l8 & 3)) {
          const uint32_t hi0 = plane_hi(c0, d0), lo0 = plane_lo(c0, d0), hi1 = plane_hi(c1, d1), lo1 = plane_lo(c1, d1);
          uint32_t* qp = reinterpret_cast<uint32_t*>(planes + row) + (l8 >> 2);
          qp[0] = hi0;
          qp[2] = hi1;
          qp[4] = lo0;
          qp[6] = lo1;
          qp[8] = hi0 ^ lo0;
          qp[10] = hi1 ^ lo1;
        }
      }
    } else {
      for (int r = lane; r < my_rows; r += 32) {
        const uint4* code = p.q_code + (seq_row + query_row(r)) * 2;
        if (!absent(r)) planes[r] = query_planes(ld_16(code), ld_16(code + 1));
      }
    }
    __syncthreads();
    if (APPEND && GROUPED) {   // a warp per row
#pragma unroll 1
      for (int r = warp; r < my_rows + (appends ? HP : 0); r += kItemWarps + 1) {
        const int h = r - my_rows;   // (a new key row)
        if (h < 0 && absent(r)) continue;
        uint2 raw = reinterpret_cast<const uint2*>(q_rows)[r * 32 + lane];
        float x[4];
        unpack4<T>(raw, x);
        if (p.ap.rope_on) {
          rope_warp<T>(x, lane, sh.cs, scaled, p.ap.rp.mscale);
          raw = make_uint2(Elem<T>::from_f2(x[0], x[1]), Elem<T>::from_f2(x[2], x[3]));
        }
        const uint32_t w = code_word_warp<T>(x, lane, p.ap.scale, PairThresholds<T>(p.ap.th));
        if (h < 0) {   // planes and, by the piece's first block, the code
          const uint32_t next = __shfl_down_sync(0xffffffffu, w, 4);
          if (first == 0 && (lane & 3) == 0) reinterpret_cast<uint32_t*>(p.ap.q_code_out)[(seq_row + query_row(r)) * (kCodeWords / 2) + (lane >> 2)] = w;
          if ((lane & 7) == 0) {   // (words 2i and 2i + 1 make word i of a plane)
            const uint32_t hi = plane_hi(w, next), lo = plane_lo(w, next);
            uint32_t* qp = reinterpret_cast<uint32_t*>(planes + r) + (lane >> 3);
            qp[0] = hi;
            qp[4] = lo;
            qp[8] = hi ^ lo;
          }
        } else {
          if (p.ap.rope_on) (static_cast<uint2*>(p.ap.k) + (static_cast<int64_t>(s) * p.H + head0 + h) * (kHeadDim / 4))[lane] = raw;
          void* kv_data = p.seqs ? p.seqs[s].kv_data : p.ap.tgt.kv_data;
          void* code_data = p.seqs ? p.seqs[s].code_data : p.ap.tgt.code_data;
          (static_cast<uint2*>(kv_data) + (sh.kv_row + h) * (kHeadDim / 4))[lane] = raw;
          if ((lane & 3) == 0) (static_cast<uint32_t*>(code_data) + (sh.code_row + h) * (kCodeWords / 2))[lane >> 2] = w;
        }
      }
      __syncthreads();
    }
    // (planes and zeroed counts are visible)
    if (GROUPED && appends && !scanning) {
      uint4* kv_data = static_cast<uint4*>(p.seqs ? p.seqs[s].kv_data : p.ap.tgt.kv_data);
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        const int h = 2 * i + (lane >> 4);
        if (h < HP) kv_data[(sh.kv_row + static_cast<int64_t>(p.page_size) * p.H + h) * 16 + (lane & 15)] = v_row[i];
      }
    }

    // ---- the new token's rows of the piece's cache heads, in the block that has the piece's first tile ----------------------
    if (!GROUPED && appends && !scanning) {
      const StepAppend& ap = p.ap;
      const bool live = (lane >> 3) < HP;
      const int h = head0 + (live ? lane >> 3 : 0);
      constexpr int kHalf = kHeadDim / 2;
      const int64_t in_off = (static_cast<int64_t>(s) * p.H + h) * kHeadDim + l8 * 8;
      T* ksrc = static_cast<T*>(ap.k) + in_off;
      const T* vsrc = static_cast<const T*>(ap.v) + in_off;
      uint4 k0 = ld_16(ksrc), k1 = ld_16(ksrc + kHalf);
      const uint4 v0 = ld_16(vsrc), v1 = ld_16(vsrc + kHalf);
      PagedTarget tgt = ap.tgt;
      if (p.seqs) {
        tgt.kv_data = p.seqs[s].kv_data;
        tgt.kv_table = p.seqs[s].kv_table;
        tgt.code_data = static_cast<uint16_t*>(p.seqs[s].code_data);
        tgt.code_table = p.seqs[s].code_table;
      }
      const int ps = tgt.page_size;
      int kv_last_page = ap.kv_last_page, kv_entry = ap.kv_entry, code_last_page = ap.code_last_page, code_entry = ap.code_entry;
      if (p.seq_len_dev) {
        kv_last_page = code_last_page = n / ps;
        kv_entry = code_entry = n - kv_last_page * ps;
      }
      const int64_t kv_page = __ldg(tgt.kv_table + kv_last_page), code_page = __ldg(tgt.code_table + code_last_page);
      float2 x[8];
      unpack_pairs<T>(k0, k1, x);
      if (ap.rope_on) {
        rope_pairs<T>(x, l8, sh.cs, scaled, ap.rp.mscale);
        pack_pairs<T>(x, &k0, &k1);
        __syncwarp();   // (lanes without a row of their own have read the first one)
        if (live) {
          st_16(ksrc, k0);
          st_16(ksrc + kHalf, k1);
        }
      }
      const uint32_t w = code_pairs<T>(x, l8, ap.scale, PairThresholds<T>(ap.th));
      if (live) {
        T* dst = static_cast<T*>(tgt.kv_data) + ((kv_page * 2 * ps + kv_entry) * p.H + h) * kHeadDim + l8 * 8;
        st_16(dst, k0);
        st_16(dst + kHalf, k1);
        dst += static_cast<int64_t>(ps) * p.H * kHeadDim;
        st_16(dst, v0);
        st_16(dst + kHalf, v1);
        uint16_t* code = tgt.code_data + ((code_page * ps + code_entry) * p.H + h) * kCodeWords + l8;
        code[0] = static_cast<uint16_t>(w);
        code[8] = static_cast<uint16_t>(w >> 16);
      }
    }

    // ---- scan -----------------------------------------------------------------------------------------------------
    // the counts in shared memory are those of the first `used` slices that the segment touches; anything behind them is counted
    // in global memory one by one
    uint32_t* hist = p.hist ? p.hist + seq_row * kSaScratchWordsPerHead : nullptr;
    uint16_t* out = static_cast<uint16_t*>(p.out) + (seq_row + (GROUPED ? 0 : head0)) * p.out_stride;
    auto to_out = [&](unsigned d) { return !APPEND && p.out_half ? __half_as_ushort(__uint2half_rn(d)) : static_cast<uint16_t>(d); };   // (exact: d <= 384)
    const int f = HP == 4 ? (lane & 7) : HP == 2 ? ((lane >> 1) & 3) : ((lane >> 2) & 1);
    uint32_t* tab = counts;   // the table of the present tokens, the token behind its slice, the tables that are left
    int use = 0, left = tables ? kTables : 0, tab_end = (slice0 + 1) * slice_tokens;
    for (int tile = scanning ? first + warp : end; tile < end; tile += kItemWarps) {
      if (slots == 3) cp_async_wait<2>(); else if (slots == 2) cp_async_wait<1>(); else cp_async_wait<0>();
      __syncwarp();
      const uint4* lrow = ring + use * (kItemBytes / 16) + lane * CPR;
#pragma unroll (GROUPED ? 1 : kGroups)
      for (int k = 0; k < kGroups; ++k) {
        const int t0 = tile * TT + k * 32, t = t0 + lane;
        for (; left > 0 && t0 >= tab_end; --left) {   // (a group never straddles two slices)
          tab += tab_rows * kItemCountWords;
          tab_end += slice_tokens;
        }
        const bool here = left > 0;
        // up to four rows' distances: segment rows r .., output rows `row` ..
        auto emit = [&](int r, int row, const unsigned* d, int many) {
          if (t >= n) return;
          uint16_t* o = (GROUPED ? out + row * p.out_stride : out) + t;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (u < many) o[u * p.out_stride] = to_out(d[u]);
          if (here) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (u < many) atomicAdd(tab + (r + u) * kItemCountWords + d[u], 1u);
          } else if (p.hist) {
            const int slice = t0 / slice_tokens;
#pragma unroll 1
            for (int u = 0; u < many; ++u) hist_count(hist, row + u, slice, u == 0 ? d[0] : u == 1 ? d[1] : u == 2 ? d[2] : d[3]);
          }
        };
        if (!GROUPED) {
          unsigned d[4];
#pragma unroll
          for (int hh = 0; hh < HP; ++hh)
            d[hh] = code_distance<METRIC>(code_planes(lrow[k * 32 * CPR + ((2 * hh) ^ f)], lrow[k * 32 * CPR + ((2 * hh + 1) ^ f)]), planes[hh]);
          emit(0, head0, d, HP);
        } else {
          // Grouped queries: a code is read once for the piece's query heads of its cache head.  The loops over groups and heads stay
          // rolled and the last one to three heads come one by one: with few items a warp passes here once, and an unrolled body
          // costs the fetch of its instructions (the step of 28 query heads over 4, 3K tokens: 15.8 us a layer unrolled, 12.3 rolled; 32 over 8,
          // 3K 16.8 / 13.2; 64 sequences x 2K x 28 over 4 103 / 81).
#pragma unroll 1
          for (int hh = 0; hh < HP; ++hh) {
            const CodePlanes key = code_planes(lrow[k * 32 * CPR + ((2 * hh) ^ f)], lrow[k * 32 * CPR + ((2 * hh + 1) ^ f)]);
            // (four distances, then their stores and counts: the counts keep the compiler from moving reads of shared memory across them)
            auto four = [&](int g, int many) {
              const QPlanes* qp = planes + hh * q_part + g;
              unsigned d[4] = {0, 0, 0, 0};
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (u < many) d[u] = code_distance<METRIC>(key, qp[u]);
              emit(hh * q_part + g, (head0 + hh) * q_group + part0 + g, d, many);
            };
            int g = 0;
            for (; g + 4 <= heads; g += 4) four(g, 4);
            for (; g < heads; ++g) four(g, 1);
          }
        }
      }
      __syncwarp();   // the slot may be filled again
      if (next < end) {
        request(next, entry, ring + use * (kItemBytes / 16));
        next += kItemWarps;
        if (next < end) fetch_entries(next, entry);
      }
      cp_async_commit();
      if (++use == slots) use = 0;
    }
    cp_async_wait<0>();
    if (tables || pos < line_end) __syncthreads();
    if (tables) {
      for (int i = tid; i < used * tab_rows * (kItemCountWords / 4); i += kItemThreads) {
        const uint4 c4 = reinterpret_cast<const uint4*>(counts)[i];
        if (c4.x | c4.y | c4.z | c4.w) {
          const int tr = i / (kItemCountWords / 4), u = tr / tab_rows, r = tr - u * tab_rows;
          uint32_t* dst = hist + static_cast<size_t>(query_row(r)) * kSaScratchWordsPerHead + (slice0 + u) * kSaBins + (i - tr * (kItemCountWords / 4)) * 4;
          if (c4.x) atomicAdd(dst, c4.x);
          if (c4.y) atomicAdd(dst + 1, c4.y);
          if (c4.z) atomicAdd(dst + 2, c4.z);
          if (c4.w) atomicAdd(dst + 3, c4.w);
        }
      }
      if (pos < line_end) __syncthreads();   // the counts may be cleared for the next segment
    }
  }
}

}  // namespace adamas
