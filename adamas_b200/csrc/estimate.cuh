// Stage 2 of the decode path: distance between the query's 2-bit code and every cached key code, and, in a decode
// step, the append of the new token (stage 1) in the same launch.
//
// The code of (token t, head h) is 32 bytes at ((page*page_size + entry)*H + h)*32 in the code cache.  Two kernels:
//
// estimate_kernel / estimate_append_kernel (here): 16, 32 or 64 heads without grouped queries, for short rows with counts, alone, in small batches
//   and in large ones, and, 32 and 64 heads, for all without (estimate_by_tiles).  Persistent, two blocks per SM; the blocks of a sequence walk its tiles of kEstTile = 32 consecutive tokens round-robin.
//   (Contiguous runs of tiles per block measured slower: 7.5 us against 6.8 for 32K tokens x 32 heads.)
//   * Two producer warps issue one bulk (TMA) copy per token (the token's H codes, H*32 contiguous bytes) into a
//     kEstStages-deep shared-memory ring; rows are padded by 16 bytes.  A "full" mbarrier per slot counts the bytes, an
//     "empty" mbarrier per slot collects one arrival per consumer warp before the slot is refilled.
//   * 16 consumer warps: lane l owns token l of the tile, a warp owns H / 16 heads whose query planes it keeps in
//     registers.  A lane reads the two 16-byte halves of a code (the row padding makes the 32 lanes hit 32 different bank
//     groups), reduces them in registers and stores the distance: the 32 lanes of a warp write 32 consecutive tokens
//     of one head, so the [H, n] output needs no transpose, no shuffle and no block barrier.  Histogram counts, where
//     they are wanted, are one L2 atomic per distance.
//
// estimate_items_kernel (estimate_items.cuh): everything else.
//
// All mbarrier waits are bounded; one that runs out sets a device error flag and the kernel finishes (with wrong
// results, which the flag reports).  The distance arithmetic on packed 2-bit codes is described at code_distance().
#pragma once
#include "common.cuh"
#include "hadamard_append.cuh"
#include "item_split.h"
#include "select_attend.cuh"

namespace adamas {

constexpr int kEstTile = 32;      // tokens per tile
constexpr int kEstConsumerWarps = 16;
constexpr int kEstProducerWarps = 2;   // see est_produce
constexpr int kEstThreads = (kEstConsumerWarps + kEstProducerWarps) * 32;
constexpr int kEstStages = 3;     // ring depth (tiles in flight per block: kEstStages - 1)
constexpr int kEstMaxBatch = 1024;

// A code's 128 dimensions as two bit planes (hi: value bit 1, lo: value bit 0) of four words: word i holds the dimensions of code words
// 2i (at the odd bits) and 2i + 1 (at the even bits).
struct CodePlanes {
  uint32_t hi[4], lo[4];
};
// A query row's planes and their difference.
struct __align__(16) QPlanes {
  uint4 hi, lo, d;   // d = hi ^ lo
};

__device__ __forceinline__ uint32_t odd_even(uint32_t a, uint32_t b) {  // the odd bits of a, the even bits of b
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(a), "r"(b), "r"(0xAAAAAAAAu));
  return d;
}
__device__ __forceinline__ uint32_t plane_hi(uint32_t w0, uint32_t w1) { return odd_even(w0, w1 >> 1); }
__device__ __forceinline__ uint32_t plane_lo(uint32_t w0, uint32_t w1) { return odd_even(w0 << 1, w1); }
__device__ __forceinline__ CodePlanes code_planes(uint4 a, uint4 b) {   // words 0 .. 3, 4 .. 7
  return CodePlanes{{plane_hi(a.x, a.y), plane_hi(a.z, a.w), plane_hi(b.x, b.y), plane_hi(b.z, b.w)},
                    {plane_lo(a.x, a.y), plane_lo(a.z, a.w), plane_lo(b.x, b.y), plane_lo(b.z, b.w)}};
}
__device__ __forceinline__ QPlanes query_planes(uint4 a, uint4 b) {
  const CodePlanes c = code_planes(a, b);
  return QPlanes{make_uint4(c.hi[0], c.hi[1], c.hi[2], c.hi[3]), make_uint4(c.lo[0], c.lo[1], c.lo[2], c.lo[3]),
                 make_uint4(c.hi[0] ^ c.lo[0], c.hi[1] ^ c.lo[1], c.hi[2] ^ c.lo[2], c.hi[3] ^ c.lo[3])};
}

// Distance of two codes.  With x = k ^ q per dimension (x1, x0):  |k - q| = x0 + 2 * (x1 & ~(x0 & (q1 ^ q0)))  (the bracket clears
// x1 for the code pairs {1, 2}); the XOR metric of the reference's CUDA kernel is the same without the bracket.  So four words
// count once and four count twice; three full adders leave five of them to count.
// Bound: logic instructions at half rate and population counts at an eighth of the issue rate.  Packed words, with x and y = x & ~... of
// whole code words and 12 counts, took 78 cycles per 32 distances and scheduler, this form 57 (with 8 counts and no adders 58; of which the
// query rows of a group share the key's planes).  The step, us a layer: 32 heads, 32K 20.2 -> 19.9; 32 query heads over 8, 30K 22.5 -> 21.1;
// 40 heads, 12K 15.8 -> 15.5.
template <int METRIC>
__device__ __forceinline__ unsigned code_distance(const CodePlanes& k, const QPlanes& q) {
  const uint32_t qh[4] = {q.hi.x, q.hi.y, q.hi.z, q.hi.w}, ql[4] = {q.lo.x, q.lo.y, q.lo.z, q.lo.w}, qd[4] = {q.d.x, q.d.y, q.d.z, q.d.w};
  uint32_t one[4], two[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    one[i] = k.lo[i] ^ ql[i];
    two[i] = k.hi[i] ^ qh[i];
    if (METRIC == 0) two[i] &= ~(one[i] & qd[i]);
  }
  auto sum = [](uint32_t a, uint32_t b, uint32_t c) { return a ^ b ^ c; };
  auto carry = [](uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (a & c) | (b & c); };
  const uint32_t s1 = sum(one[0], one[1], one[2]), c1 = carry(one[0], one[1], one[2]);
  const uint32_t s2 = sum(two[0], two[1], two[2]), c2 = carry(two[0], two[1], two[2]);
  const uint32_t s3 = sum(s2, two[3], c1), c3 = carry(s2, two[3], c1);
  return (__popc(s1) + __popc(one[3])) + 2 * __popc(s3) + 4 * (__popc(c2) + __popc(c3));
}

template <typename OutT>
__device__ __forceinline__ OutT dist_to_out(unsigned d);
template <>
__device__ __forceinline__ uint16_t dist_to_out<uint16_t>(unsigned d) {
  return static_cast<uint16_t>(d);
}
template <>
__device__ __forceinline__ __half dist_to_out<__half>(unsigned d) {
  return __uint2half_rn(d);  // exact: d <= 384
}

// The decode append inside the estimate.  Every block codes all query heads of the sequences it works on by itself
// (the rows come from L2), so no block waits for another.  The new token's K and V rows, the key's code and the query
// codes are stored by one block each (estimate_append_kernel) or by the blocks that start a piece of its heads
// (estimate_items_kernel); none of this is read by the scan, which leaves the newest token out, and the kernel after
// this one finds all of it complete.
// rope_on: q and k arrive un-rotated.  The position's 64 (cos, sin) pairs are formed once per block and sequence, the
// query rows are rotated in registers before they are coded, the appending block stores the rotated key into the cache
// and back into the caller's k.  The caller's q is NOT rotated here (other blocks are still reading it): the
// select+attend launch that follows rotates it the same way for its own use and writes it back.
struct StepAppend {
  const void* q;           // [rows, 128]; null: no append, the query codes are given
  void* k;                 // [H,128] per sequence
  const void* v;
  uint16_t* q_code_out;    // [rows, 16]
  PagedTarget tgt;
  int kv_last_page, kv_entry, code_last_page, code_entry;   // slot of the new token (host lengths)
  float scale;
  Thresholds th;
  int rope_on;
  RopeParams rp;
};

struct EstimateParams {
  const uint4* codes;
  const int32_t* page_table;
  const uint4* q_code;   // the query codes (no append)
  void* out;             // [rows, out_stride] u16 or fp16 distances
  int64_t out_stride;
  int out_half;
  int n_tokens;     // distances per row (host lengths)
  int H;            // heads of the code cache
  int chip_warps;   // estimate_items_kernel: scanning warps that are resident at once on the device
  int q_group;      // query heads per cache head: out, hist, q and q_code have H * q_group rows per sequence
  int page_size;
  int ps_shift;     // log2(page_size) or -1
  int batch;
  // optional: the sequence length (tokens, the newest included) lives on the device; n_tokens is then *seq_len_dev - 1.
  // Read before the kernel's dependency resolves: the value must be final before the kernel that precedes this
  // one in the stream starts.
  const int32_t* seq_len_dev;
  // optional: per-slice histograms of the distance rows for select_attend, in the histogram rows of its
  // scratch table ([rows][kSaScratchWordsPerHead] u32, rows zero on entry); slice = token / (8 * sa_granules_per_block(n_tokens, hist_cl))
  uint32_t* hist;
  int hist_cl;
  // optional (needs seq_len_dev): a batch of sequences.  Everything on the query side has one row per (sequence, query
  // head); codes, page table and length are the sequence's.
  const SeqDesc* seqs;
  StepAppend ap;
};

// Tiles of `tile_tokens` tokens of the batch's sequences in front of each one -> cum[0 .. batch], and, MOST, the most that one has ->
// cum[batch + 1]; one warp.
template <bool MOST = false>
__device__ __forceinline__ void est_line(const EstimateParams& p, int tile_tokens, int lane, int* cum) {
  int base = 0, most = 0;
  for (int s0 = 0; s0 < p.batch; s0 += 32) {
    int v = s0 + lane < p.batch ? est_tiles(__ldg(p.seq_len_dev + s0 + lane) - 1, tile_tokens) : 0;
    most = max(most, v);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (s0 + lane < p.batch) cum[s0 + lane + 1] = base + v;
    base += __shfl_sync(0xffffffffu, v, 31);
  }
  if (lane == 0) cum[0] = 0;
  if (MOST) {
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) cum[p.batch + 1] = most;
  }
}

// What a block works on: tiles rank, rank + blocks, ... of one sequence; nothing to scan where rank == blocks.
struct EstGeom {
  int n_tokens;
  int num_tiles;
  int slice_tokens;   // tokens per histogram slice (a multiple of 32)
  const uint4* codes;
  const int32_t* page_table;
  int seq;
  int rank, blocks;
  bool appends;       // stores the sequence's new token
  int row0;           // first row of this sequence in q_code, out and hist
};
// Called by all threads of the block.  A batch's sequences get one block each and the other blocks in proportion to their
// tiles (32 sequences of 4-8K tokens x 32 heads with equal shares of the blocks: 42 us, the longest sequence's share;
// in proportion 35).
__device__ __forceinline__ EstGeom est_geom(const EstimateParams& p, int* cum) {
  EstGeom g;
  g.codes = p.codes;
  g.page_table = p.page_table;
  g.seq = 0;
  g.rank = blockIdx.x;
  g.blocks = gridDim.x;
  g.n_tokens = p.n_tokens;
  if (p.seqs) {   // (the table of sequences is set up once, long before this launch)
    if (threadIdx.x < 32) est_line(p, kEstTile, threadIdx.x, cum);
    __syncthreads();
    const int64_t total = max(cum[p.batch], 1), spare = static_cast<int>(gridDim.x) - p.batch;
    auto first_block = [&](int s) { return s + static_cast<int>(cum[s] * spare / total); };
    int lo = 0, hi = p.batch - 1;
    while (lo < hi) {   // the last sequence that starts at or before this block
      const int mid = (lo + hi + 1) >> 1;
      if (first_block(mid) <= g.rank) lo = mid; else hi = mid - 1;
    }
    g.seq = lo;
    const int f = first_block(lo);
    g.rank -= f;
    g.blocks = first_block(lo + 1) - f;
    g.n_tokens = __ldg(p.seq_len_dev + lo) - 1;
    g.codes = static_cast<const uint4*>(p.seqs[lo].code_data);
    g.page_table = p.seqs[lo].code_table;
  } else if (p.seq_len_dev) {
    g.n_tokens = __ldg(p.seq_len_dev) - 1;
  }
  g.row0 = g.seq * p.H;
  g.num_tiles = (g.n_tokens + kEstTile - 1) / kEstTile;
  // The sequence's last block appends.  It scans nothing where that gives no other block a tile more: with tiles to scan
  // as well it finished 1 to 2 us after all the others (one sequence, 4K to 128K tokens x 32 heads).  Where every block
  // has many tiles it scans its own after the append (appending after them: 80.0 us a layer for 8 x 32K, before 79.5).
  g.appends = g.rank == g.blocks - 1;
  if (p.ap.q && g.blocks > 1 && (g.num_tiles + g.blocks - 1) / g.blocks == (g.num_tiles + g.blocks - 2) / (g.blocks - 1)) --g.blocks;
  g.slice_tokens = p.hist ? 8 * sa_granules_per_block(g.n_tokens, p.hist_cl) : 1;
  return g;
}

__device__ __forceinline__ void hist_count(uint32_t* hist, int head, int slice, unsigned d) {
  uint32_t* a = hist + static_cast<size_t>(head) * kSaScratchWordsPerHead + (slice << 9) + d;
  asm volatile("red.global.add.u32 [%0], 1;" ::"l"(a) : "memory");
}

// ---- the two halves of the copy pipeline, shared by the kernels below --------------------------------
// Geometry of the ring for H heads: a token's codes are 2H 16-byte chunks, padded by one chunk so
// that lanes reading one chunk position of 32 consecutive tokens hit 32 different bank groups.
struct EstRing {
  uint4* base;
  uint64_t* full_bar;
  uint64_t* empty_bar;
  int cpt;            // 16-byte chunks per token (2H)
  int row_chunks;     // padded row
  int stage_chunks;   // chunks per ring slot
};

__device__ __forceinline__ int est_tiles_of_block(const EstGeom& g) { return g.rank < g.blocks ? max(0, (g.num_tiles - g.rank + g.blocks - 1) / g.blocks) : 0; }

// Producer warps: one bulk copy per token (its H codes) into the padded ring slot.
// A bulk copy with a different address in every lane is issued lane after lane, about 45 ns each
// (measured: the 32 copies of a tile kept a single producer warp busy for 1.4 us, so that it needed
// over 4 us to ask for the first three tiles and the ring was never ahead of the consumers; the SM's
// copy unit itself takes a request every 2 ns).  So the copies of a tile are split over
// kEstProducerWarps warps: producer `pw` issues the tokens tl with (tl / 16) % kEstProducerWarps == pw,
// 16 lanes at a time.  Producer 0 also announces the tile's bytes on the "full" barrier; a copy of
// another producer that lands before that announcement only makes the barrier's byte count negative
// for a moment, which it allows.
__device__ __forceinline__ void est_token_slot(const EstimateParams& p, int t, int* lp, int* e) {
  if (p.ps_shift >= 0) {
    *lp = t >> p.ps_shift;
    *e = t & (p.page_size - 1);
  } else {
    *lp = t / p.page_size;
    *e = t - *lp * p.page_size;
  }
}

__device__ __forceinline__ void est_produce(const EstimateParams& p, const EstGeom& g, const EstRing& r, int my_tiles,
                                            int lane, int pw) {
  const unsigned token_bytes = static_cast<unsigned>(r.cpt) * 16u;
  // this lane's tokens of a tile: tl = first_tl, first_tl + 16 * kEstProducerWarps * 2, ... (lanes 0-15 and
  // 16-31 of a producer take alternate 16-token runs of its share)
  const int first_tl = ((lane >> 4) * kEstProducerWarps + pw) * 16 + (lane & 15);
  int slot = 0;
  unsigned parity = 0;   // parity of the previous use of the slot, for the empty barrier
  for (int j = 0; j < my_tiles; ++j) {
    const int tile0 = (g.rank + j * g.blocks) * kEstTile;
    const int tile_tokens = min(kEstTile, g.n_tokens - tile0);
    // the physical page of the first token does not depend on the slot: fetch it before waiting
    int64_t tok_first = 0;
    if (first_tl < tile_tokens) {
      int lp, e;
      est_token_slot(p, tile0 + first_tl, &lp, &e);
      tok_first = static_cast<int64_t>(__ldg(g.page_table + lp)) * p.page_size + e;
    }
    if (j >= kEstStages) {
      // every consumer warp has finished reading the tile that used this slot before
      if (!mbar_wait_bounded(&r.empty_bar[slot], parity, 1u << 20)) atomicOr(&g_adamas_error, kErrEstimateTimeout);
    }
    if (pw == 0 && lane == 0) mbar_arrive_expect_tx(&r.full_bar[slot], static_cast<unsigned>(tile_tokens) * token_bytes);
    __syncwarp();
    for (int tl = first_tl; tl < tile_tokens; tl += 32 * kEstProducerWarps) {
      int64_t tok = tok_first;
      if (tl != first_tl) {
        int lp, e;
        est_token_slot(p, tile0 + tl, &lp, &e);
        tok = static_cast<int64_t>(__ldg(g.page_table + lp)) * p.page_size + e;
      }
      bulk_copy_g2s(r.base + slot * r.stage_chunks + tl * r.row_chunks, g.codes + tok * r.cpt, token_bytes,
                    &r.full_bar[slot]);
    }
    if (++slot == kEstStages) {
      slot = 0;
      if (j >= kEstStages) parity ^= 1u;
    }
  }
}

// Consumer warp: lane = token of the tile; the warp covers heads warp*HPW .. (query planes in registers).
template <int METRIC, typename OutT, int HPW>
__device__ __forceinline__ void est_consume(const EstimateParams& p, const EstGeom& g, const EstRing& r, int my_tiles,
                                            int lane, int warp, const QPlanes (&qp)[HPW]) {
  OutT* out = static_cast<OutT*>(p.out) + static_cast<int64_t>(g.row0) * p.out_stride;   // this sequence's rows
  uint32_t* hist = p.hist ? p.hist + static_cast<size_t>(g.row0) * kSaScratchWordsPerHead : nullptr;
  int slot = 0;
  unsigned parity = 0;
  for (int j = 0; j < my_tiles; ++j) {
    const int tile0 = (g.rank + j * g.blocks) * kEstTile;
    const int tile_tokens = min(kEstTile, g.n_tokens - tile0);
    const int slice = p.hist ? tile0 / g.slice_tokens : 0;   // a 32-token group never straddles two slices
    // bounded wait for this tile's bytes; on failure flag the error and carry on (results are then
    // wrong, which the flag reports, but nothing spins forever)
    if (!mbar_wait_bounded(&r.full_bar[slot], parity, 1u << 20)) atomicOr(&g_adamas_error, kErrEstimateTimeout);
    const uint4* row = r.base + slot * r.stage_chunks + lane * r.row_chunks;
    OutT* o = out + tile0 + lane;
    unsigned d[HPW];
#pragma unroll
    for (int hh = 0; hh < HPW; ++hh) {
      const int h = warp * HPW + hh;
      d[hh] = code_distance<METRIC>(code_planes(row[2 * h], row[2 * h + 1]), qp[hh]);
    }
    if (lane < tile_tokens) {
#pragma unroll
      for (int hh = 0; hh < HPW; ++hh)
        o[static_cast<int64_t>(warp * HPW + hh) * p.out_stride] = dist_to_out<OutT>(d[hh]);
      if (p.hist) {
#pragma unroll
        for (int hh = 0; hh < HPW; ++hh) hist_count(hist, warp * HPW + hh, slice, d[hh]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&r.empty_bar[slot]);
    if (++slot == kEstStages) {
      slot = 0;
      parity ^= 1u;
    }
  }
}

__device__ __forceinline__ EstRing est_ring_init(uint4* smem, uint64_t* full_bar, uint64_t* empty_bar, int H,
                                                 int tid) {
  EstRing r;
  r.base = smem;
  r.full_bar = full_bar;
  r.empty_bar = empty_bar;
  r.cpt = 2 * H;
  r.row_chunks = r.cpt + 1;
  r.stage_chunks = kEstTile * r.row_chunks;
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kEstStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], kEstConsumerWarps);
    }
    mbar_fence_init();
  }
  return r;
}

// Dynamic shared memory: kEstStages * kEstTile * (2H + 1) * 16 bytes.  H == kEstConsumerWarps * HPW: warp w keeps the
// query planes of heads w*HPW .. in registers.
template <int METRIC, typename OutT, int HPW>
__global__ void __launch_bounds__(kEstThreads) estimate_kernel(const EstimateParams p) {
  extern __shared__ uint4 est_smem[];
  __shared__ __align__(8) uint64_t full_bar[kEstStages];
  __shared__ __align__(8) uint64_t empty_bar[kEstStages];
  __shared__ int cum[kEstMaxBatch + 1];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const EstRing ring = est_ring_init(est_smem, full_bar, empty_bar, p.H, tid);
  const EstGeom geom = est_geom(p, cum);
  const uint4* q_code = p.q_code + 2 * geom.row0;   // this sequence's query codes
  __syncthreads();
  const int my_tiles = est_tiles_of_block(geom);
  if (warp >= kEstConsumerWarps) {
    est_produce(p, geom, ring, my_tiles, lane, warp - kEstConsumerWarps);
    grid_launch_dependents();
    return;
  }
  // The cached codes the producers stream were final before the preceding kernel started; the query
  // code is that kernel's output, so the consumers wait for it here (the producers do not).
  grid_dependency_wait();
  grid_launch_dependents();
  QPlanes qp[HPW];
#pragma unroll
  for (int hh = 0; hh < HPW; ++hh) qp[hh] = query_planes(ld_16(q_code + 2 * (warp * HPW + hh)), ld_16(q_code + 2 * (warp * HPW + hh) + 1));
  est_consume<METRIC, OutT, HPW>(p, geom, ring, my_tiles, lane, warp, qp);
}

// ---- estimate with the decode append inside: the same pipeline; warp w loads the query rows of its HPW heads (one
// half-warp per row), transforms, buckets and packs them, and spreads the 16 code words of each head over the warp
// through shared memory.
template <typename T, int HPW, bool ROPE>
__global__ void __launch_bounds__(kEstThreads) estimate_append_kernel(const EstimateParams p) {
  static_assert(HPW == 1 || HPW == 2 || HPW == 4, "heads per warp");
  extern __shared__ uint4 est_smem[];
  __shared__ __align__(8) uint64_t full_bar[kEstStages];
  __shared__ __align__(8) uint64_t empty_bar[kEstStages];
  __shared__ int cum[kEstMaxBatch + 1];
  __shared__ __align__(16) uint16_t s_code[kEstConsumerWarps][32];   // a warp's two rows of code words
  __shared__ float2 s_cs[ROPE ? kHeadDim / 2 : 1];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const StepAppend& a = p.ap;
  const EstRing ring = est_ring_init(est_smem, full_bar, empty_bar, p.H, tid);
  __syncthreads();
  const EstGeom geom = est_geom(p, cum);
  const int my_tiles = est_tiles_of_block(geom);
  if (warp >= kEstConsumerWarps) {
    // the cached codes were final before the preceding kernel started: stream them right away
    est_produce(p, geom, ring, my_tiles, lane, warp - kEstConsumerWarps);
    grid_launch_dependents();
    return;
  }
  if (ROPE) {
    // the new token sits at position n_tokens (= tokens before it)
    if (tid < kHeadDim / 2) s_cs[tid] = rope_cos_sin(tid, static_cast<float>(geom.n_tokens), a.rp);
    asm volatile("bar.sync 1, %0;" ::"n"(kEstConsumerWarps * 32) : "memory");   // the consumer warps only
  }
  // q, k, v are the preceding kernel's output
  grid_dependency_wait();
  grid_launch_dependents();

  const unsigned l16 = lane & 15;
  const int half = lane >> 4;
  constexpr int kPasses = (HPW + 1) / 2;
  // row of a pass for this half-warp: head warp*HPW + 2*pass + half (HPW == 1: both halves take the one head, half 0 stores)
  const int head0 = warp * HPW + (HPW == 1 ? 0 : half);
  const bool writer = HPW > 1 || half == 0;
  const int64_t in_off0 = static_cast<int64_t>(geom.row0 + head0) * kHeadDim + l16 * 8;   // rows of q, k, v: (sequence, head)
  if (geom.appends) {   // block-uniform
    // slot of the new token: from the host, or from the device-resident sequence length (position n)
    int kv_last_page = a.kv_last_page, kv_entry = a.kv_entry, code_last_page = a.code_last_page, code_entry = a.code_entry;
    if (p.seq_len_dev) {
      kv_last_page = code_last_page = geom.n_tokens / p.page_size;
      kv_entry = code_entry = geom.n_tokens - kv_last_page * p.page_size;
    }
    PagedTarget tgt = a.tgt;
    if (p.seqs) {
      const SeqDesc sd = p.seqs[geom.seq];
      tgt.kv_data = sd.kv_data;
      tgt.kv_table = sd.kv_table;
      tgt.code_data = static_cast<uint16_t*>(sd.code_data);
      tgt.code_table = sd.code_table;
    }
    uint4 kraw[kPasses], vraw[kPasses];
#pragma unroll
    for (int pass = 0; pass < kPasses; ++pass) {
      kraw[pass] = ld_16(static_cast<const T*>(a.k) + in_off0 + 2 * pass * kHeadDim);
      vraw[pass] = ld_16(static_cast<const T*>(a.v) + in_off0 + 2 * pass * kHeadDim);
    }
    const int64_t kv_page = __ldg(tgt.kv_table + kv_last_page), code_page = __ldg(tgt.code_table + code_last_page);
    const int64_t v_delta = static_cast<int64_t>(p.page_size) * p.H * kHeadDim;
#pragma unroll
    for (int pass = 0; pass < kPasses; ++pass) {
      const int head = head0 + 2 * pass;
      T* slot = static_cast<T*>(tgt.kv_data) + ((kv_page * 2 * p.page_size + kv_entry) * p.H + head) * kHeadDim + l16 * 8;
      float x[8];
      unpack8<T>(kraw[pass], x);
      if (ROPE) {
        rope_halfwarp_cs<T>(x, l16, s_cs, a.rp.inv_freq != nullptr, a.rp.mscale);
        kraw[pass] = pack8<T>(x);
        if (writer) st_16(static_cast<T*>(a.k) + in_off0 + 2 * pass * kHeadDim, kraw[pass]);
        unpack8<T>(kraw[pass], x);
      }
      if (writer) {
        st_16(slot, kraw[pass]);
        st_16(slot + v_delta, vraw[pass]);
      }
      wht128_halfwarp(x, l16);
      scale_round<T>(x, a.scale);
      if (writer) tgt.code_data[((code_page * p.page_size + code_entry) * p.H + head) * kCodeWords + l16] = bucketize_pack8(x, a.th);
    }
  }
  if (geom.rank >= geom.blocks) return;
  QPlanes qp[HPW];
#pragma unroll
  for (int pass = 0; pass < kPasses; ++pass) {
    float x[8];
    unpack8<T>(ld_16(static_cast<const T*>(a.q) + in_off0 + 2 * pass * kHeadDim), x);
    if (ROPE) rope_halfwarp_cs<T>(x, l16, s_cs, a.rp.inv_freq != nullptr, a.rp.mscale);
    wht128_halfwarp(x, l16);
    scale_round<T>(x, a.scale);
    const unsigned word = bucketize_pack8(x, a.th);   // code word l16 of the row
    if (geom.rank == 0 && writer) a.q_code_out[(geom.row0 + head0 + 2 * pass) * kCodeWords + l16] = static_cast<uint16_t>(word);
    // spread the 16 code words of each row over the warp: through shared memory (one 2-byte store per
    // lane, two 16-byte broadcast loads per head)
    __syncwarp();
    s_code[warp][lane] = static_cast<uint16_t>(word);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < (HPW == 1 ? 1 : 2); ++s) {
      const uint4* cw = reinterpret_cast<const uint4*>(&s_code[warp][16 * s]);
      const int hh = (HPW == 1) ? 0 : 2 * pass + s;
      qp[hh] = query_planes(cw[0], cw[1]);
    }
  }
  est_consume<0, uint16_t, HPW>(p, geom, ring, my_tiles, lane, warp, qp);
}

}  // namespace adamas
