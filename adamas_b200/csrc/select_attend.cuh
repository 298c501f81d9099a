// Stages 3 + 4 of the decode path in one kernel: per head, pick the k smallest of n integer distances
// (ties to the lower position) and run the decode attention over the picked tokens plus the newest
// token.  Used by the fused decode step; the separate top-k and decode kernels remain for callers
// that want the stages one by one.
//
// The kernel does not count anything itself.  The estimate kernels (or dist_histogram_kernel, for a
// caller that only has a distance row) leave, per head, one 512-bin histogram per SLICE of the row
// in a global table [H][kSaMaxSlices][512] u32: a slice covers the granules (8 distances) of one block of
// the head, or of two neighbouring ones.  A distance is at most 3 * 128 = 384; larger values count as 511.
//
// CL <= 16 blocks x 128 threads per head (grid (CL, H)); the blocks of a head never wait for one another.
// Block `cr`:
//   load   its slice of the distance row (asynchronous copies into the shared memory that later holds K and V rows), the
//          head's CL histograms (four bins per thread) and the query, all in flight together;
//   cut    block-wide scan of the summed histogram: the cut distance, how many cut-valued elements
//          are taken in all, how many of them and how many smaller elements lie in lower-ranked
//          slices (= this slice's tie quota and its offset in the output list).  Every block
//          derives this by itself from the same table: no exchange between blocks;
//   pick   ordered compaction of the block's winners into a list in shared memory;
//   attend the rows of the list are dealt out evenly to the 4 warps; a warp gathers the K and V rows of
//          its tokens itself, 24 at a time (16-byte asynchronous copies into its own tile), and works on
//          them alone (q.K on the tensor cores, attend_tile.cuh): no block barrier inside the attention;
//   merge  the 4 warps' partial (o, m, l) are merged in shared memory and the block's partial goes to
//          the head's slot table in global scratch; the block that arrives LAST at the head's counter
//          merges the CL partials, writes the head's output, clears the head's histogram rows and the
//          counter.  Every other block is gone by then.
// Bound: a chain of short dependent phases for one sequence, HBM (the gathered rows) for the longest of them; latency times
// rows in flight for batches.  Blocks are therefore small: four to an SM, so that the chains of different rows overlap, and
// up to 16 to a row, so that a block's winners fit its warps' tiles in one round and a thread has a granule or two.  What
// does not depend on the preceding kernel (length, page numbers, rotation table) is done before its completion.
// Measured, the whole step: blocks of 512 threads with the distances in registers, two to an SM, took 22.7 us per layer for
// one sequence (32 heads, 32K tokens, budget 1024), 103 us for 8 x 32K and 125 us for 32 x 4-8K; this form 20.7, 79 and 81.
// (Blocks of 256 threads, three to an SM: 26.0 / - / 122.  16 rows per tile: a second round for half of the warps.)
// A warp has few others to hide behind (four to a scheduler), so its instructions count: rows are copied, multiplied and weighted
// eight at a time, as many as there are, P.V runs on paired fp32 multiply-adds with the weights from shared memory instead of a
// shuffle per row, and half of the histogram loads are behind one branch (us a layer: 40 heads, 12K 15.5 -> 14.9; 32 over 8, 30K 21.1 -> 20.7; 32 x
// 4-8K 69.0 -> 67.9; 32 heads, 32K 19.9 -> 19.7).
#pragma once
#include "attend_tile.cuh"
#include "common.cuh"
#include "hadamard_append.cuh"

namespace adamas {

constexpr int kSaThreads = 128;
constexpr int kSaWarps = kSaThreads / 32;
constexpr int kSaBlocksPerSm = 4;
constexpr int kSaBins = 512;
constexpr int kSaMaxSlices = 16;      // histogram rows per head = largest number of blocks per head
constexpr int kSaRows = 24;           // rows of a warp's tile
constexpr int kSaWarpBytes = 2 * kSaRows * kHeadDim * 2;
constexpr int kSaTileBytes = kSaWarps * kSaWarpBytes;
constexpr int kSaMaxBlockTokens = 32768;
constexpr int kSaMaxCluster = 8;      // largest value of adamas_set_max_cluster: as many blocks per head as are of use

// Scratch words (32 bit) per head: kSaMaxSlices histogram rows of 512 counts, then kSaMaxSlices slots of
// kSaSlotWords floats for the blocks' partial results (128 outputs, running max, running sum; word 130
// of slot 0 is the head's arrival counter).
constexpr int kSaSlotWords = 132;
constexpr int kSaScratchWordsPerHead = kSaMaxSlices * kSaBins + kSaMaxSlices * kSaSlotWords;

// Granules (8 distances) of a row that each of `cl` blocks owns: a multiple of 4, so that a slice
// starts on a multiple of 32 tokens and no 32-token tile of an estimate kernel straddles two slices.
__host__ __device__ __forceinline__ int sa_granules_per_block(int n, int cl) {
  const int g = ((n + 7) >> 3);
  return (((g + cl - 1) / cl) + 3) & ~3;
}

struct SelectAttendParams {
  const uint16_t* dist;     // [H, dist_stride] u16 distances, rows 16-byte aligned
  int64_t dist_stride;
  uint32_t* hist;           // [H][kSaScratchWordsPerHead]: per-slice histograms of the rows (cleared on exit),
                            // then the slots of the blocks' partial results and the arrival counter
  const int2* ext_cut;      // optional [H]: (cut distance, cut-valued winners this call takes), decided
                            // elsewhere (sequence shards); k is then unused
  const int32_t* seq_len_dev;  // optional: n = *seq_len_dev - 1 and the newest token sits at position n
  const SeqDesc* seqs;      // optional (needs seq_len_dev): a batch of sequences, grid.z = sequence; dist, hist, q, o,
                            // lse and out_idx have one row per (sequence, head); cache, page table and length are the sequence's
  int n;                    // distances per head (tokens 0 .. n-1) when seq_len_dev is null
  int k;                    // winners per head, 1 <= k <= n
  const void* q;            // [H, 128]; read after the preceding kernel has completed
  void* o;                  // [H, 128] in the cache's element type, or null
  float* o_f32;             // [H, 128] fp32 (partial result of a sequence shard), or null
  float* lse;               // [H] or null (base 2)
  const void* kv;           // [pages, 2, page_size, H, 128]
  const int32_t* kv_table;  // logical page -> physical page
  int page_size;
  int ps_shift;             // log2(page_size) or -1
  int H;                    // heads of the KV cache
  int q_group;              // query heads per cache head (grouped-query attention; 1 otherwise): the grid, dist,
                            // hist, q, o, lse and out_idx have H * q_group rows; row r attends cache head r / q_group
  int tail_mode;            // 0: no newest token; 1: it is at tail_slot; 2: at logical position n
  unsigned tail_slot;       // physical slot of the newest token (tail_mode 1)
  int32_t* out_idx;         // optional [H, out_stride]: physical slots of the winners, ascending position
  int64_t out_stride;
  int slices;               // histogram rows per head
  int share_shift;          // 0 or 1: 1 << share_shift blocks share one
  int staged_granules;      // granules of a slice staged in the tiles' memory
  int pages_at;             // where in shared memory the block's page numbers go; 0: they are not staged
  int bin_threads;          // threads that read histogram bins (four each): the bins that can be in use
  int list_capacity;        // entries of the shared-memory winner list (a block's winners at most, plus the newest token)
  float scale_log2;
  // q arrives un-rotated (the append-fused estimate in front of this launch has coded the rotated query but left
  // q alone): every block rotates it for position n for its own use, the block that finishes a head writes
  // the rotated row back into q
  int rope_on;
  RopeParams rope;
};

struct SaShared {
  float ml[kSaWarps][2];
  uint2 warp_sum[kSaWarps];
  unsigned cut, need_eq, lt_before, eq_before;
  unsigned tail_slot;
  unsigned last;   // this block arrived last at the head's counter
  alignas(16) uint16_t q[kHeadDim];   // the head's query row, rotated
  float2 cs[kHeadDim / 2];   // rope_on: (cos, sin) of the position
};

// The 8 values of a granule against the cut: bit i of *lt / *eq where value i is below it / equal to it.  Compared in pairs as
// fp16 numbers: a bit pattern up to 512 is a denormal, and those are in the order of the integers (values beyond 511 are
// clamped first, the others might be NaNs).  18 instructions besides the clamps; whole-number arithmetic on halfwords took 50.
// With the list written 32 tokens at a time instead of 8, us a layer: 32 heads, 32K 20.4 -> 20.2, 128K 45.1 -> 44.0; 8 x 32K 79.1 -> 76.1;
// 32 x 4-8K 71.9 -> 69.0.
__device__ __forceinline__ unsigned sa_gather_bits(unsigned w0, unsigned w1, unsigned w2, unsigned w3) {   // halfwords 0 or 0xffff -> bits
  const unsigned a = __byte_perm(w0, w1, 0x6420) & 0x08040201u, b = __byte_perm(w2, w3, 0x6420) & 0x80402010u;
  return __dp4a(a | b, 0x01010101u, 0u);
}
__device__ __forceinline__ void sa_compare(uint4 v, __half2 cut, unsigned* lt, unsigned* eq) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  unsigned l[4], e[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned x = __vminu2(w[i], 0x01ff01ffu);
    l[i] = __hlt2_mask(*reinterpret_cast<const __half2*>(&x), cut);
    e[i] = __heq2_mask(*reinterpret_cast<const __half2*>(&x), cut);
  }
  *lt = sa_gather_bits(l[0], l[1], l[2], l[3]);
  *eq = sa_gather_bits(e[0], e[1], e[2], e[3]);
}

// Dynamic shared memory: the warps' tiles (12 KB each; first the staged distances, at the end a warp parks
// its partial output in its tile) | winner list (list_capacity * 2 B) | page numbers.
template <typename T>
__global__ void __launch_bounds__(kSaThreads, kSaBlocksPerSm) select_attend_kernel(const SelectAttendParams p) {
  static_assert(4 * kSaThreads == kSaBins && kSaThreads == kHeadDim, "four histogram bins and one output per thread");
  extern __shared__ __align__(128) uint8_t sa_smem[];
  __shared__ __align__(16) SaShared sh;

  const unsigned CL = gridDim.x;
  const unsigned cr = blockIdx.x;
  const int head = blockIdx.z * gridDim.y + blockIdx.y;   // row of dist, hist, q, o, lse, out_idx: (sequence, query head)
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int H = p.H;
  const int head_kv = p.q_group == 1 ? blockIdx.y : blockIdx.y / p.q_group;
  const int32_t* kv_table = p.kv_table;
  const void* kv_base = p.kv;
  const int32_t* seq_len_dev = p.seq_len_dev;
  if (p.seqs) {   // (the table of sequences is set up once, long before this launch)
    kv_table = p.seqs[blockIdx.z].kv_table;
    kv_base = p.seqs[blockIdx.z].kv_data;
    seq_len_dev += blockIdx.z;
  }

  uint16_t* s_list = reinterpret_cast<uint16_t*>(sa_smem + kSaTileBytes);             // the block's winners in position order: tokens behind its first
  uint32_t* head_scratch = p.hist + static_cast<size_t>(head) * kSaScratchWordsPerHead;
  float* slots = reinterpret_cast<float*>(head_scratch + kSaMaxSlices * kSaBins);     // [CL][kSaSlotWords]

  // ---- set-up that does not depend on the preceding kernel (overlaps its tail) ------------------------
  // (a device-resident length and the page tables are final before the kernel in front of this one starts)
  if (tid == 0) sh.cut = 0xffffffffu;
  const int n = seq_len_dev ? (__ldg(seq_len_dev) - 1) : p.n;
  const int G = (n + 7) >> 3;
  // slice of the histograms, and this block's part of it (one or two blocks share a slice; the second one counts what lies in front
  // of it in the first part by itself)
  const int per_slice = sa_granules_per_block(n, p.slices);
  const int slice = cr >> p.share_shift, per_part = (per_slice + p.share_shift) >> p.share_shift;
  const bool second = cr & p.share_shift;
  const int seg_first = slice * per_slice, seg_end = min(G, seg_first + per_slice);
  const int pre = second ? max(0, min(per_part, seg_end - seg_first)) : 0;      // granules of the slice in front of this block's
  const int blk_first = seg_first + pre, blk_count = max(0, min(second ? per_slice - per_part : per_part, seg_end - blk_first));
  // the page numbers of the block's tokens, where they fit
  const unsigned ps = static_cast<unsigned>(p.page_size);
  auto page_of = [&](unsigned t) { return p.ps_shift >= 0 ? t >> p.ps_shift : t / ps; };
  int32_t* pages = reinterpret_cast<int32_t*>(sa_smem + p.pages_at);   // (behind the list)
  const unsigned page0 = page_of(static_cast<unsigned>(blk_first) * 8);
  const int n_pages = p.pages_at && blk_count > 0 ? static_cast<int>(page_of(min(static_cast<unsigned>(blk_first + blk_count) * 8, static_cast<unsigned>(n)) - 1) - page0) + 1 : 0;
  for (int i = tid; i < n_pages; i += kSaThreads) pages[i] = __ldg(kv_table + page0 + i);
  // (rope_on: the position's cos / sin pairs)
  if (p.rope_on && tid < kHeadDim / 2) sh.cs[tid] = rope_cos_sin(tid, static_cast<float>(n), p.rope);
  // the newest token rides with the last slice
  const bool tail_here = p.tail_mode != 0 && cr == CL - 1;
  if (tail_here && tid == 0) {
    sh.tail_slot = p.tail_slot;
    if (p.tail_mode == 2) {
      const unsigned un = static_cast<unsigned>(n), pg = page_of(un);
      sh.tail_slot = static_cast<unsigned>(__ldg(kv_table + pg)) * ps + (un - pg * ps);
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();

  // ---- loads: histograms, query, distances, all in flight together ------------------------------------
  const uint4* gbase = reinterpret_cast<const uint4*>(p.dist + static_cast<int64_t>(head) * p.dist_stride) + seg_first;
  uint4* staged = reinterpret_cast<uint4*>(sa_smem);   // granule g of the slice at g + g / 8: reads of neighbouring threads' runs do not conflict
  const int n_staged = min(pre + blk_count, p.staged_granules);
  uint4 tot = make_uint4(0u, 0u, 0u, 0u), low = tot;   // bins 4 * tid ..: the whole row; lower-ranked slices
  const T* q_row = static_cast<const T*>(p.q) + static_cast<int64_t>(head) * kHeadDim;
  uint16_t q_own, q_pair = 0;                          // the query's element tid, and the one it rotates with
  {
    const uint4* hrow = reinterpret_cast<const uint4*>(head_scratch) + tid;
    constexpr unsigned kHalf = kSaMaxSlices / 2;
    uint4 c[kSaMaxSlices];
    auto load = [&](unsigned r) { c[r] = r < static_cast<unsigned>(p.slices) && tid < p.bin_threads ? __ldcg(hrow + r * (kSaBins / 4)) : make_uint4(0u, 0u, 0u, 0u); };
    auto add = [&](unsigned r) {
      tot.x += c[r].x; tot.y += c[r].y; tot.z += c[r].z; tot.w += c[r].w;
      if (r < static_cast<unsigned>(slice)) { low.x += c[r].x; low.y += c[r].y; low.z += c[r].z; low.w += c[r].w; }
    };
#pragma unroll
    for (unsigned r = 0; r < kHalf; ++r) load(r);
    if (p.slices > static_cast<int>(kHalf)) {
#pragma unroll
      for (unsigned r = kHalf; r < kSaMaxSlices; ++r) load(r);
    }
    q_own = reinterpret_cast<const uint16_t*>(q_row)[tid];
    if (p.rope_on) q_pair = reinterpret_cast<const uint16_t*>(q_row)[tid ^ (kHeadDim / 2)];
    for (int g = tid; g < n_staged; g += kSaThreads) cp_async_16(staged + g + (g >> 3), gbase + g);
    cp_async_commit();
#pragma unroll
    for (unsigned r = 0; r < kHalf; ++r) add(r);
    if (p.slices > static_cast<int>(kHalf)) {
#pragma unroll
      for (unsigned r = kHalf; r < kSaMaxSlices; ++r) add(r);
    }
  }

  // ---- cut ----------------------------------------------------------------------------------------------
  {
    const unsigned t4 = (tot.x + tot.y) + (tot.z + tot.w), l4 = (low.x + low.y) + (low.z + low.w);
    unsigned it = t4, il = l4;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, it, o);
      const unsigned u = __shfl_up_sync(0xffffffffu, il, o);
      if (lane >= o) {
        it += t;
        il += u;
      }
    }
    if (lane == 31) sh.warp_sum[warp] = make_uint2(it, il);
    __syncthreads();
    unsigned below = it - t4, below_low = il - l4;   // elements below this thread's first bin: whole row, lower-ranked slices
#pragma unroll
    for (int w2 = 0; w2 < kSaWarps - 1; ++w2) {
      const uint2 v = sh.warp_sum[w2];
      below += w2 < warp ? v.x : 0u;
      below_low += w2 < warp ? v.y : 0u;
    }
    const unsigned tb[4] = {tot.x, tot.y, tot.z, tot.w}, lb[4] = {low.x, low.y, low.z, low.w};
    if (p.ext_cut) {
      // (a cut of 512, beyond every bin: the whole row wins; the last thread stands in, there are no ties)
      const int2 e = __ldg(p.ext_cut + head);
      const bool all_win = e.x >= kSaBins;
      const int bin = min(e.x, kSaBins - 1);
      if (tid == bin >> 2) {
        unsigned lt = below_low;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i < (bin & 3) || all_win) lt += lb[i];
          if (i == (bin & 3)) sh.eq_before = all_win ? 0u : lb[i];
        }
        sh.cut = all_win ? static_cast<unsigned>(kSaBins) : static_cast<unsigned>(bin);
        sh.need_eq = all_win ? 0u : static_cast<unsigned>(e.y);
        sh.lt_before = lt;
      }
    } else {
      const unsigned want = static_cast<unsigned>(p.k);
      if (below < want && below + t4 >= want) {   // exactly one thread
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (below < want && below + tb[i] >= want) {
            sh.cut = 4 * tid + i;
            sh.need_eq = want - below;     // cut-valued winners in all
            sh.lt_before = below_low;      // smaller-valued elements in lower-ranked slices
            sh.eq_before = lb[i];          // cut-valued elements in lower-ranked slices
          }
          below += tb[i];
          below_low += lb[i];
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads();   // the cut is known, the staged distances are visible
  }
  unsigned cut = sh.cut;
  unsigned need_eq = sh.need_eq, lt_before = sh.lt_before, eq_before = sh.eq_before;
  if (cut == 0xffffffffu) {
    // the table does not describe this row (fewer than k entries): take nothing but the newest token
    if (tid == 0) atomicOr(&g_adamas_error, kErrHistogram);
    cut = need_eq = lt_before = eq_before = 0;
  }

  // ---- pick: ordered compaction of this block's winners -----------------------------------------------
  // A thread owns `run` consecutive granules, four of them (32 tokens) to a pair of words: which elements are below the cut, which
  // at it.  It counts them; a block scan gives it its place in the list, and a second look at the words writes the winners.  (The words
  // of the first four stay in registers, the others take the place of the first of their granules.)
  const unsigned cut2 = cut * 0x00010001u;
  const __half2 cut_h = *reinterpret_cast<const __half2*>(&cut2);
  const int run = (blk_count + kSaThreads - 1) / kSaThreads;
  const int g_first = pre + tid * run, g_end = min(pre + blk_count, g_first + run);
  // (All four are read before the first is compared: where a block's part is longer than what is staged, the last threads read theirs
  // from L2.  One after the other, us a layer: 2 x 375K of 4 heads 44.8, now 36.4; 8 x 30K of 64 heads, one block per head, 123.7 -> 117.3.)
  auto masks = [&](int g, int end) {   // of granules g .. min(g + 4, end)
    uint2 m = make_uint2(0u, 0u);
    uint4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (g + i < end) v[i] = g + i < n_staged ? staged[g + i + ((g + i) >> 3)] : ld_16(gbase + g + i);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (g + i < end) {
        unsigned lt, eq;
        sa_compare(v[i], cut_h, &lt, &eq);
        m.x |= lt << (8 * i);
        m.y |= eq << (8 * i);
      }
    }
    const int left = n - (seg_first + g) * 8;   // (the row may end inside the last granule)
    if (left < 32) {
      const unsigned valid = left > 0 ? (1u << left) - 1u : 0u;
      m.x &= valid;
      m.y &= valid;
    }
    return m;
  };
  auto counts_of = [](uint2 m) { return static_cast<unsigned>(__popc(m.x) + (__popc(m.y) << 16)); };
  unsigned packed = 0, ahead = 0;   // elements below the cut | elements at the cut << 16 (a block holds at most 32768)
  uint2 mask0 = make_uint2(0u, 0u);
  if (g_first < g_end) mask0 = masks(g_first, g_end);
  packed = counts_of(mask0);
  for (int g = g_first + 4; g < g_end; g += 4) {
    const uint2 m = masks(g, g_end);
    if (g < n_staged) *reinterpret_cast<uint2*>(staged + g + (g >> 3)) = m;
    packed += counts_of(m);
  }
  if (pre > 0) {
    const int pre_run = (pre + kSaThreads - 1) / kSaThreads, pre_end = min(pre, (tid + 1) * pre_run);
    for (int g = tid * pre_run; g < pre_end; g += 4) ahead += counts_of(masks(g, pre_end));
  }
  unsigned incl = packed;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (p.share_shift) ahead = __reduce_add_sync(0xffffffffu, ahead);
  if (lane == 31) sh.warp_sum[warp] = make_uint2(incl, ahead);   // (the readers of the cut phase are past a block barrier)
  if (p.rope_on) {   // (rope_halfwarp_cs, one element per thread)
    const float2 cs = sh.cs[tid & (kHeadDim / 2 - 1)];
    const float x = Elem<T>::to_f2(q_own).x, other = Elem<T>::to_f2(q_pair).x;
    float r = tid >= kHeadDim / 2 ? fmaf(other, cs.y, x * cs.x) : fmaf(-other, cs.y, x * cs.x);
    if (p.rope.inv_freq) r *= p.rope.mscale;
    q_own = static_cast<uint16_t>(Elem<T>::from_f2(r, 0.f));
  }
  sh.q[tid] = q_own;
  __syncthreads();
  unsigned before = incl - packed, blk_tot = 0;
#pragma unroll
  for (int w2 = 0; w2 < kSaWarps; ++w2) {
    const uint2 a = sh.warp_sum[w2];
    before += (w2 < warp) ? a.x : 0u;
    blk_tot += a.x;
    lt_before += a.y & 0xffffu;
    eq_before += a.y >> 16;
  }
  const unsigned take_eq = need_eq > eq_before ? need_eq - eq_before : 0u;   // this block's tie quota
  const int n_win = static_cast<int>((blk_tot & 0xffffu) + min(blk_tot >> 16, take_eq));
  const int n_loc = min(n_win + (tail_here ? 1 : 0), p.list_capacity);
  // of a thread's cut-valued elements the first `quota` win; its winners are neighbours in the list
  unsigned quota = take_eq > (before >> 16) ? min(take_eq - (before >> 16), packed >> 16) : 0u;
  unsigned pos = (before & 0xffffu) + min(before >> 16, take_eq);
  if ((packed & 0xffffu) + quota) {
    const bool all_eq = quota == packed >> 16;
    for (int g = g_first; g < g_end; g += 4) {
      const uint2 m = g == g_first ? mask0 : g < n_staged ? *reinterpret_cast<const uint2*>(staged + g + (g >> 3)) : masks(g, g_end);
      unsigned win = m.x;
      if (all_eq) {
        win |= m.y;
      } else {
        for (unsigned eq = m.y; eq && quota; --quota) {
          win |= eq & -eq;
          eq &= eq - 1;
        }
      }
      const unsigned t0 = static_cast<unsigned>(g - pre) * 8;
      while (win) {
        if (pos < static_cast<unsigned>(p.list_capacity)) s_list[pos] = static_cast<uint16_t>(t0 + __ffs(win) - 1);
        win &= win - 1;
        ++pos;
      }
    }
  }
  __syncthreads();   // the list and the query are complete, the staged distances are read

  // ---- attend: warp w takes rows w*rpw .. of the list, 24 at a time --------------------------------------
  uint8_t* tile = sa_smem + warp * kSaWarpBytes;
  float m_run = -INFINITY, l_run = 0.f;
  float2 acc_lo = make_float2(0.f, 0.f), acc_hi = acc_lo;   // dimensions 4 * lane ..
  const int rpw = (n_loc + kSaWarps - 1) / kSaWarps;
  const int my_first = warp * rpw;
  const int my_total = max(0, min(rpw, n_loc - my_first));
  if (my_total > 0) {
    const uint32_t row_bytes = static_cast<uint32_t>(H) * kHeadDim * 2;   // (H <= 1024)
    const uint8_t* kbase = reinterpret_cast<const uint8_t*>(static_cast<const T*>(kv_base) + head_kv * kHeadDim);
    const uint8_t* vbase = kbase + static_cast<uint64_t>(p.page_size) * row_bytes;
    int32_t* oi = p.out_idx ? p.out_idx + static_cast<int64_t>(head) * p.out_stride + lt_before + min(eq_before, need_eq) : nullptr;
    uint4 q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = lane < 4 ? reinterpret_cast<const uint4*>(sh.q)[4 * j + lane] : make_uint4(0, 0, 0, 0);
    for (int done = 0; done < my_total; done += kSaRows) {
      // K rows as one commit group, V rows as a second: the logits are formed while the V rows are still on their way
      // (lanes beyond the rows borrow the last one)
      const int at = my_first + min(done + lane, my_total - 1);
      unsigned slot;
      if (at < n_win) {
        const unsigned t = static_cast<unsigned>(blk_first) * 8 + s_list[at], pg = page_of(t);   // logical token position
        slot = static_cast<unsigned>(n_pages ? pages[pg - page0] : __ldg(kv_table + pg)) * ps + (t - pg * ps);
        if (oi && done + lane < my_total && lane < kSaRows) oi[at] = static_cast<int32_t>(slot);
      } else {
        slot = sh.tail_slot;
      }
      const int row = static_cast<int>(slot + page_of(slot) * ps);   // page * 2 ps + entry
      const int rem = my_total - done;
      auto copy = [&](const uint8_t* base, uint8_t* to) {   // (eight rows at a time, as many as there are)
        tile_copy8<0>(base, row_bytes, row, to, lane);
        if (rem > 8) tile_copy8<8>(base, row_bytes, row, to, lane);
        if (rem > 16) tile_copy8<16>(base, row_bytes, row, to, lane);
        cp_async_commit();
      };
      copy(kbase, tile);
      copy(vbase, tile + kSaRows * 256);
      float sc[kSaRows / 4];
      cp_async_wait<1>();
      __syncwarp();
      tile_logits8<T, kSaRows>(tile, q, rem, p.scale_log2, lane, sc);
      // softmax in base 2 (the head's logits are in lanes 0 .. 3) and P.V with four
      // dimensions per lane: one query row leaves the matrix form an eighth used and its accumulators cost 28 registers
      float m_new = sc[0];
#pragma unroll
      for (int u = 1; u < kSaRows / 4; ++u) m_new = fmaxf(m_new, sc[u]);
      m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 1));
      m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 2));
      m_new = fmaxf(m_run, __shfl_sync(0xffffffffu, m_new, 0));
      const float base = m_new == -INFINITY ? 0.f : m_new;   // (no logit above -inf so far: no weight)
      const float rescale = exp2f(m_run - base);
      m_run = m_new;
      l_run *= rescale;
      acc_lo.x *= rescale; acc_lo.y *= rescale; acc_hi.x *= rescale; acc_hi.y *= rescale;
#pragma unroll
      for (int u = 0; u < kSaRows / 4; ++u) {
        sc[u] = exp2f(sc[u] - base);
        l_run += sc[u];
        sc[u] = fmaxf(sc[u], 1.4e-45f);   // (0 times an infinity, in the row that an absent one borrows, would be a NaN)
      }
      // the weights go through shared memory (the K rows' place: they are read), each twice: a pair of them is an operand of the paired
      // multiply-add
      float4* weights = reinterpret_cast<float4*>(tile);
      __syncwarp();
      if (lane < 4) {
#pragma unroll
        for (int u = 0; u < kSaRows / 8; ++u) weights[4 * u + lane] = make_float4(sc[2 * u], sc[2 * u], sc[2 * u + 1], sc[2 * u + 1]);
      }
      cp_async_wait<0>();
      __syncwarp();
      const uint8_t* vrow = tile + kSaRows * 256 + (lane & 1) * 8;
      auto weigh8 = [&](int first) {
#pragma unroll
        for (int j = first; j < first + 8; j += 2) {
          const float4 pp = weights[j >> 1];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint2 vv = *reinterpret_cast<const uint2*>(vrow + (j + i) * 256 + (((lane >> 1) ^ tile_swizzle(j + i)) << 4));
            const float2 pj = i == 0 ? make_float2(pp.x, pp.y) : make_float2(pp.z, pp.w);
            acc_lo = fma2(pj, Elem<T>::to_f2(vv.x), acc_lo);
            acc_hi = fma2(pj, Elem<T>::to_f2(vv.y), acc_hi);
          }
        }
      };
      weigh8(0);
      if (rem > 8) weigh8(8);
      if (rem > 16) weigh8(16);
      __syncwarp();   // the tile may be filled again
    }
  }

  // ---- merge: warps -> block -> head ----------------------------------------------------------------------
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);   // (lanes 0 .. 3)
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  __syncwarp();
  reinterpret_cast<float4*>(tile)[lane] = make_float4(acc_lo.x, acc_lo.y, acc_hi.x, acc_hi.y);
  if (lane == 0) {
    sh.ml[warp][0] = m_run;
    sh.ml[warp][1] = l_run;
  }
  __syncthreads();
  float od = 0.f, L = 0.f, M = -INFINITY;
#pragma unroll
  for (int w2 = 0; w2 < kSaWarps; ++w2) M = fmaxf(M, sh.ml[w2][0]);
#pragma unroll
  for (int w2 = 0; w2 < kSaWarps; ++w2) {
    const float m = sh.ml[w2][0];
    const float w = (m == -INFINITY) ? 0.f : exp2f(m - M);
    L += w * sh.ml[w2][1];
    const float part = reinterpret_cast<const float*>(sa_smem + w2 * kSaWarpBytes)[tid];
    if (w != 0.f) od += w * part;   // (it may be infinite)
  }
  unsigned* counter = head_scratch + kSaMaxSlices * kSaBins + kHeadDim + 2;   // word 130 of slot 0
  if (CL > 1) {
    float* slot = slots + cr * kSaSlotWords;
    __stcg(slot + tid, od);
    if (tid == 0) __stcg(reinterpret_cast<float2*>(slot + kHeadDim), make_float2(M, L));
    // the block that arrives last at the head's counter merges; nobody waits.  The block barrier orders
    // the slot stores of all threads before thread 0's release at the counter; the last block's acquire
    // there, followed by the second barrier, orders its loads of the slots after every block's stores.
    __syncthreads();
    if (tid == 0) {
      unsigned ticket;
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(counter) : "memory");
      sh.last = (ticket == CL - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (!sh.last) return;
    // lane r of every warp takes block r's (max, sum); all loads of the partials are issued before the first is used
    float2 ml = make_float2(-INFINITY, 0.f);
    if (lane < static_cast<int>(CL)) ml = __ldcg(reinterpret_cast<const float2*>(slots + lane * kSaSlotWords + kHeadDim));
    float po[kSaMaxSlices];
#pragma unroll
    for (unsigned r = 0; r < kSaMaxSlices; ++r) po[r] = r < CL ? __ldcg(slots + r * kSaSlotWords + tid) : 0.f;
    M = ml.x;
#pragma unroll
    for (int o = 1; o < kSaMaxSlices; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float w = (ml.x == -INFINITY) ? 0.f : exp2f(ml.x - M);
    L = w * ml.y;
#pragma unroll
    for (int o = 1; o < kSaMaxSlices; o <<= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    // (lanes 16 .. 31 hold no block)
    M = __shfl_sync(0xffffffffu, M, 0);
    L = __shfl_sync(0xffffffffu, L, 0);
    od = 0.f;
#pragma unroll
    for (unsigned r = 0; r < kSaMaxSlices; ++r) {
      const float wr = __shfl_sync(0xffffffffu, w, r);
      if (wr != 0.f) od = fmaf(wr, po[r], od);
    }
  }
  const float res = L > 0.f ? od / L : 0.f;
  const float res1 = __shfl_down_sync(0xffffffffu, res, 1);
  if (p.o_f32) p.o_f32[static_cast<int64_t>(head) * kHeadDim + tid] = res;
  if (p.o && (tid & 1) == 0)
    reinterpret_cast<uint32_t*>(static_cast<T*>(p.o) + static_cast<int64_t>(head) * kHeadDim)[tid >> 1] =
        Elem<T>::from_f2(res, res1);
  if (tid == 0 && p.lse) p.lse[head] = L > 0.f ? M + log2f(L) : -INFINITY;
  // every block of the head has read the histograms and the un-rotated query long ago: clear the table and the counter
  // for the next launch
  for (int r = 0; r < p.slices; ++r) reinterpret_cast<uint4*>(head_scratch)[r * (kSaBins / 4) + tid] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) *counter = 0u;
  if (p.rope_on && tid < 16)
    st_16(const_cast<T*>(q_row) + tid * 8, reinterpret_cast<const uint4*>(sh.q)[tid]);
}

// Per-slice histograms of distance rows, for callers of select_attend that did not get them from an
// estimate kernel: grid (cl, H); block (r, h) counts slice r of head h in shared memory and STORES the
// row (the table needs no clearing beforehand).
struct DistHistogramParams {
  const uint16_t* dist;
  int64_t dist_stride;
  uint32_t* hist;
  int n;                        // distances per row
  int cl;
};

// Per-slice histograms of given distance rows: grid (slices, rows).  Used where the rows exist already (the stand-alone
// select_attend call): a block counts its slice in shared memory and stores 512 totals.
__global__ void __launch_bounds__(kSaBins) dist_histogram_kernel(const DistHistogramParams p) {
  __shared__ unsigned h_local[kSaBins];
  const int tid = threadIdx.x;
  const int r = blockIdx.x;
  const int head = blockIdx.y;
  h_local[tid] = 0;
  __syncthreads();
  grid_dependency_wait();
  grid_launch_dependents();
  const int n = p.n, G = (n + 7) >> 3;
  const int gpb = sa_granules_per_block(n, p.cl);
  const int g_end = min(G, (r + 1) * gpb);
  const uint4* gbase = reinterpret_cast<const uint4*>(p.dist + static_cast<int64_t>(head) * p.dist_stride);
  for (int g = r * gpb + tid; g < g_end; g += kSaBins) {
    const uint4 v = ld_16(gbase + g);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const int valid = min(8, n - g * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned d = (w[j >> 1] >> ((j & 1) * 16)) & 0xffffu;
      if (j < valid) atomicAdd(&h_local[min(d, static_cast<unsigned>(kSaBins - 1))], 1u);
    }
  }
  __syncthreads();
  p.hist[static_cast<size_t>(head) * kSaScratchWordsPerHead + r * kSaBins + tid] = h_local[tid];
}

// ---- a sequence split over several GPUs: one cut for all shards -----------------------------------------------
// Every shard counts its own distances (estimate kernel, per-slice histograms).  hist_rowsum_kernel adds
// a shard's slices to one 512-bin histogram per head; the shards exchange those ([G][H][512], one
// all-gather); global_cut_kernel then derives, identically on every shard, the cut distance of the k
// smallest distances of the whole sequence and this shard's share of the cut-valued elements (shards
// hold ascending token ranges, so "the lower position wins a tie" means: lower shards first): the
// ext_cut input of select_attend_kernel.  No candidate list ever crosses the link.
__global__ void __launch_bounds__(kSaBins) hist_rowsum_kernel(const uint32_t* __restrict__ scratch, int slices,
                                                              uint32_t* __restrict__ out) {
  const int head = blockIdx.x, tid = threadIdx.x;
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t* rows = scratch + static_cast<size_t>(head) * kSaScratchWordsPerHead + tid;
  uint32_t c = 0;
  for (int r = 0; r < slices; ++r) c += __ldcg(rows + r * kSaBins);
  out[static_cast<size_t>(head) * kSaBins + tid] = c;
}

// all: [G][H][512] counts; ext_cut[h] = (cut distance, cut-valued elements shard `rank` takes).  If the
// whole sequence holds fewer than k distances every element wins: cut = 512, nothing to share out.
__global__ void __launch_bounds__(kSaBins) global_cut_kernel(const uint32_t* __restrict__ all, int G, int rank, int H,
                                                             int k, int2* __restrict__ ext_cut) {
  __shared__ unsigned warp_tot[kSaBins / 32];
  __shared__ int2 result;
  const int head = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) result = make_int2(kSaBins, 0);
  unsigned tot = 0, low = 0, own = 0;
  for (int g = 0; g < G; ++g) {
    const unsigned c = all[(static_cast<size_t>(g) * H + head) * kSaBins + tid];
    tot += c;
    if (g < rank) low += c;
    if (g == rank) own = c;
  }
  unsigned incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  unsigned before = 0;
  for (int w2 = 0; w2 < warp; ++w2) before += warp_tot[w2];
  const unsigned excl = before + incl - tot;
  const unsigned want = static_cast<unsigned>(k);
  if (excl < want && excl + tot >= want) {   // exactly one thread, if the sequence holds k distances
    const unsigned need = want - excl;       // cut-valued winners in all
    const unsigned take = need > low ? min(need - low, own) : 0u;
    result = make_int2(tid, static_cast<int>(take));
  }
  __syncthreads();
  if (tid == 0) ext_cut[head] = result;
}

}  // namespace adamas
