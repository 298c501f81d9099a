// Stage 4 of the decode path: decode attention of one query row per head over a list of token slots in the
// paged KV cache: a per-head list of selected slots (plus an always-attended tail), or, in the dense layers,
// every token of the sequence through its page table.
//
// Bound: HBM (512 bytes of K and V per attended token and cache head; the contraction is one to a few query
// rows deep).  What the kernel is built around is therefore bytes in flight and few instructions per byte:
//   * A warp works alone on tiles of 16 tokens of one cache head, gathered by its own 16-byte asynchronous copies
//     into a ring of kDecStages tiles (8 KB each) in shared memory: no block barrier, and 16 KB on their way per
//     warp whatever the warp is doing.  (The same tiles loaded straight into registers measured 160-185 us instead
//     of 126: the loads shared scoreboards with the softmax's shuffles, which then waited for memory.)
//   * q.K and P.V run on the tensor cores (mma.sync m16n8k16, fp32 accumulation) for up to 8 query heads that
//     share the cache head (grouped queries), so a K/V row is read once per group and not once per query head.
//     See attend_tile.cuh.
// A block is 4 warps that deal out the tiles of one row group (a cache head and its query heads), two blocks per SM.
// The work of a launch is a line of tiles, row group after row group; each block takes an equal piece of it (so that
// sequences of different lengths and head counts that do not divide the chip leave nothing idle), or, for small
// launches where the latency of a second row group would count, an equal share of one.  A row group cut over several
// blocks is merged by the block that arrives last at its counter (no block ever waits for another).
// Measured, append and attention over all tokens of a layer: 32 heads x 32768 tokens, fp16: 128 -> 92 us (537 MB: 5.8 TB/s, 90 %
// of the copy rate, the append's launch included); 21 sequences x 64 query heads over 8 x 7366 tokens: 1097 -> 118 us.  One block of 8 warps per SM: 4 us
// more (the end of a piece leaves the SM idle); three blocks of 4 with two ring slots: 6 us more.  Blocks that take four
// neighbouring heads of a token (1 KB in a row) measured no better than one head per block.
#pragma once
#include "attend_tile.cuh"
#include "common.cuh"

namespace adamas {

constexpr int kDecTile = kTileRows;   // tokens per warp tile
constexpr int kDecWarps = 4;
constexpr int kDecBlocksPerSm = 2;
constexpr int kDecThreads = kDecWarps * 32;
constexpr int kDecStages = 3;
constexpr int kDecTileBytes = kTileBytes;
constexpr int kDecMaxGroup = 8;     // query heads per matrix instruction; larger groups are split
constexpr int kDecMaxBatch = 1024;
constexpr int kDecMinTiles = 6;     // tiles a block is worth starting for

// Blocks per row group for `rows` row groups of `tiles` tiles each, or 0: cut the line of all tiles evenly.  With little
// work latency counts, so a block gets a share of ONE row group (a second one would be a second pass through index
// list, rows and merge).  A group of query heads (gs > 1) has as many results to merge per part: half as many parts;
// measured at 28 query heads over 4 x 2001 tokens: 11.9 us with 6 tiles per block, 10.7 with 12; one query head per
// row, 512 tokens: 7.4 / 8.3.
__host__ __device__ __forceinline__ int dec_splits(int rows, int tiles, int gs, int slots) {
  if (rows > slots || static_cast<int64_t>(rows) * tiles >= static_cast<int64_t>(slots) * kDecWarps * 4) return 0;
  const int min_tiles = gs > 1 ? 2 * kDecMinTiles : kDecMinTiles;
  const int most = slots / rows, wanted = (tiles + min_tiles - 1) / min_tiles;
  return wanted < 1 ? 1 : wanted < most ? wanted : most;
}

struct DecodeParams {
  const void* q;          // [rows, 128]
  void* o;                // [rows, 128] in the cache's element type, or null
  float* o_f32;           // [rows, 128] fp32 output (partial results of a sequence shard), or null
  float* lse;             // [rows] or null (base-2 log-sum-exp of the scaled logits)
  const void* kv;         // [pages, 2, page_size, H, 128]
  const int32_t* indices; // [q heads, idx_stride], or one row for all heads (idx_stride 0)
  int64_t idx_stride;
  int n_listed;           // tokens the index list stands for
  int idx_unit;           // token slots covered by one index
  int page_size;
  int ps_shift;           // log2(page_size) or -1
  int H;                  // heads of the KV cache
  int q_heads;
  // row heads: what a tile belongs to.  One list for all heads: the cache heads, each with `group` query heads in
  // `subs` parts of at most `gs`.  A list per query head: the query heads, group 1 (row_to_kv of them share a cache head).
  int row_heads, row_to_kv, group, subs, gs;
  int batch;
  unsigned tail_slot0;    // physical token slot of the first tail token (tokens n_listed ..)
  int n_tokens;
  int splits;             // > 0: blocks per row group; 0: the line of all tiles is cut evenly over the grid
  int slots;              // blocks resident at once on the device
  float* partial_o;       // [units * gs, 128]
  float* partial_ml;      // [units * gs, 2]
  unsigned* counters;     // [row groups], zero on entry and on exit
  float scale_log2;       // sm_scale * log2(e)
  // optional: attend to EVERY token of a sequence whose length lives on the device (the dense layers of a
  // graph-captured decode step): `indices` is then the page table
  const int32_t* seq_len_dev;
  // optional (needs seq_len_dev): a batch of sequences.  q, o, o_f32 and lse have one row per (sequence, head); the
  // cache, its page table and the length are the sequence's.
  const SeqDesc* seqs;
};

// The token list of one row.
struct DecRow {
  const int32_t* idx;
  int n_listed, n_tokens;
  unsigned tail_slot0;
};

// The list entry token j is looked up by (a page number or a slot; requested well before it is needed) ...
__device__ __forceinline__ int dec_list_entry(const DecodeParams& p, const DecRow& r, int j) {
  if (j >= min(r.n_listed, r.n_tokens)) return 0;
  const unsigned uj = static_cast<unsigned>(j);
  const unsigned item = p.idx_unit == 1 ? uj : p.ps_shift >= 0 ? uj >> p.ps_shift : uj / static_cast<unsigned>(p.page_size);
  return __ldg(r.idx + item);
}
// ... and the row of the cache (in units of H * 128 elements, K part) it stands for, or -1: absent, or a hole in the list.
__device__ __forceinline__ int dec_cache_row(const DecodeParams& p, const DecRow& r, int j, int entry) {
  if (j >= r.n_tokens) return -1;
  const unsigned ps = static_cast<unsigned>(p.page_size), uj = static_cast<unsigned>(j);
  unsigned page, off;
  if (j < r.n_listed && p.idx_unit != 1) {   // whole pages: idx_unit == page_size
    page = static_cast<unsigned>(entry);
    off = p.ps_shift >= 0 ? uj & (ps - 1) : uj % ps;
  } else {
    if (j < r.n_listed && entry < 0) return -1;
    const unsigned slot = j < r.n_listed ? static_cast<unsigned>(entry) : r.tail_slot0 + static_cast<unsigned>(j - r.n_listed);
    page = p.ps_shift >= 0 ? slot >> p.ps_shift : slot / ps;
    off = slot - page * ps;
  }
  return static_cast<int>(page * (2 * ps) + off);
}

// Requests tile `tile` (16 K rows, 16 V rows) into a ring slot and returns the mask of its tokens that exist.  An
// absent token counts with weight 0, but its values still go through P.V and have to be finite: it borrows the row
// of one that exists (a tile without any is skipped by its consumer).
template <typename T>
__device__ __forceinline__ unsigned dec_request(const DecodeParams& p, const DecRow& r, int tile, int entry, const T* kbase,
                                                int64_t row_elems, uint8_t* slot, int lane) {
  int row = dec_cache_row(p, r, tile * kDecTile + (lane & 15), entry);
  const unsigned mask = __ballot_sync(0xffffffffu, row >= 0) & 0xffffu;
  const int safe = __shfl_sync(0xffffffffu, row, mask ? __ffs(mask) - 1 : 0);
  row = max(row >= 0 ? row : safe, 0);
  tile_copy<T>(kbase, p.page_size * row_elems, row_elems, row, slot, lane);
  return mask;
}

// A warp's piece of a row group once more, token by token with fp32 weights, for pieces whose result is not finite: a V row with
// an infinity or a NaN then counts as weight times value does, and not at all where its weight is 0.  `at`: the group's results
// (128 floats each), `ml`: their (max, sum).
template <typename T>
__device__ __noinline__ void dec_plain(const DecodeParams& p, DecRow r, const T* kbase, int64_t row_elems, const T* q, int gsub,
                                       int first, int end, int lane, float* at, float (*ml)[2]) {
  auto row4 = [&](const T* src) {
    const uint2 u = *reinterpret_cast<const uint2*>(src + 4 * lane);
    const float2 a = Elem<T>::to_f2(u.x), b = Elem<T>::to_f2(u.y);
    return make_float4(a.x, a.y, b.x, b.y);
  };
  for (int h = 0; h < gsub; ++h) {
    const float4 qv = row4(q + h * kHeadDim);
    float m = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int tile = first; tile < end; tile += kDecWarps) {
      const int j0 = tile * kDecTile + (lane & 15), rows = dec_cache_row(p, r, j0, dec_list_entry(p, r, j0));
      for (int j = 0; j < kDecTile; ++j) {
        const int row = __shfl_sync(0xffffffffu, rows, j);
        if (row < 0) continue;
        const T* krow = kbase + row * row_elems;
        const float4 k = row4(krow), v = row4(krow + p.page_size * row_elems);
        float s = fmaf(qv.x, k.x, fmaf(qv.y, k.y, fmaf(qv.z, k.z, qv.w * k.w)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        s *= p.scale_log2;
        const float m_new = fmaxf(m, s), base = m_new == -INFINITY ? 0.f : m_new;
        const float rescale = exp2f(m - base), w = exp2f(s - base);
        m = m_new;
        l = fmaf(l, rescale, w);
        if (rescale == 0.f) acc = make_float4(0.f, 0.f, 0.f, 0.f);
        acc.x *= rescale; acc.y *= rescale; acc.z *= rescale; acc.w *= rescale;
        add_weighted(acc, w, v);
      }
    }
    reinterpret_cast<float4*>(at + h * kHeadDim)[lane] = acc;
    if (lane == 0) {
      ml[h][0] = m;
      ml[h][1] = l;
    }
  }
}

struct DecShared {
  float ml[kDecWarps][kDecMaxGroup][2];
  int cum[kDecMaxBatch + 1];     // tiles of the sequences before (batched launches)
  unsigned last;
};

// Dynamic shared memory: the rings, [4 warps][kDecStages][16 K rows, 16 V rows]; a warp parks its results in its own ring.
template <typename T>
__global__ void __launch_bounds__(kDecThreads, kDecBlocksPerSm) paged_decode_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(128) uint8_t dec_smem[];
  __shared__ DecShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  // The index list and the query are the preceding kernels' output (a RoPE-fused append rotates q in place), so
  // nothing of them is touched before the dependency has resolved.  A dense step over a device-resident length is
  // different: the length, the page tables and every cached row but the newest token's were final before the
  // preceding kernel, the append, started, so the first tiles are requested while that one still runs.
  bool waited = p.seq_len_dev == nullptr;
  if (waited) grid_dependency_wait();
  grid_launch_dependents();

  const int rps = p.row_heads * p.subs;   // row groups per sequence
  if (p.seqs) {
    if (warp == 0) {
      int base = 0;
      for (int s0 = 0; s0 < p.batch; s0 += 32) {
        int v = s0 + lane < p.batch ? (__ldg(p.seq_len_dev + s0 + lane) + kDecTile - 1) / kDecTile : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        if (s0 + lane < p.batch) sh.cum[s0 + lane + 1] = base + v;
        base += __shfl_sync(0xffffffffu, v, 31);
      }
      if (lane == 0) sh.cum[0] = 0;
    }
  } else if (tid == 0) {
    sh.cum[0] = 0;
    sh.cum[1] = ((p.seq_len_dev ? __ldg(p.seq_len_dev) : p.n_tokens) + kDecTile - 1) / kDecTile;
  }
  __syncthreads();

  const int total = sh.cum[p.batch] * rps;
  // (with the lengths on the device the work may be far less than the grid was sized for: every piece has tiles)
  const int b = blockIdx.x, B = max(1, min(static_cast<int>(gridDim.x), total / kDecMinTiles));
  auto line_start = [&](int blk) { return static_cast<int>(static_cast<int64_t>(blk) * total / B); };
  auto block_of = [&](int tile) {   // the block whose piece of the line holds `tile`
    int k = static_cast<int>((static_cast<int64_t>(tile) * B) / total);
    while (k + 1 < B && line_start(k + 1) <= tile) ++k;
    return k;
  };

  // (sequences with their lengths on the device are cut as the host cuts those whose lengths it knows, so that neither the
  // result nor the time depends on the capacity)
  const int splits = p.seq_len_dev ? dec_splits(p.batch * rps, (sh.cum[p.batch] + p.batch - 1) / p.batch, p.gs, p.slots) : p.splits;
  if (splits == 0 ? b >= B : b >= p.batch * rps * splits) return;
  int pos = splits > 0 ? 0 : line_start(b);
  const int line_end = splits > 0 ? 1 : line_start(b + 1);
  while (pos < line_end) {
    // ---- this block's next piece: tiles [a, e) of row group x of sequence s ------------------------------
    int s, x, a, e, nparts, part, unit;
    if (splits > 0) {
      const int r = b / splits;
      part = b - r * splits;
      s = r / rps;
      x = r - s * rps;
      const int nt = sh.cum[s + 1] - sh.cum[s];
      a = static_cast<int>(static_cast<int64_t>(nt) * part / splits);
      e = static_cast<int>(static_cast<int64_t>(nt) * (part + 1) / splits);
      nparts = splits;
      unit = b;
      pos = line_end;
    } else {
      int lo = 0, hi = p.batch - 1;
      while (lo < hi) {   // the last sequence that starts at or before pos
        const int mid = (lo + hi + 1) >> 1;
        if (sh.cum[mid] * rps <= pos) lo = mid; else hi = mid - 1;
      }
      s = lo;
      const int nt = sh.cum[s + 1] - sh.cum[s], seq0 = sh.cum[s] * rps;
      x = (pos - seq0) / nt;
      a = pos - seq0 - x * nt;
      e = min(nt, a + line_end - pos);
      const int row0 = seq0 + x * nt;
      const int first = block_of(row0), last = block_of(row0 + nt - 1);
      nparts = last - first + 1;
      part = b - first;
      unit = b + s * rps + x;   // strictly increasing along the line
      pos += e - a;
    }
    const int rh = x / p.subs, sub = x - rh * p.subs;         // row head
    const int gsub = min(p.gs, p.group - sub * p.gs);         // query heads of this part
    const int kv_head = rh / p.row_to_kv;
    const int q_row0 = s * p.q_heads + rh * p.group + sub * p.gs;

    const T* kvp = static_cast<const T*>(p.kv);
    DecRow row;
    row.idx = p.indices + (p.idx_stride ? static_cast<int64_t>(rh * p.group) * p.idx_stride : 0);
    row.n_listed = p.n_listed;
    row.n_tokens = p.n_tokens;
    row.tail_slot0 = p.tail_slot0;
    if (p.seqs) {
      kvp = static_cast<const T*>(p.seqs[s].kv_data);
      row.idx = p.seqs[s].kv_table;
    }
    if (p.seq_len_dev) row.n_tokens = row.n_listed = __ldg(p.seq_len_dev + s);
    const int64_t row_elems = static_cast<int64_t>(p.H) * kHeadDim;
    const T* kbase = kvp + kv_head * kHeadDim;

    TileState st;
    st.m = -INFINITY;
    st.l = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) st.o[j][i] = 0.f;

    uint8_t* ring = dec_smem + warp * kDecStages * kDecTileBytes;
    {
      // tiles a + warp, + kDecWarps, ...: the list entries of a tile are fetched a round before its rows are requested, its
      // rows kDecStages - 1 rounds before they are used
      const int lane_tok = lane & 15;
      int req = a + warp, entry = req < e ? dec_list_entry(p, row, req * kDecTile + lane_tok) : 0;
      unsigned masks[kDecStages - 1];
#pragma unroll
      for (int i = 0; i < kDecStages - 1; ++i) {
        masks[i] = 0;
        if (req < e) {
          const int cur = entry, nxt = req + kDecWarps;
          entry = nxt < e ? dec_list_entry(p, row, nxt * kDecTile + lane_tok) : 0;
          if (!waited && (req + 1) * kDecTile >= row.n_tokens) {   // (the newest token's tile)
            grid_dependency_wait();
            waited = true;
          }
          masks[i] = dec_request<T>(p, row, req, cur, kbase, row_elems, ring + i * kDecTileBytes, lane);
          req = nxt;
        }
        cp_async_commit();
      }
      if (!waited) {
        grid_dependency_wait();
        waited = true;
      }
      // query fragments: head g, dims 32j + 8t .. + 7 (zeros for heads beyond the group)
      uint4 q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        q[j] = g < gsub ? ld_16(static_cast<const T*>(p.q) + static_cast<int64_t>(q_row0 + g) * kHeadDim + j * 32 + t * 8)
                        : make_uint4(0, 0, 0, 0);
      int use = 0, fill = kDecStages - 1;
      for (int tile = a + warp; tile < e; tile += kDecWarps) {
        unsigned mask_new = 0;
        if (req < e) {
          const int cur = entry, nxt = req + kDecWarps;
          entry = nxt < e ? dec_list_entry(p, row, nxt * kDecTile + lane_tok) : 0;
          mask_new = dec_request<T>(p, row, req, cur, kbase, row_elems, ring + fill * kDecTileBytes, lane);
          req = nxt;
        }
        cp_async_commit();
        cp_async_wait<kDecStages - 1>();
        __syncwarp();
        if (masks[0]) {
          float sc[4];
          tile_logits<T>(ring + use * kDecTileBytes, q, masks[0], p.scale_log2, lane, sc);
          tile_softmax_pv<T>(st, ring + use * kDecTileBytes, sc, lane);
        }
        __syncwarp();   // the slot may be filled again
#pragma unroll
        for (int i = 0; i + 1 < kDecStages - 1; ++i) masks[i] = masks[i + 1];
        masks[kDecStages - 2] = mask_new;
        use = use + 1 == kDecStages ? 0 : use + 1;
        fill = fill + 1 == kDecStages ? 0 : fill + 1;
      }
      cp_async_wait<0>();
      __syncwarp();
    }
    // ---- the warps of a head -> one result per query head ---------------------------------------------------
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) st.o[j][i] *= 1.f / Mma<T>::kScale;
    st.l += __shfl_xor_sync(0xffffffffu, st.l, 1);
    st.l += __shfl_xor_sync(0xffffffffu, st.l, 2);
    float* mine = reinterpret_cast<float*>(ring);
    float z = 0.f;   // NaN where a result is not finite
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) z = fmaf(st.o[j][i], 0.f, z);
    if (__any_sync(0xffffffffu, z != z)) {
      dec_plain<T>(p, row, kbase, row_elems, static_cast<const T*>(p.q) + static_cast<int64_t>(q_row0) * kHeadDim, gsub, a + warp, e, lane,
                   mine, sh.ml[warp]);
    } else {
      if (t == 0) {
        sh.ml[warp][g][0] = st.m;
        sh.ml[warp][g][1] = st.l;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int h = 2 * t + i;
        if (h < gsub) {
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            *reinterpret_cast<float4*>(mine + h * kHeadDim + g * 8 + j) =
                make_float4(st.o[j][i], st.o[j + 1][i], st.o[j + 2][i], st.o[j + 3][i]);
            *reinterpret_cast<float4*>(mine + h * kHeadDim + 64 + g * 8 + j) =
                make_float4(st.o[j][2 + i], st.o[j + 1][2 + i], st.o[j + 2][2 + i], st.o[j + 3][2 + i]);
          }
        }
      }
    }
    __syncthreads();
    // a warp takes a query head: four dims per lane
    auto finish = [&](int h, float M, float L, float4 acc) {
      const int out = q_row0 + h;
      const float inv = L > 0.f ? 1.f / L : 0.f;   // nothing attended: zeros and lse = -inf
      acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
      // (results need the alignment of a 32-bit word only; whole vectors where the buffers have theirs)
      if (p.o_f32) {
        float* dst = p.o_f32 + static_cast<int64_t>(out) * kHeadDim + 4 * lane;
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
          *reinterpret_cast<float4*>(dst) = acc;
        } else {
          dst[0] = acc.x; dst[1] = acc.y; dst[2] = acc.z; dst[3] = acc.w;
        }
      }
      if (p.o) {
        uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<T*>(p.o) + static_cast<int64_t>(out) * kHeadDim) + 2 * lane;
        const uint32_t a = Elem<T>::from_f2(acc.x, acc.y), b = Elem<T>::from_f2(acc.z, acc.w);
        if ((reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
          *reinterpret_cast<uint2*>(dst) = make_uint2(a, b);
        } else {
          dst[0] = a; dst[1] = b;
        }
      }
      if (lane == 0 && p.lse) p.lse[out] = L > 0.f ? M + log2f(L) : -INFINITY;
    };
    for (int h = warp; h < gsub; h += kDecWarps) {
      float M = -INFINITY, L = 0.f;
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, sh.ml[w][h][0]);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        const float m = sh.ml[w][h][0];
        const float wt = m == -INFINITY ? 0.f : exp2f(m - M);
        const float4 v = reinterpret_cast<const float4*>(dec_smem + w * kDecStages * kDecTileBytes + h * kHeadDim * 4)[lane];
        L += wt * sh.ml[w][h][1];
        add_weighted(acc, wt, v);
      }
      if (nparts > 1) {
        const int64_t at = static_cast<int64_t>(unit) * p.gs + h;
        __stcg(reinterpret_cast<float4*>(p.partial_o + at * kHeadDim) + lane, acc);
        if (lane == 0) __stcg(reinterpret_cast<float2*>(p.partial_ml) + at, make_float2(M, L));
      } else {
        finish(h, M, L, acc);
      }
    }
    __syncthreads();   // the parked results are read (the rings are free for the next piece), the parts are stored
    if (nparts > 1) {
      unsigned* counter = p.counters + s * rps + x;
      if (tid == 0) {
        unsigned ticket;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(counter) : "memory");
        sh.last = ticket == static_cast<unsigned>(nparts - 1);
      }
      __syncthreads();
      if (sh.last) {
        if (tid == 0) *counter = 0u;
        // a warp takes a query head, or, where those are few, one of `sharing` shares of a head's parts (the append and attention
        // of a single head over 60000 tokens, 296 parts: 41.8 us with one warp at work, 20.5 with four)
        const int sharing = nparts <= 8 || gsub > 2 ? 1 : kDecWarps / gsub;
        for (int h = warp / sharing; h < gsub; h += kDecWarps / sharing) {
          const int64_t at0 = static_cast<int64_t>(unit - part) * p.gs + h;
          float M = -INFINITY, L = 0.f;
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int p0 = warp % sharing * 8; p0 < nparts; p0 += 8 * sharing) {   // eight parts' loads in flight
            float2 ml[8];
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              ml[u] = make_float2(-INFINITY, 0.f);
              v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (p0 + u < nparts) {
                ml[u] = __ldcg(reinterpret_cast<const float2*>(p.partial_ml) + at0 + (p0 + u) * p.gs);
                v[u] = __ldcg(reinterpret_cast<const float4*>(p.partial_o + (at0 + (p0 + u) * p.gs) * kHeadDim) + lane);
              }
            }
            float m_new = M;
#pragma unroll
            for (int u = 0; u < 8; ++u) m_new = fmaxf(m_new, ml[u].x);
            const float r = M == -INFINITY ? 0.f : exp2f(M - m_new);
            L *= r;
            if (r == 0.f) acc = make_float4(0.f, 0.f, 0.f, 0.f);
            acc.x *= r; acc.y *= r; acc.z *= r; acc.w *= r;
            M = m_new;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const float wt = ml[u].x == -INFINITY ? 0.f : exp2f(ml[u].x - M);
              L += wt * ml[u].y;
              add_weighted(acc, wt, v[u]);
            }
          }
          if (sharing == 1) {
            finish(h, M, L, acc);
          } else {   // (one head per warp)
            reinterpret_cast<float4*>(ring)[lane] = acc;
            if (lane == 0) {
              sh.ml[warp][0][0] = M;
              sh.ml[warp][0][1] = L;
            }
          }
        }
        if (sharing > 1) {
          __syncthreads();
          if (warp % sharing == 0) {
            float M = -INFINITY, L = 0.f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w = warp; w < warp + sharing; ++w) M = fmaxf(M, sh.ml[w][0][0]);
            for (int w = warp; w < warp + sharing; ++w) {
              const float m = sh.ml[w][0][0], wt = m == -INFINITY ? 0.f : exp2f(m - M);
              const float4 v = reinterpret_cast<const float4*>(dec_smem + w * kDecStages * kDecTileBytes)[lane];
              L += wt * sh.ml[w][0][1];
              add_weighted(acc, wt, v);
            }
            finish(warp / sharing, M, L, acc);
          }
          __syncthreads();   // (the rings are free for the next piece)
        }
      }
    }
  }
}

// Merge P already-normalised partial results (o_parts [P,H,128] fp32, lse_parts [P,H] base 2).
template <typename T>
__global__ void __launch_bounds__(kHeadDim)
merge_states_kernel(const float* __restrict__ o_parts, const float* __restrict__ lse_parts, int P,
                    int H, T* __restrict__ o, float* __restrict__ lse) {
  const int head = blockIdx.x;
  const int d = threadIdx.x;
  float M = -INFINITY;
  for (int p = 0; p < P; ++p) M = fmaxf(M, lse_parts[static_cast<int64_t>(p) * H + head]);
  float acc = 0.f, den = 0.f;
  for (int p = 0; p < P; ++p) {
    const float l = lse_parts[static_cast<int64_t>(p) * H + head];
    const float w = (l == -INFINITY) ? 0.f : exp2f(l - M);
    den += w;
    if (w != 0.f) acc += w * o_parts[(static_cast<int64_t>(p) * H + head) * kHeadDim + d];
  }
  // every part empty (lse = -inf everywhere): zeros and lse = -inf, as the decode kernel itself writes
  const float r = den > 0.f ? acc / den : 0.f;
  const float r1 = __shfl_down_sync(0xffffffffu, r, 1);
  if ((d & 1) == 0)
    reinterpret_cast<uint32_t*>(o + static_cast<int64_t>(head) * kHeadDim)[d >> 1] =
        Elem<T>::from_f2(r, r1);
  if (d == 0 && lse) lse[head] = den > 0.f ? M + log2f(den) : -INFINITY;
}

}  // namespace adamas
