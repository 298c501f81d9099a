// The distance estimate (and decode append) for any head count and for grouped queries; the tile pipeline
// for 16, 32 and 64 heads is in estimate.cuh, with the parameters and the distance arithmetic.
//
// Bound: integer issue (56 instructions, 12 of them population counts at quarter rate, per 32 distances) for grouped
// queries, HBM for long rows, fill and drain for short ones.  One persistent block of 16 warps (8 with little work) per SM;
// every warp works alone:
//   * its unit of work is an item of 4 KB of codes: 128 / HP tokens x HP heads (HP = 4, 2 or 1, the largest that divides
//     the head count).  Its own 16-byte asynchronous copies bring items into its own ring of two or three slots: no
//     producer warp, no barrier between warps.  (A bulk copy with a different address in every lane is issued lane after
//     lane, 45 ns each, which bounded small head counts in a pipeline with producer warps.)
//   * lane = token: a lane reads the two halves of a code (chunk c of row r is stored at c ^ f(r), which makes 32 rows hit
//     different bank groups) and the query's planes from shared memory (all lanes the same address).  With grouped
//     queries the code is read once for all query heads of the cache head, or, with fewer items than warps, once for each
//     of the parts in which several warps take them (item_query_heads).  The 32 lanes store 32 consecutive tokens
//     of one output row.
//   * the distances are counted in shared memory (16-bit counts, two to a word, one table per query row) and added to
//     the global per-slice histograms once per block: one L2 atomic per (block, distance value) instead of one per distance.
// All items of a launch, sequence after sequence, form one line that is cut evenly over the blocks, so sequences of
// different lengths and any head count load all SMs alike (with little work every block keeps to one sequence).  The first items are requested before the kernel's dependency
// resolves (the cached codes are final).
// Measured (with counts): 8 cache heads / 64 query heads, 64K tokens: 31 -> 21 us; 4 heads, 128K: 14.4 -> 7.4 us with the
// append inside; 32 query heads over 8, 30K tokens: 9.3 us before and now; over 2, 16K: 6.8 -> 7.3 (17.9 with
// undivided groups).  Lane = head with four tokens
// per lane (one 4 KB run of codes per warp) was slower than lane = token: 36.9 us.
#pragma once
#include "estimate.cuh"

namespace adamas {

constexpr int kItemWarps = 16;           // warps of a block, or half as many (see the host's rule)
constexpr int kItemThreads = kItemWarps * 32;
constexpr int kItemBytes = 4096;
constexpr int kItemCountWords = 196;     // per query row: 392 16-bit counts (a distance is at most 384)

// Query heads of a cache head that a warp takes at a time.  The group of a cache head is halved as long as every part still
// finds a warp of its own (`warps` on the chip; `items` are those of undivided groups): a second round costs more than it saves
// (32 query heads over 2, 60K tokens: 14.3 us in two parts, one round; 17.9 in three parts, two rounds).
__host__ __device__ __forceinline__ int item_query_heads(int items, int q_group, int warps) {
  int heads = q_group;
  for (; heads > 1 && items <= warps / 2; items *= 2) heads = (heads + 1) / 2;
  return heads;
}

// 128-point transform of a row spread over 8 lanes, 16 elements each: the butterflies of wht128_halfwarp in the
// same order, so the same bits.
__device__ __forceinline__ void wht128_8lanes(float (&x)[16], unsigned l8) {
#pragma unroll
  for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & s) == 0) {
        const float a = x[i], b = x[i + s];
        x[i] = __fadd_rn(a, b);
        x[i + s] = __fsub_rn(a, b);
      }
    }
  }
#pragma unroll
  for (unsigned m = 1; m < 8; m <<= 1) {
    const float sgn = (l8 & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, x[i], m);
      x[i] = __fmaf_rn(x[i], sgn, other);
    }
  }
}

// rope_halfwarp_cs for a row spread over 8 lanes: dimension pairs sit in lanes l and l ^ 4.
template <typename T>
__device__ __forceinline__ void rope_8lanes(float (&x)[16], unsigned l8, const float2* cs_table, bool scaled, float mscale) {
  const bool upper = (l8 & 4) != 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float other = __shfl_xor_sync(0xffffffffu, x[i], 4);
    const float2 cs = cs_table[static_cast<int>(l8 & 3) * 16 + i];
    float r = upper ? fmaf(other, cs.y, x[i] * cs.x) : fmaf(-other, cs.y, x[i] * cs.x);
    if (scaled) r *= mscale;
    x[i] = Elem<T>::round(r);
  }
}

template <typename T>
__device__ __forceinline__ void unpack16(uint4 a, uint4 b, float (&x)[16]) {
  float lo[8], hi[8];
  unpack8<T>(a, lo);
  unpack8<T>(b, hi);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[i] = lo[i];
    x[8 + i] = hi[i];
  }
}

// transform, scale, bucketize: this lane's 32-bit word of the row's code
template <typename T>
__device__ __forceinline__ uint32_t code_word_8lanes(float (&x)[16], unsigned l8, float scale, const Thresholds& th) {
  wht128_8lanes(x, l8);
  float lo[8], hi[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    lo[i] = Elem<T>::round(__fmul_rn(x[i], scale));
    hi[i] = Elem<T>::round(__fmul_rn(x[8 + i], scale));
  }
  return static_cast<uint32_t>(bucketize_pack8(lo, th)) | (static_cast<uint32_t>(bucketize_pack8(hi, th)) << 16);
}

struct EstShared {
  float2 cs[kHeadDim / 2];
  int cum[kEstMaxBatch + 1];   // token tiles of the sequences before
};

// Dynamic shared memory: rings | planes [rows of a sequence][2] | counts [rows][kItemCountWords] (count_local).
// GROUPED: several query heads per cache head (q_group > 1).
template <typename T, int METRIC, int HP, bool GROUPED>
__global__ void __launch_bounds__(kItemThreads, 1) estimate_items_kernel(const EstimateParams p, int slots) {
  constexpr int TT = 128 / HP;          // tokens of an item
  constexpr int kGroups = TT / 32;      // ... in groups of 32
  constexpr int CPR = 2 * HP;           // 16-byte chunks per token of an item
  extern __shared__ __align__(128) uint8_t item_smem[];
  __shared__ EstShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int threads = blockDim.x, warps = threads >> 5;
  const int q_group = GROUPED ? p.q_group : 1;
  const int rows = p.H * q_group;       // query rows of a sequence
  QPlanes* planes = reinterpret_cast<QPlanes*>(item_smem + warps * slots * kItemBytes);
  uint32_t* counts = reinterpret_cast<uint32_t*>(planes + 2 * rows);
  uint4* ring = reinterpret_cast<uint4*>(item_smem + warp * (slots * kItemBytes));

  // ---- the line of items: token tile after token tile, `pieces` each: HP heads with a part of their query heads ---
  int tiles_all;
  if (p.seqs) {
    if (warp == 0) est_line(p, TT, lane, sh.cum);
    __syncthreads();
    tiles_all = sh.cum[p.batch];
  } else {
    tiles_all = est_tiles(p.seq_len_dev ? __ldg(p.seq_len_dev) - 1 : p.n_tokens, TT);
  }
  const int q_part = GROUPED ? item_query_heads(tiles_all * (p.H / HP), q_group, p.chip_warps) : 1;
  const int q_split = q_part == q_group ? 1 : (q_group + q_part - 1) / q_part, pieces = p.H / HP * q_split;
  const float split_inv = 1.f / static_cast<float>(q_split);
  auto heads_of = [&](int piece) { return q_split == 1 ? piece : __float2int_rz((static_cast<float>(piece) + 0.5f) * split_inv); };   // piece / q_split (exact: pieces <= 1024)
  const int total = tiles_all * pieces;   // (below 2^31: checked on the host)
  if (total == 0) return;
  // (with the lengths on the device there may be fewer items than blocks: every block that takes part has some)
  const int b = blockIdx.x, B = min(static_cast<int>(gridDim.x), total);
  auto line_start = [&](int blk) { return static_cast<int>(static_cast<int64_t>(blk) * total / B); };
  int pos, line_end;
  int nblk = B, my_blk = b;   // blocks that share out the appends of a piece's sequence, and which of them this one is
  // A batch with little work: every block takes a piece of ONE sequence, the blocks dealt out in proportion to the items.  (A
  // block that the line takes into a second sequence codes two queries, one after the other, and the launch waits for it:
  // 2 sequences of 1250 and 2500 tokens, 32 query heads over 8: 15.2 us, 9.2 this way.)
  const bool apart = p.seqs && p.batch <= static_cast<int>(gridDim.x) && total <= 2 * p.chip_warps;
  if (apart) {
    const int spare = gridDim.x - p.batch;
    auto first_block = [&](int s) { return s + static_cast<int>(static_cast<int64_t>(sh.cum[s]) * spare / tiles_all); };
    int lo = 0, hi = p.batch - 1;
    while (lo < hi) {   // the last sequence that starts at or before this block
      const int mid = (lo + hi + 1) >> 1;
      if (first_block(mid) <= b) lo = mid; else hi = mid - 1;
    }
    const int seq_items = (sh.cum[lo + 1] - sh.cum[lo]) * pieces;
    nblk = min(first_block(lo + 1) - first_block(lo), seq_items);
    my_blk = b - first_block(lo);
    if (my_blk >= nblk) return;
    pos = sh.cum[lo] * pieces + static_cast<int>(static_cast<int64_t>(seq_items) * my_blk / nblk);
    line_end = sh.cum[lo] * pieces + static_cast<int>(static_cast<int64_t>(seq_items) * (my_blk + 1) / nblk);
  } else {
    if (b >= B) return;
    pos = line_start(b);
    line_end = line_start(b + 1);
  }
  bool waited = false;

  while (pos < line_end) {
    // ---- this block's next piece of a sequence: items [first, end) ------------------------------------------
    int s = 0, seq0 = 0, seq1 = total;
    if (p.seqs) {
      int lo = 0, hi = p.batch - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sh.cum[mid] * pieces <= pos) lo = mid; else hi = mid - 1;
      }
      s = lo;
      seq0 = sh.cum[s] * pieces;
      seq1 = sh.cum[s + 1] * pieces;
    }
    const int end = min(seq1, line_end) - seq0, first = pos - seq0;
    pos = seq0 + end;
    const int n = p.seq_len_dev ? __ldg(p.seq_len_dev + s) - 1 : p.n_tokens;
    const uint4* codes = p.codes;
    const int32_t* table = p.page_table;
    if (p.seqs) {
      codes = static_cast<const uint4*>(p.seqs[s].code_data);
      table = p.seqs[s].code_table;
    }

    // ---- copies -----------------------------------------------------------------------------------------------
    // the page numbers of an item's tokens (lane = token of each group of 32) are fetched one item ahead of its copies
    int item_q = first + warp, tile_q = item_q / pieces, piece_q = item_q - tile_q * pieces;
    const int dt = warps / pieces, dp = warps - dt * pieces;
    auto step = [&](int& tile, int& piece) {
      tile += dt;
      piece += dp;
      if (piece >= pieces) {
        piece -= pieces;
        ++tile;
      }
    };
    int entry[kGroups];
    auto fetch_entries = [&](int tile) {
#pragma unroll
      for (int k = 0; k < kGroups; ++k) {
        const unsigned t = static_cast<unsigned>(min(tile * TT + k * 32 + lane, max(n - 1, 0)));   // (absent tokens: the last one's codes)
        entry[k] = __ldg(table + (p.ps_shift >= 0 ? t >> p.ps_shift : t / static_cast<unsigned>(p.page_size)));
      }
    };
    auto request = [&](int tile, int piece, uint4* slot) {
      int tok[kGroups];
#pragma unroll
      for (int k = 0; k < kGroups; ++k) {
        const unsigned t = static_cast<unsigned>(min(tile * TT + k * 32 + lane, max(n - 1, 0))), ps = static_cast<unsigned>(p.page_size);
        tok[k] = entry[k] * p.page_size + static_cast<int>(p.ps_shift >= 0 ? t & (ps - 1) : t % ps);
      }
      constexpr int RPI = 32 / CPR;   // tokens per copy instruction
      const int c = lane & (CPR - 1), r0 = lane / CPR;
      const uint4* base = codes + heads_of(piece) * CPR + c;
      const int64_t stride = 2 * p.H;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * RPI + r0;   // r / 32 == i * RPI / 32
        const int slot_of = __shfl_sync(0xffffffffu, tok[i * RPI / 32], r & 31);
        const int f = HP == 4 ? (r & 7) : HP == 2 ? ((r >> 1) & 3) : ((r >> 2) & 1);
        cp_async_16(slot + r * CPR + (c ^ f), base + slot_of * stride);
      }
    };
    auto request_next = [&](int slot) {
      if (item_q < end) {
        request(tile_q, piece_q, ring + slot * (kItemBytes / 16));
        step(tile_q, piece_q);
        item_q += warps;
        if (item_q < end) fetch_entries(tile_q);
      }
      cp_async_commit();
    };
    int tile_u = tile_q, piece_u = piece_q;   // the item in use
#pragma unroll
    for (int k = 0; k < kGroups; ++k) entry[k] = 0;
    if (item_q < end) fetch_entries(tile_q);
    for (int i = 0; i < slots; ++i) request_next(i);

    // ---- the sequence's query: codes, planes; the new token's rows ---------------------------------------------
    if (p.ap.rope_on) {
      // the new token sits at position n (= tokens before it)
      if (tid < kHeadDim / 2) sh.cs[tid] = rope_cos_sin(tid, static_cast<float>(n), p.ap.rp);
    }
    if (p.count_local)
      for (int i = tid; i < rows * (kItemCountWords / 4); i += threads) reinterpret_cast<uint4*>(counts)[i] = make_uint4(0, 0, 0, 0);
    if (p.ap.rope_on) __syncthreads();
    if (!waited) {
      grid_dependency_wait();   // q, k, v or the query codes are the preceding kernel's output
      grid_launch_dependents();
      waited = true;
    }
    if (p.ap.q) {
      const StepAppend& ap = p.ap;
      const unsigned l8 = lane & 7;
      const bool scaled = ap.rp.inv_freq != nullptr;
      if (p.seqs && !apart) {
        auto block_of = [&](int item) {
          int k = static_cast<int>(static_cast<int64_t>(item) * B / total);
          while (line_start(k + 1) <= item) ++k;
          return k;
        };
        const int bf = block_of(seq0);
        nblk = block_of(seq1 - 1) - bf + 1;
        my_blk = b - bf;
      }
      for (int r0 = 0; r0 < rows; r0 += threads / 8) {
        if (r0 + warp * 4 >= rows) break;   // (warp-uniform)
        const int r = r0 + (tid >> 3);
        const bool live = r < rows;
        const T* src = static_cast<const T*>(ap.q) + (static_cast<int64_t>(s) * rows + (live ? r : 0)) * kHeadDim + l8 * 16;
        float x[16];
        unpack16<T>(ld_16(src), ld_16(src + 8), x);
        if (ap.rope_on) rope_8lanes<T>(x, l8, sh.cs, scaled, ap.rp.mscale);
        const uint32_t w = code_word_8lanes<T>(x, l8, ap.scale, ap.th);
        if (live) {
          uint32_t* qp = reinterpret_cast<uint32_t*>(planes + 2 * r + (l8 >> 2)) + (l8 & 3);
          qp[0] = w;
          qp[4] = qplane_d(w);
          if ((r / q_group) % nblk == my_blk)
            reinterpret_cast<uint32_t*>(ap.q_code_out)[(static_cast<int64_t>(s) * rows + r) * (kCodeWords / 2) + l8] = w;
        }
      }
      for (int h = my_blk + nblk * (tid >> 3); h - nblk * ((tid >> 3) & 3) < p.H; h += nblk * (threads / 8)) {
        // (warp-uniform trip count: the four rows of a warp advance together)
        const bool live = h < p.H;
        const int64_t in_off = (static_cast<int64_t>(s) * p.H + (live ? h : 0)) * kHeadDim + l8 * 16;
        T* ksrc = static_cast<T*>(ap.k) + in_off;
        const T* vsrc = static_cast<const T*>(ap.v) + in_off;
        uint4 k0 = ld_16(ksrc), k1 = ld_16(ksrc + 8);
        const uint4 v0 = ld_16(vsrc), v1 = ld_16(vsrc + 8);
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
        float x[16];
        unpack16<T>(k0, k1, x);
        if (ap.rope_on) {
          rope_8lanes<T>(x, l8, sh.cs, scaled, ap.rp.mscale);
          const float a[8] = {x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]};
          const float c[8] = {x[8], x[9], x[10], x[11], x[12], x[13], x[14], x[15]};
          k0 = pack8<T>(a);
          k1 = pack8<T>(c);
          if (live) {
            st_16(ksrc, k0);
            st_16(ksrc + 8, k1);
          }
        }
        const uint32_t w = code_word_8lanes<T>(x, l8, ap.scale, ap.th);
        if (live) {
          T* dst = static_cast<T*>(tgt.kv_data) + ((kv_page * 2 * ps + kv_entry) * p.H + h) * kHeadDim + l8 * 16;
          st_16(dst, k0);
          st_16(dst + 8, k1);
          dst += static_cast<int64_t>(ps) * p.H * kHeadDim;
          st_16(dst, v0);
          st_16(dst + 8, v1);
          reinterpret_cast<uint32_t*>(tgt.code_data)[((code_page * ps + code_entry) * p.H + h) * (kCodeWords / 2) + l8] = w;
        }
      }
    } else {
      for (int c = tid; c < 2 * rows; c += threads) planes[c] = make_qplanes(__ldg(p.q_code + static_cast<int64_t>(s) * 2 * rows + c));
    }
    __syncthreads();   // planes and zeroed counts are visible

    // ---- scan -----------------------------------------------------------------------------------------------------
    const int slice_tokens = p.hist ? 8 * sa_granules_per_block(max(n, 1), p.hist_cl) : 1;
    // the counts in shared memory are those of the slice in which this piece starts; tokens of later slices (few, unless
    // the sequences are far shorter than a block's share) are counted in global memory one by one
    const int slice0 = p.hist ? first / pieces * TT / slice_tokens : 0;
    // (a 16-bit count must not overflow)
    const int slice0_end = p.count_local ? min((slice0 + 1) * slice_tokens, first / pieces * TT + 65504) : 0;
    uint32_t* hist = p.hist ? p.hist + static_cast<size_t>(s) * rows * kSaScratchWordsPerHead : nullptr;
    uint16_t* out = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(s) * rows * p.out_stride;
    auto to_out = [&](unsigned d) { return p.out_half ? __half_as_ushort(__uint2half_rn(d)) : static_cast<uint16_t>(d); };   // (exact: d <= 384)
    auto count_here = [&](int r, unsigned d) { atomicAdd(counts + r * kItemCountWords + (d >> 1), 1u << ((d & 1) * 16)); };
    auto count_there = [&](int r, int t0, unsigned d) { hist_count(hist, r, t0 / slice_tokens, d); };
    const int f = HP == 4 ? (lane & 7) : HP == 2 ? ((lane >> 1) & 3) : ((lane >> 2) & 1);
    int use = 0;
    for (int item = first + warp; item < end; item += warps) {
      if (slots == 3) cp_async_wait<2>(); else if (slots == 2) cp_async_wait<1>(); else cp_async_wait<0>();
      __syncwarp();
      const uint4* lrow = ring + use * (kItemBytes / 16) + lane * CPR;
      if (!GROUPED) {
        const int r_first = piece_u * HP;                        // first query row of the item
        const QPlanes* qp0 = planes + 2 * r_first;
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
          const int t0 = tile_u * TT + k * 32, t = t0 + lane;
          unsigned d[HP];
#pragma unroll
          for (int hh = 0; hh < HP; ++hh)
            d[hh] = chunk_distance<METRIC>(lrow[k * 32 * CPR + ((2 * hh) ^ f)], qp0[2 * hh]) +
                    chunk_distance<METRIC>(lrow[k * 32 * CPR + ((2 * hh + 1) ^ f)], qp0[2 * hh + 1]);
          if (t < n) {
            uint16_t* o = out + r_first * p.out_stride + t;
#pragma unroll
            for (int hh = 0; hh < HP; ++hh) {
              *o = to_out(d[hh]);
              o += p.out_stride;
            }
            if (t0 < slice0_end) {   // (a group never straddles two slices)
#pragma unroll
              for (int hh = 0; hh < HP; ++hh) count_here(r_first + hh, d[hh]);
            } else if (hist) {
#pragma unroll
              for (int hh = 0; hh < HP; ++hh) count_there(r_first + hh, t0, d[hh]);
            }
          }
        }
      } else {
        // grouped queries: a code is read once for the item's query heads of its cache head
        auto grouped = [&](int r_first, int heads) {
#pragma unroll
          for (int k = 0; k < kGroups; ++k) {
            const int t0 = tile_u * TT + k * 32, t = t0 + lane;
#pragma unroll
            for (int hh = 0; hh < HP; ++hh) {
              const uint4 k0 = lrow[k * 32 * CPR + ((2 * hh) ^ f)], k1 = lrow[k * 32 * CPR + ((2 * hh + 1) ^ f)];
              const int r1 = r_first + hh * q_group;
              uint16_t* o = out + r1 * p.out_stride + t;
#pragma unroll 4
              for (int g = 0; g < heads; ++g) {
                const int r = r1 + g;
                const unsigned d = chunk_distance<METRIC>(k0, planes[2 * r]) + chunk_distance<METRIC>(k1, planes[2 * r + 1]);
                if (t < n) {
                  *o = to_out(d);
                  if (t0 < slice0_end) count_here(r, d);
                  else if (hist) count_there(r, t0, d);
                }
                o += p.out_stride;
              }
            }
          }
        };
        if (q_split == 1) {
          grouped(piece_u * HP * q_group, q_group);   // (a trip count that is the same for all warps)
        } else {
          const int heads0 = heads_of(piece_u), g0 = (piece_u - heads0 * q_split) * q_part;
          grouped(heads0 * HP * q_group + g0, min(q_part, q_group - g0));
        }
      }
      __syncwarp();   // the slot may be filled again
      request_next(use);
      step(tile_u, piece_u);
      if (++use == slots) use = 0;
    }
    cp_async_wait<0>();
    if (p.hist || pos < line_end) __syncthreads();
    if (p.count_local) {
      uint32_t* dst = hist + slice0 * kSaBins;
      for (int i = tid; i < rows * (kItemCountWords / 4); i += threads) {
        const uint4 c4 = reinterpret_cast<const uint4*>(counts)[i];
        if (c4.x | c4.y | c4.z | c4.w) {
          const int r = i / (kItemCountWords / 4);
          uint32_t* at = dst + static_cast<size_t>(r) * kSaScratchWordsPerHead + (i - r * (kItemCountWords / 4)) * 8;
          const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            if (c[w] & 0xffffu) atomicAdd(at + 2 * w, c[w] & 0xffffu);
            if (c[w] >> 16) atomicAdd(at + 2 * w + 1, c[w] >> 16);
          }
        }
      }
      if (pos < line_end) __syncthreads();   // the counts may be cleared for the next sequence
    }
  }
}

}  // namespace adamas
