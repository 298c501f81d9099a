// Stage 1 of the decode path: 128-point Walsh-Hadamard transform, 2-bit bucketize, pack, and the
// append of new keys/values/codes to the paged caches.
//
// Work decomposition: one half-warp (16 lanes) per 128-element row, 8 elements (16 bytes) per lane.
// Butterfly strides 1,2,4 run inside a lane's registers, strides 8..64 through shfl.xor with lane
// masks 1,2,4,8.  Arithmetic is fp32 add/sub in a fixed order plus one multiply, then a round to
// the storage type, so the result is bit-identical to the CPU restatement.  After the transform
// lane w holds dimensions 8w..8w+7, which is exactly packed code word w.
#pragma once
#include "common.cuh"

namespace adamas {

// In-place 128-point WHT over the 16 lanes of a half-warp. `l16` = lane index within the half-warp.
__device__ __forceinline__ void wht128_halfwarp(float (&x)[8], unsigned l16) {
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if ((i & s) == 0) {
        float a = x[i], b = x[i + s];
        x[i] = __fadd_rn(a, b);
        x[i + s] = __fsub_rn(a, b);
      }
    }
  }
#pragma unroll
  for (unsigned m = 1; m < 16; m <<= 1) {
    // lower lane holds a and receives b: a + b; upper lane holds b and receives a: a - b.  Written as
    // one fused multiply-add with a factor of +-1: the product is exact, so the single rounding is that
    // of the plain add or subtract.
    const float sgn = (l16 & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, x[i], m);
      x[i] = __fmaf_rn(x[i], sgn, other);
    }
  }
}

template <typename T>
__device__ __forceinline__ void scale_round(float (&x)[8], float scale) {
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = Elem<T>::round(__fmul_rn(x[i], scale));
}

// 8 values -> one packed word: value i at bits [2i, 2i+1]; bucket = #thresholds strictly below.
__device__ __forceinline__ uint16_t bucketize_pack8(const float (&x)[8], Thresholds th) {
  unsigned w = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    unsigned b = (x[i] > th.t0) + (x[i] > th.t1) + (x[i] > th.t2);
    w |= b << (2 * i);
  }
  return static_cast<uint16_t>(w);
}

// Llama rotary embedding (rotate-half form) of one 128-dim row spread over a half-warp: element e of
// the first half pairs with e + 64, which lives in lane l16 ^ 8.  angle = pos * inv_freq(e % 64) with
// inv_freq(j) = (1 / rope_scale) / theta^(2j/128), all in fp32 as the reference's kernel and the HF
// module compute it (kernels/include/decode/decode_page.cuh:642-690).  The result is rounded to the
// storage type, as the in-place reference operator leaves it.
// With `inv_freq` (64 floats on the device: one rotation frequency per dimension pair, position scaling
// already folded in) the angle is pos * inv_freq[j] and the rotated values are multiplied by `mscale`:
// the form YaRN-scaled models use (per-dimension interpolation ramp, attention factor on cos and sin).
struct RopeParams {
  float rcp_scale;
  float theta;
  const float* inv_freq;
  float mscale;
};

// (cos, sin) of dimension pair j at position pos: the one expression every kernel that rotates a decode
// token uses, so that all of them produce the same bits.
// (In two parts: the frequency does not depend on the position, which may still be on its way from memory.  A table is read where
// the call stands: its maker may be the kernel in front.)
__device__ __forceinline__ float rope_inv_freq(int j, const RopeParams& rp) {
  return rp.inv_freq ? ld_coherent(rp.inv_freq + j) : rp.rcp_scale / powf(rp.theta, static_cast<float>(2 * j) * (1.0f / kHeadDim));
}
__device__ __forceinline__ float2 rope_cos_sin_at(float inv_freq, float pos) {
  float sn, cs;
  sincosf(pos * inv_freq, &sn, &cs);
  return make_float2(cs, sn);
}
__device__ __forceinline__ float2 rope_cos_sin(int j, float pos, const RopeParams& rp) {
  return rope_cos_sin_at(rope_inv_freq(j, rp), pos);
}

// The same rotation with the 64 (cos, sin) pairs of the position given (shared memory): what the decode
// append uses, where every row of the launch sits at the same position.
template <typename T>
__device__ __forceinline__ void rope_halfwarp_cs(float (&x)[8], unsigned l16, const float2* cs_table, bool scaled,
                                                 float mscale) {
  const bool upper = (l16 & 8) != 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float other = __shfl_xor_sync(0xffffffffu, x[i], 8);
    const float2 cs = cs_table[static_cast<int>(l16 & 7) * 8 + i];
    float r = upper ? fmaf(other, cs.y, x[i] * cs.x) : fmaf(-other, cs.y, x[i] * cs.x);
    if (scaled) r *= mscale;
    x[i] = Elem<T>::round(r);
  }
}

// ---- a row spread over 8 lanes -----------------------------------------------------------------------------------
// Pair i of lane l8: dimensions 8 * l8 + i and 64 + 8 * l8 + i, the two of a rotation.  A lane reads two 16-byte chunks, l8 and 8 + l8, and
// every step but the last of the transform works on both halves of a pair at once.  Same operations in the same order as above,
// so the same bits: 28 instructions a row for the transform instead of 44, 18 for the code instead of 38.
template <typename T>
__device__ __forceinline__ void unpack_pairs(uint4 lo, uint4 hi, float2 (&x)[8]) {
  float a[8], b[8];
  unpack8<T>(lo, a);
  unpack8<T>(hi, b);
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = make_float2(a[i], b[i]);
}
// rotation and rounding to the storage type; cs_table: the 64 (cos, sin) pairs of the position
template <typename T>
__device__ __forceinline__ void rope_pairs(float2 (&x)[8], unsigned l8, const float2* cs_table, bool scaled, float mscale) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 cs = cs_table[l8 * 8 + i];
    float a = fmaf(-x[i].y, cs.y, x[i].x * cs.x), b = fmaf(x[i].x, cs.y, x[i].y * cs.x);
    if (scaled) {
      a *= mscale;
      b *= mscale;
    }
    x[i] = make_float2(Elem<T>::round(a), Elem<T>::round(b));
  }
}
template <typename T>
__device__ __forceinline__ void pack_pairs(const float2 (&x)[8], uint4* lo, uint4* hi) {
  const float a[8] = {x[0].x, x[1].x, x[2].x, x[3].x, x[4].x, x[5].x, x[6].x, x[7].x};
  const float b[8] = {x[0].y, x[1].y, x[2].y, x[3].y, x[4].y, x[5].y, x[6].y, x[7].y};
  *lo = pack8<T>(a);
  *hi = pack8<T>(b);
}
__device__ __forceinline__ void wht128_pairs(float2 (&x)[8], unsigned l8) {
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if ((i & s) == 0) {
        const float2 a = x[i], b = x[i + s];
        x[i] = add2(a, b);
        x[i + s] = sub2(a, b);
      }
    }
  }
#pragma unroll
  for (unsigned m = 1; m < 8; m <<= 1) {
    const float sgn = (l8 & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 other = make_float2(__shfl_xor_sync(0xffffffffu, x[i].x, m), __shfl_xor_sync(0xffffffffu, x[i].y, m));
      x[i] = fma2(x[i], make_float2(sgn, sgn), other);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = make_float2(__fadd_rn(x[i].x, x[i].y), __fsub_rn(x[i].x, x[i].y));
}
// The thresholds in the storage type, rounded down: a number of that type is above one exactly where it is above the original.
template <typename T>
struct PairThresholds {
  uint32_t t0, t1, t2;
  __device__ __forceinline__ explicit PairThresholds(const Thresholds& th)
      : t0(Elem<T>::floor2(th.t0)), t1(Elem<T>::floor2(th.t1)), t2(Elem<T>::floor2(th.t2)) {}
};
// How many thresholds each half of v is above, at bits `at` .. (low half) and 16 + 2 + `at` .. (high half).
template <typename T>
__device__ __forceinline__ uint32_t buckets2(uint32_t v, const PairThresholds<T>& th, int at) {
  const uint32_t m0 = Elem<T>::above2(v, th.t0), m1 = Elem<T>::above2(v, th.t1), m2 = Elem<T>::above2(v, th.t2);
  const uint32_t odd = m0 ^ m1 ^ m2, two = (m0 & m1) | (m0 & m2) | (m1 & m2);
  return (odd & (0x00040001u << at)) | (two & (0x00080002u << at));
}
// Transform, scale, round, bucketize: code word l8 in the low half, word 8 + l8 in the high one.
template <typename T>
__device__ __forceinline__ uint32_t code_pairs(float2 (&x)[8], unsigned l8, float scale, const PairThresholds<T>& th) {
  wht128_pairs(x, l8);
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = mul2(x[i], make_float2(scale, scale));
  uint32_t w[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[h] |= buckets2<T>(h == 0 ? Elem<T>::from_f2(x[2 * j].x, x[2 * j + 1].x) : Elem<T>::from_f2(x[2 * j].y, x[2 * j + 1].y), th, 4 * j);
    w[h] |= w[h] >> 16;
  }
  return __byte_perm(w[0], w[1], 0x5410);
}

// In-place rotary embedding of q [seq, Hq, 128] and k [seq, Hk, 128]; token s has position past_len + s.
//
// Bound: HBM (q and k are read and written once).  A block takes kRopeTokens consecutive tokens (one for short
// calls, so that the grid still covers the chip): its 64 (cos, sin) pairs per token are formed once, one pair
// per thread, and shared by all rows of the token.  A power and a sine/cosine per ELEMENT, as the kernel before
// this one had it, was bound by those: 32768 tokens x (32 + 32) heads took 1220 us against 166 us of traffic; 212 us
// with two rows in flight per thread and the pairs of a lane 64 bytes apart in shared memory (bank conflicts), 178 us now.
// Eight lanes per row, each with 8 dimensions of the lower half and their 8 partners of the upper half: no
// exchange between lanes, and every access is a full 128-byte line.
// The rotation, the stand-alone transform and the append of a prompt are programmatic dependent launches: rotation and append of
// 777 tokens (32 query heads over 8), two layers: 20.5 us launched plainly, 16.4 now.  The first two let the kernel behind them
// start only after their own wait, so that whatever it reads early was final before they started.
constexpr int kRopeThreads = 256;
constexpr int kRopeTokens = 4;
constexpr int kRopeRows = 4;      // rows in flight per thread

template <typename T>
__device__ __forceinline__ T* rope_row(T* q, T* k, int64_t tok, int r, int hq, int hk) {
  return r < hq ? q + (tok * hq + r) * kHeadDim : k + (tok * hk + (r - hq)) * kHeadDim;
}

template <typename T>
__global__ void __launch_bounds__(kRopeThreads) rope_kernel(T* q, T* k, int seq, int hq, int hk,
                                                            int past_len, int tokens_per_block, RopeParams rp) {
  constexpr int kRows = kRopeThreads / 8;   // rows per pass of the block
  __shared__ float2 s_cs[kRopeTokens][8][8];   // [token][i][l8]: the pair of element i of lane l8 (no bank conflicts)
  const int tid = threadIdx.x;
  const int l8 = tid & 7;
  const int rows = hq + hk;
  const int64_t tok0 = static_cast<int64_t>(blockIdx.x) * tokens_per_block;
  const int nt = min(tokens_per_block, static_cast<int>(seq - tok0));
  const int all = nt * rows;   // rows of the block: token after token
  const bool scaled = rp.inv_freq != nullptr;
  // kRopeRows rows in flight per thread, the first ones while the table is formed
  T* at[kRopeRows];
  int t[kRopeRows];
  uint4 lo[kRopeRows], hi[kRopeRows];
  auto load = [&](int r0) {
#pragma unroll
    for (int u = 0; u < kRopeRows; ++u) {
      const int r = r0 + u * kRows;
      t[u] = r / rows;
      if (r < all) {
        at[u] = rope_row(q, k, tok0 + t[u], r - t[u] * rows, hq, hk) + l8 * 8;
        lo[u] = ld_16(at[u]);
        hi[u] = ld_16(at[u] + kHeadDim / 2);
      }
    }
  };
  auto form_table = [&]() {
    for (int i = tid; i < nt * (kHeadDim / 2); i += kRopeThreads)
      s_cs[i >> 6][i & 7][(i & 63) >> 3] = rope_cos_sin(i & 63, static_cast<float>(past_len + tok0 + (i >> 6)), rp);
  };
  // (a short call forms the table while the kernel in front ends, a long one while its first rows are on their way; a caller's
  // frequencies may be what the kernel in front writes)
  const bool early = tokens_per_block == 1 && !scaled;
  if (early) form_table();
  grid_dependency_wait();
  grid_launch_dependents();
  int r0 = tid >> 3;
  load(r0);
  if (!early) form_table();
  __syncthreads();
  while (true) {
#pragma unroll
    for (int u = 0; u < kRopeRows; ++u) {
      if (r0 + u * kRows < all) {
        float a[8], b[8];
        unpack8<T>(lo[u], a);
        unpack8<T>(hi[u], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 cs = s_cs[t[u]][i][l8];
          // lower half: x*cos - partner*sin; upper half: x*cos + partner*sin
          float x = fmaf(-b[i], cs.y, a[i] * cs.x);
          float y = fmaf(a[i], cs.y, b[i] * cs.x);
          if (scaled) {
            x *= rp.mscale;
            y *= rp.mscale;
          }
          a[i] = x;
          b[i] = y;
        }
        st_16(at[u], pack8<T>(a));
        st_16(at[u] + kHeadDim / 2, pack8<T>(b));
      }
    }
    r0 += kRopeRows * kRows;
    if (r0 >= all) break;
    load(r0);
  }
}

// y = round(scale * WHT(x)), rows x 128.
template <typename T>
__global__ void __launch_bounds__(256) hadamard_kernel(const T* x, T* y,
                                                       int64_t rows, float scale) {
  const unsigned l16 = threadIdx.x & 15;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
  const bool valid = row < rows;
  float v[8];
  uint4 raw = make_uint4(0, 0, 0, 0);
  grid_dependency_wait();
  grid_launch_dependents();
  if (valid) raw = ld_16(x + row * kHeadDim + l16 * 8);
  unpack8<T>(raw, v);
  wht128_halfwarp(v, l16);
  scale_round<T>(v, scale);
  if (valid) st_16(y + row * kHeadDim + l16 * 8, pack8<T>(v));
}

// codes[row, w] = pack(bucketize(h[row, 8w..8w+7]))
template <typename T>
__global__ void __launch_bounds__(256) bucketize_pack_kernel(const T* __restrict__ h,
                                                             uint16_t* __restrict__ codes,
                                                             int64_t rows, Thresholds th) {
  const unsigned l16 = threadIdx.x & 15;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
  if (row >= rows) return;
  float v[8];
  unpack8<T>(ld_16(h + row * kHeadDim + l16 * 8), v);
  codes[row * kCodeWords + l16] = bucketize_pack8(v, th);
}

struct PagedTarget {
  void* kv_data;
  const int32_t* kv_table;
  uint16_t* code_data;
  const int32_t* code_table;
  int page_size;
  int num_heads;
};

// Decode append: one half-warp per head.  FUSED: qh = q, kh = k and the transform runs here;
// otherwise qh/kh point at rows 0/1 of the pre-transformed h.  Grouped-query attention (FUSED only):
// q has q_heads = group * H rows and the caches H; half-warp i takes query row i and K/V row i, each
// where it exists.  ROPE (needs FUSED): q and k arrive
// un-rotated; they are rotated for position `pos`, written back in place (the attention reads the
// rotated q, the caller's k stays consistent with the cache) and then coded.
// (The rows may be what a rotation or transform in front is still writing when this launch starts, and k and kh are one buffer
// in the FUSED form: no restrict qualifiers, which would let their reads move in front of the wait.)
template <typename T, bool FUSED, bool ROPE = false>
__global__ void __launch_bounds__(256)
append_decode_kernel(T* k, const T* v, T* qh, const T* kh, uint16_t* q_code_out, PagedTarget tgt,
                     int kv_last_page, int kv_entry, int code_last_page, int code_entry, float scale,
                     Thresholds th, float pos, RopeParams rp, const int32_t* seq_len_dev, int q_heads,
                     const SeqDesc* seqs) {
  // The kernel after this one (the estimate) may become resident right away: its producer warps only
  // read the code cache as it was before this step, and its consumers wait for this grid to complete,
  // which in turn waits for the grid before it.  (Two appends to one cache back to back, followed by an
  // estimate, are outside this reasoning: the estimate's early reads could then see the first append's
  // slot unwritten.  A decode step appends once.)
  grid_launch_dependents();
  grid_dependency_wait();
  if (seqs) {
    // a batch of sequences (grid.y = sequence): rows of q, k, v and the query codes are (sequence, head)
    const int b = blockIdx.y;
    tgt.kv_data = seqs[b].kv_data;
    tgt.kv_table = seqs[b].kv_table;
    tgt.code_data = static_cast<uint16_t*>(seqs[b].code_data);
    tgt.code_table = seqs[b].code_table;
    const int64_t kv_rows = static_cast<int64_t>(b) * tgt.num_heads * kHeadDim;
    const int64_t q_rows = static_cast<int64_t>(b) * q_heads * kHeadDim;
    k += kv_rows;
    v += kv_rows;
    kh += FUSED ? kv_rows : 0;
    qh += q_rows;
    q_code_out += static_cast<int64_t>(b) * q_heads * kCodeWords;
    seq_len_dev += b;
  }
  if (seq_len_dev) {
    // the token being appended sits at position *seq_len_dev - 1 of both caches
    const int t = __ldg(seq_len_dev) - 1;
    kv_last_page = code_last_page = t / tgt.page_size;
    kv_entry = code_entry = t - kv_last_page * tgt.page_size;
    pos = static_cast<float>(t);
  }
  // ROPE: the 64 (cos, sin) pairs of the position, once per block (every row of the launch has the same
  // position; a sine/cosine of an angle beyond 1e5 rad takes the slow argument reduction, and eight of them
  // one after the other in every lane cost 6 us per layer at 128K tokens)
  __shared__ float2 s_cs[kHeadDim / 2];
  if (ROPE) {
    if (threadIdx.x < kHeadDim / 2) s_cs[threadIdx.x] = rope_cos_sin(threadIdx.x, pos, rp);
    __syncthreads();
  }
  // physical pages of the slot being written: last entries of the two page tables
  const int kv_page = __ldg(tgt.kv_table + kv_last_page);
  const int code_page = __ldg(tgt.code_table + code_last_page);
  const unsigned l16 = threadIdx.x & 15;
  const int head = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const int H = tgt.num_heads;
  const bool valid = head < H;            // a K/V row of the caches
  const bool valid_q = head < q_heads;    // a query row
  const int hh = valid ? head : 0;
  const int hq = valid_q ? head : 0;
  const int64_t in_off = static_cast<int64_t>(hh) * kHeadDim + l16 * 8;
  const int64_t q_off = static_cast<int64_t>(hq) * kHeadDim + l16 * 8;

  // copy K and V rows into the page slot
  T* kv = static_cast<T*>(tgt.kv_data);
  const int64_t k_off =
      ((static_cast<int64_t>(kv_page) * 2 * tgt.page_size + kv_entry) * H + hh) * kHeadDim + l16 * 8;
  const int64_t v_delta = static_cast<int64_t>(tgt.page_size) * H * kHeadDim;
  uint4 kraw = ld_16(k + in_off);
  uint4 vraw = ld_16(v + in_off);
  float a[8], b[8];
  unpack8<T>(ld_16(qh + q_off), a);
  if (ROPE) {
    unpack8<T>(kraw, b);
    rope_halfwarp_cs<T>(a, l16, s_cs, rp.inv_freq != nullptr, rp.mscale);
    rope_halfwarp_cs<T>(b, l16, s_cs, rp.inv_freq != nullptr, rp.mscale);
    kraw = pack8<T>(b);
    if (valid_q) st_16(qh + q_off, pack8<T>(a));
    if (valid) st_16(k + in_off, kraw);
  }
  if (valid) {
    st_16(kv + k_off, kraw);
    st_16(kv + k_off + v_delta, vraw);
  }

  if (FUSED) {
    unpack8<T>(kraw, b);
    wht128_halfwarp(a, l16);
    wht128_halfwarp(b, l16);
    scale_round<T>(a, scale);
    scale_round<T>(b, scale);
  } else {
    unpack8<T>(ld_16(kh + in_off), b);
  }
  if (valid_q) q_code_out[hq * kCodeWords + l16] = bucketize_pack8(a, th);
  if (valid) {
    const int64_t c_off =
        ((static_cast<int64_t>(code_page) * tgt.page_size + code_entry) * H + hh) * kCodeWords + l16;
    tgt.code_data[c_off] = bucketize_pack8(b, th);
  }
}

// Prefill append: eight lanes per (token, head) row; token n sits at position start_pos + n.  Bound: HBM (K and V read once
// and written once, and the codes); with half-warps per row and the codes element by element it was instructions (32768 tokens x 32 heads,
// us: fp16 199 -> 162, bf16 218 -> 163; 162 without the transform).  (Two or four rows per half-warp in flight, streaming stores, and the rows from the
// last one to the first, behind a rotation that has left its last ones in L2, measured no better.)
// Blocks of 16 rows: a lane's transform is 48 shuffles, and with few rows those of a block's warps are what takes time: us for 32 / 256 /
// 2048 / 16384 rows of 16 heads, a block of 256 threads 1.54 / 1.65 / 1.75 / 3.28, of 128 1.34 / 1.44 / 1.54 / 3.08, of 64 1.34 / 1.44 / 1.54 / 3.20, of 32
// 1.34 / 1.44 / 1.65 / 4.30; half-warps per row in blocks of 256 took 1.24 / 1.44 / 1.54 / 3.90.
constexpr int kPrefillThreads = 128;
template <typename T, bool FUSED>
__global__ void __launch_bounds__(kPrefillThreads)
append_prefill_kernel(const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ h,
                      int64_t rows, int64_t start_pos, PagedTarget tgt, float scale, Thresholds th) {
  const unsigned l8 = threadIdx.x & 7;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  const bool valid = row < rows;
  const int64_t r = valid ? row : 0;
  const int H = tgt.num_heads;
  const int64_t in_off = r * kHeadDim + l8 * 8;
  // (32-bit divisions wherever they hold the numbers: positions are below 2^31)
  const int64_t n = rows <= 0x7fffffff ? static_cast<int64_t>(static_cast<unsigned>(r) / static_cast<unsigned>(H)) : r / H;
  const int head = static_cast<int>(r - n * H);
  const unsigned pos = static_cast<unsigned>(start_pos + n), lp = pos / static_cast<unsigned>(tgt.page_size);
  const int e = static_cast<int>(pos - lp * static_cast<unsigned>(tgt.page_size));
  const PairThresholds<T> pt(th);
  // (Nothing behind this launch is let start before it is done: an estimate reads cached codes before its own wait.)
  grid_dependency_wait();
  const uint4 k0 = ld_stream_16(k + in_off), k1 = ld_stream_16(k + in_off + kHeadDim / 2);
  const uint4 v0 = ld_stream_16(v + in_off), v1 = ld_stream_16(v + in_off + kHeadDim / 2);
  const int64_t kv_page = tgt.kv_table[lp];
  if (valid) {
    T* dst = static_cast<T*>(tgt.kv_data) + ((kv_page * 2 * tgt.page_size + e) * H + head) * kHeadDim + l8 * 8;
    st_16(dst, k0);
    st_16(dst + kHeadDim / 2, k1);
    dst += static_cast<int64_t>(tgt.page_size) * H * kHeadDim;
    st_16(dst, v0);
    st_16(dst + kHeadDim / 2, v1);
  }
  uint16_t c0, c1;
  if (FUSED) {
    float2 x[8];
    unpack_pairs<T>(k0, k1, x);
    const uint32_t w = code_pairs<T>(x, l8, scale, pt);
    c0 = static_cast<uint16_t>(w);
    c1 = static_cast<uint16_t>(w >> 16);
  } else {
    float x[8];
    unpack8<T>(ld_stream_16(h + in_off), x);
    c0 = bucketize_pack8(x, th);
    unpack8<T>(ld_stream_16(h + in_off + kHeadDim / 2), x);
    c1 = bucketize_pack8(x, th);
  }
  if (valid) {
    const int64_t code_page = tgt.code_table[lp];
    uint16_t* dst = tgt.code_data + ((code_page * tgt.page_size + e) * H + head) * kCodeWords + l8;
    dst[0] = c0;
    dst[8] = c1;
  }
}

}  // namespace adamas
