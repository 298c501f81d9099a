// A warp's attention over a tile of 16 (select+attend: up to 24) gathered K and V rows, on the tensor cores (mma.sync m16n8k16, fp32
// accumulation): up to 8 query rows at once.  Used by the decode attention (all query heads of a cache head) and by
// select+attend (one query row: q.K only).
//
// The order of the 128 dimensions is free in q.K, and of the output rows in P.V, so every lane reads whole 16-byte
// chunks: chunk 4j + t of K rows g and g + 8, chunks g and 8 + g of V rows 2t, 2t + 1, 2t + 8, 2t + 9 (g = lane / 4,
// t = lane % 4).  Chunk c of row r is stored at c ^ tile_swizzle(r), which makes both patterns free of bank conflicts.
// P enters P.V as a sum of 16-bit numbers (its rounding, the rounding of the remainder, ...) that holds what fp32 arithmetic
// keeps: for fp16 rows two of 11 bits each, of 2^15 P, so that weights far below the maximum stay clear of fp16's lower end,
// 2^-24 (no weight is off by more than 2^-40 of the largest; without the factor a token at the maximum and 131072 at 2^-25 of it
// lost the 0.4 % that these make up); for bf16 rows three of 8 bits.  The products of a tile are added to those of the
// tiles before by ordinary fp32 additions: the matrix instruction cuts off what it adds to its accumulator instead of
// rounding it.  Error of the 32-bit result against 64 bits, attention over 32768 tokens x 32 heads: 2e-6 to 6e-6 with the sum
// left in the accumulators, 1e-7 to 5e-7 this way and with fp32 multiply-adds alike.
#pragma once
#include "common.cuh"

namespace adamas {

constexpr int kTileRows = 16;
constexpr int kTileBytes = 2 * kTileRows * kHeadDim * 2;   // 16 K rows, 16 V rows

template <typename T>
struct Mma;
template <>
struct Mma<__half> {
  static constexpr float kScale = 32768.f;   // of P in P.V (fp16 ends at 65504)
  static constexpr int kParts = 2;
  static __device__ __forceinline__ void run(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <>
struct Mma<__nv_bfloat16> {
  static constexpr float kScale = 1.f;
  static constexpr int kParts = 3;
  static __device__ __forceinline__ void run(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

// State of a warp over the tiles it has seen: head g = lane / 4 in m, l (l: this lane's tokens only);
// o[j]: kScale times output dims (8g' + j, 64 + 8g' + j) of heads 2t, 2t + 1 with g' = lane / 4 (the C fragment of P.V).
struct TileState {
  float m, l;
  float o[8][4];
};

// acc += w v; nothing where w is 0, whatever v is.
__device__ __forceinline__ void add_weighted(float4& acc, float w, float4 v) {
  if (w != 0.f) {
    acc.x = fmaf(w, v.x, acc.x);
    acc.y = fmaf(w, v.y, acc.y);
    acc.z = fmaf(w, v.z, acc.z);
    acc.w = fmaf(w, v.w, acc.w);
  }
}

__device__ __forceinline__ int tile_swizzle(int r) { return (r & 6) ^ ((r & 1) << 2); }

__device__ __forceinline__ uint32_t word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Requests a tile's K and V rows with 16-byte asynchronous copies: lane l holds the cache row of token l (of 16 tokens:
// lanes l and l + 16), in units of row_elems elements behind kbase; its V row lies v_delta elements behind its K row.
template <typename T>
__device__ __forceinline__ void tile_copy(const T* kbase, int64_t v_delta, int64_t row_elems, int row, uint8_t* slot, int lane) {
  const int half = lane >> 4, c = lane & 15;
#pragma unroll
  for (int i = 0; i < kTileRows / 2; ++i) {   // a half-warp per row
    const int rr = 2 * i + half;
    const T* src = kbase + __shfl_sync(0xffffffffu, row, rr) * row_elems + c * 8;
    uint8_t* dst = slot + rr * 256 + ((c ^ tile_swizzle(rr)) << 4);
    cp_async_16(dst, src);
    cp_async_16(dst + kTileRows * 256, src + v_delta);
  }
}

// 8 rows of one kind (select+attend): lane l holds the cache row of token l, in units of row_bytes
// behind `base`; the copies go behind `slot`.  FIRST: which 8.
template <int FIRST>
__device__ __forceinline__ void tile_copy8(const uint8_t* base, uint32_t row_bytes, int row, uint8_t* slot, int lane) {
  const int half = lane >> 4, c = lane & 15;
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // a half-warp per row
    const int rr = FIRST + 2 * i + half;
    const uint32_t r = static_cast<uint32_t>(__shfl_sync(0xffffffffu, row, rr));
    cp_async_16(slot + rr * 256 + ((c ^ tile_swizzle(rr)) << 4), base + static_cast<uint64_t>(r) * row_bytes + c * 16);
  }
}

// Scaled logits of a tile: s[2u], s[2u + 1] are head g's for tokens 8u + 2t, 8u + 2t + 1; -inf for tokens
// outside `mask`.
template <typename T>
__device__ __forceinline__ void tile_logits(const uint8_t* slot, const uint4 (&q)[4], unsigned mask, float scale_log2, int lane,
                                            float (&s)[kTileRows / 4]) {
  constexpr int ROWS = kTileRows;
  const int g = lane >> 2, t = lane & 3;
  float c[ROWS / 8][2][4] = {};   // (two accumulators per 8 rows: shorter chains)
  const uint8_t* krow = slot + g * 256;
  const int ksw = tile_swizzle(g);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int u = 0; u < ROWS / 8; ++u) {
      const uint4 k = *reinterpret_cast<const uint4*>(krow + u * 2048 + (((4 * j + t) ^ ksw) << 4));
      Mma<T>::run(c[u][0], q[j].x, 0u, q[j].y, 0u, k.x, k.y);
      Mma<T>::run(c[u][1], q[j].z, 0u, q[j].w, 0u, k.z, k.w);
    }
  }
#pragma unroll
  for (int u = 0; u < ROWS / 4; ++u) {
    const int tok = 8 * (u >> 1) + 2 * t + (u & 1);
    s[u] = (mask >> tok) & 1u ? (c[u >> 1][0][u & 1] + c[u >> 1][1][u & 1]) * scale_log2 : -INFINITY;
  }
}

// The same for one query row and the first `rem` tokens (8 at a time; ROWS at most).
template <typename T, int ROWS>
__device__ __forceinline__ void tile_logits8(const uint8_t* slot, const uint4 (&q)[4], int rem, float scale_log2, int lane, float (&s)[ROWS / 4]) {
  const int g = lane >> 2, t = lane & 3;
  const uint8_t* krow = slot + g * 256;
  const int ksw = tile_swizzle(g);
#pragma unroll
  for (int u = 0; u < ROWS / 8; ++u) {
    s[2 * u] = s[2 * u + 1] = -INFINITY;
    if (u == 0 || rem > 8 * u) {
      float c[2][4] = {};   // (two accumulators: shorter chains)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 k = *reinterpret_cast<const uint4*>(krow + u * 2048 + (((4 * j + t) ^ ksw) << 4));
        Mma<T>::run(c[0], q[j].x, 0u, q[j].y, 0u, k.x, k.y);
        Mma<T>::run(c[1], q[j].z, 0u, q[j].w, 0u, k.z, k.w);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (8 * u + 2 * t + i < rem) s[2 * u + i] = (c[0][i] + c[1][i]) * scale_log2;
    }
  }
}

// Softmax in base 2 and P.V over a tile of 16 tokens; at least one token must exist, and absent ones must hold the row of one that
// does.  A V row with an infinity or a NaN ends as a NaN whatever its weight is (the matrix form multiplies it by every part
// of every weight, zeros and negative ones among them): the caller looks for that at the end.
template <typename T>
__device__ __forceinline__ void tile_softmax_pv(TileState& st, const uint8_t* slot, const float (&s)[4], int lane) {
  const int g = lane >> 2, t = lane & 3;
  uint4 v[4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int rr = 2 * t + (u & 1) + 8 * (u >> 1);
    const uint8_t* vrow = slot + kTileRows * 256 + rr * 256;
#pragma unroll
    for (int h = 0; h < 2; ++h) v[u][h] = *reinterpret_cast<const uint4*>(vrow + (((g + 8 * h) ^ tile_swizzle(rr)) << 4));
  }
  float m_new = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
  m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 1));
  m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 2));
  m_new = fmaxf(m_new, st.m);
  if (__any_sync(0xffffffffu, m_new > st.m)) {
    const float r = (st.m == -INFINITY) ? 0.f : exp2f(st.m - m_new);
    st.l *= r;
    st.m = m_new;
    const float r0 = __shfl_sync(0xffffffffu, r, 8 * t), r1 = __shfl_sync(0xffffffffu, r, 8 * t + 4);   // heads 2t, 2t + 1
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      st.o[j][0] *= r0;
      st.o[j][1] *= r1;
      st.o[j][2] *= r0;
      st.o[j][3] *= r1;
    }
  }
  float pr[4];
  const float base = st.m == -INFINITY ? 0.f : st.m;   // (no logit above -inf so far: no weight)
#pragma unroll
  for (int u = 0; u < 4; ++u) pr[u] = exp2f(s[u] - base);   // (a masked token: exp2(-inf) = 0)
  st.l += (pr[0] + pr[1]) + (pr[2] + pr[3]);
  // B fragments of P.V: tokens 2t, 2t + 1 and 2t + 8, 2t + 9 of head g
  uint32_t b[Mma<T>::kParts][2];
#pragma unroll
  for (int u = 0; u < 4; ++u) pr[u] *= Mma<T>::kScale;
#pragma unroll
  for (int i = 0; i < Mma<T>::kParts; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      b[i][h] = Elem<T>::from_f2(pr[2 * h], pr[2 * h + 1]);
      const float2 f = Elem<T>::to_f2(b[i][h]);
      pr[2 * h] -= f.x;
      pr[2 * h + 1] -= f.y;
    }
  }
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    uint32_t a[2][4];   // [even / odd dimension of the word][a0 .. a3]
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // rows g (dims 8g ..) and g + 8 (dims 64 + 8g ..)
      const uint32_t v0 = word_of(v[0][h], w), v1 = word_of(v[1][h], w);
      const uint32_t v2 = word_of(v[2][h], w), v3 = word_of(v[3][h], w);
      a[0][h] = __byte_perm(v0, v1, 0x5410);
      a[1][h] = __byte_perm(v0, v1, 0x7632);
      a[0][2 + h] = __byte_perm(v2, v3, 0x5410);
      a[1][2 + h] = __byte_perm(v2, v3, 0x7632);
    }
    float c[2][4] = {};
#pragma unroll
    for (int i = Mma<T>::kParts - 1; i >= 0; --i)   // (the small parts first)
#pragma unroll
      for (int e = 0; e < 2; ++e) Mma<T>::run(c[e], a[e][0], a[e][1], a[e][2], a[e][3], b[i][0], b[i][1]);
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int i = 0; i < 4; ++i) st.o[2 * w + e][i] += c[e][i];
  }
}

}  // namespace adamas
