// Row formats of gemm_tmem.cu: how the 128-element units of a warp's 32 packed weight rows reach its slot in shared memory,
// and how a thread turns the unit of its row into operand values: load() takes the unit from the slot into registers (the
// slot is then free for the next copy), expand() hands out four pieces of 32 values, two to a register.  The arithmetic is
// that of row_expand.cuh, value for value.
//
// The copies are TMA boxes of 32 rows (copy(), issued by one lane): the same bytes by cp.async cost the warp 5 to 16
// instructions per granule column, a sixth of everything it issued.  Boxes 32, 64 or 128 bytes wide take the swizzle of that
// width, others are an odd number of granules wide: either way a lane per row reads 16 bytes without bank conflicts.  Q6_K rows start
// on any even byte, which TMA cannot address: but for rows of a multiple of eight blocks they take the 16-byte cp.async
// of the granules that cover them (a bulk copy per row and run of granules was 1.5 times slower: its requests do not keep up).
#pragma once
#include <cuda.h>

#include "row_expand.cuh"
#include "umma.cuh"

namespace lb {
namespace {

// x / d for the small divisors of group and block sizes: a shift when d is a power of two
struct Div {
  int d, shift;  // shift < 0: divide
  __host__ static Div of(int d) {
    int s = 0;
    while ((1 << s) < d) s++;
    return Div{d, (1 << s) == d ? s : -1};
  }
  __device__ __forceinline__ int operator()(int x) const { return shift >= 0 ? x >> shift : x / d; }
};

// two f32 in one 64-bit register pair: sm_100 adds and multiplies both with one instruction, each rounded as on its own
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2_bits(uint32_t a, uint32_t b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r.v) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(F2 p) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(p.v));
  return pack2<BF16>(a, b);
}

struct Box {  // one tensor map: `bytes` wide at row offset x, or with its own pitch
  int bytes, swizzle;
};
inline CUtensorMapSwizzle swizzle_of(int bytes) {
  return bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
}
// a 32-row box of the (rows, row bytes) matrix: columns x .., rows y ..
__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap *m, uint32_t bar, uint32_t x, int y) {
  umma::tma_load_2d(dst, m, bar, (int)x, y);
}
// 16-byte chunk j of row r in a box of 64 / 128-byte rows under the swizzle of that width
__device__ __forceinline__ uint32_t sw64(int r, int j) { return (uint32_t)(r * 64 + ((j ^ ((r >> 1) & 3)) << 4)); }
__device__ __forceinline__ uint32_t sw128(int r, int j) { return (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)); }
__device__ __forceinline__ void to_words(const uint4 &v, uint32_t *w) { w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w; }

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
template <int N>
__device__ __forceinline__ void lds_words(uint32_t a, uint32_t (&w)[N]) {  // 16-byte aligned, N a multiple of 4
#pragma unroll
  for (int i = 0; i < N / 4; i++) {
    const uint4 v = lds128(a + 16 * i);
    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
  }
}
// N words that start `skew` bytes (even, < 16) into consecutive granules of a slot: whole granules are read (a lane's slot
// is an odd number of granules, so 16-byte reads meet every bank once; single words at lane-dependent skews met four-way
// conflicts) and the words moved down by two selects and one funnel shift.
template <int N>
__device__ __forceinline__ void lds_skewed(uint32_t a, uint32_t skew, uint32_t (&o)[N]) {
  constexpr int W = (N * 4 + 14 + 15) / 16 * 4;
  uint32_t w[W];
  lds_words(a, w);
  const bool s1 = skew & 4u, s2 = skew & 8u;
  const uint32_t sh = (skew & 2u) * 8u;
#pragma unroll
  for (int i = 0; i < N + 3; i++) w[i] = s1 ? (i + 1 < W ? w[i + 1] : 0u) : w[i];
#pragma unroll
  for (int i = 0; i < N + 1; i++) w[i] = s2 ? (i + 2 < W ? w[i + 2] : 0u) : w[i];
#pragma unroll
  for (int i = 0; i < N; i++) o[i] = __funnelshift_r(w[i], w[i + 1], sh);
}

// ---- Q4_K: a unit is the block's 16-byte header and 64 of its 128 code bytes
struct TmQ4K {
  struct Ctx { const uint8_t *w; };
  static constexpr int SLOT = 32 * 80, BYTES = 32 * 80, BOXES = 2;  // codes, then headers
  static constexpr Box BOX[2] = {{64, 64}, {16, 0}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)(K >> 8) * 144; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) {
    tma_rows(slot, m, bar, (uint32_t)((u >> 1) * 144 + 16 + 64 * (u & 1)), y);
    tma_rows(slot + 32 * 64, m + 1, bar, (uint32_t)((u >> 1) * 144), y);
  }
  uint4 h;
  uint32_t q[16];
  __device__ __forceinline__ TmQ4K(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &, int, int) {}
  __device__ __forceinline__ void fetch_scales(const Ctx &, int) {}
  __device__ __forceinline__ void load(uint32_t slot, int) {
    const int r = threadIdx.x & 31;
    h = lds128(slot + 32 * 64 + 16 * r);
#pragma unroll
    for (int j = 0; j < 4; j++) to_words(lds128(slot + sw64(r, j)), q + 4 * j);
  }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int u, Put &&put) const {
    const __half2 dd = bits_h2(h.x);  // (d, dmin)
    const __half2 d2 = __low2half2(dd);
    const float dmin = __high2float(dd);
    // six-bit scales and minimums of the unit's four sub-blocks, one to a byte
    const uint32_t sc = u & 1 ? (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu;
    const uint32_t mn = u & 1 ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;
#pragma unroll
    for (int p = 0; p < 4; p++) {  // sub-block p: the low (p even) or high nibbles of eight code words
      const __half2 s = __half2half2(__uint2half_rn((sc >> (8 * p)) & 63));
      const __half2 c = __hmul2(s, __float2half2_rn(p & 1 ? -64.f : -1024.f));  // exact
      const __half2 nm = __float2half2_rn(-dmin * (float)((mn >> (8 * p)) & 63));
      const uint32_t mask = p & 1 ? 0x00F000F0u : 0x000F000Fu, magic = p & 1 ? 0x54005400u : 0x64006400u;
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {  // word i: k = 4 i .. 4 i + 3 in the order 0, 2, 1, 3
        const uint32_t a = q[8 * (p >> 1) + i];
        o[2 * i] = h2_bits(__hfma2(__hfma2(bits_h2(and_or(a, mask, magic)), s, c), d2, nm));
        o[2 * i + 1] = h2_bits(__hfma2(__hfma2(bits_h2(and_or(a >> 8, mask, magic)), s, c), d2, nm));
      }
      put(p, o);
    }
  }
};

// ---- Q6_K: a unit is half a 210-byte block: of the 14 granules that cover the block, five hold its 64 bytes of ql, three
// its 32 of qh, and the last two the scales
struct Q6KUnit {
  uint32_t ql[16], qh[8], sc[2];
  float d;
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
    const __half2 off = __float2half2_rn(-1056.f);
#pragma unroll
    for (int q = 0; q < 4; q++) {  // group q: nibble q / 2 of ql[32 (q % 2) ..] and bits 2 q of qh, scales 2 q and 2 q + 1 of the half
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const __half2 ds = __float2half2_rn(d * (float)(int8_t)((sc[q >> 1] >> (16 * (q & 1) + 8 * (i >> 2))) & 0xff));
        const uint32_t wq = ql[8 * (q & 1) + i] >> (4 * (q >> 1)), wh = qh[i];
        const uint32_t hi2 = q == 0 ? (wh << 4) : q == 1 ? (wh << 2) : q == 2 ? wh : (wh >> 2);
        const uint32_t v = and_or(wq, 0x0F0F0F0Fu, hi2 & 0x30303030u);
        const uint32_t p02 = __byte_perm(v, 0x64646464u, 0x4240), p13 = __byte_perm(v, 0x64646464u, 0x4341);
        o[2 * i] = h2_bits(__hmul2(__hadd2(bits_h2(p02), off), ds));
        o[2 * i + 1] = h2_bits(__hmul2(__hadd2(bits_h2(p13), off), ds));
      }
      put(q, o);
    }
  }
};

// Rows at any even byte, by cp.async.
struct TmQ6K : Q6KUnit {
  struct Ctx { const uint8_t *w; };
  static constexpr int PITCH = 176, SLOT = 32 * PITCH, BYTES = 0, BOXES = 0;
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)(K >> 8) * 210; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  // granule number (of the 14 that cover the block, the first one holding the block's first byte) of piece i of half h
  static __device__ __forceinline__ int number(int h, int i) { return i < 5 ? 4 * h + i : i < 8 ? 3 + 2 * h + i : 4 + i; }
  uint32_t low;  // low bits of the row's address: a block starts on any even byte
  __device__ __forceinline__ TmQ6K(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &c, int r, int K) { low = (uint32_t)(uintptr_t)(c.w + (size_t)r * stride(K)); }
  __device__ __forceinline__ void fetch_scales(const Ctx &, int) {}
  __device__ __forceinline__ void load(uint32_t slot, int u) {
    slot += (threadIdx.x & 31) * PITCH;
    const uint32_t skew = (low + (uint32_t)(u >> 1) * 210u) & 15u, sh = (skew & 2u) * 8u;
    lds_skewed(slot, skew, ql);
    lds_skewed(slot + 80, skew, qh);
    const uint32_t sa = slot + 128 + 8 * (u & 1) + (skew & ~3u);  // piece 8 holds block bytes 192 ..: the scales, then d
    const uint32_t c0 = lds32(sa), c1 = lds32(sa + 4), c2 = lds32(sa + 8);
    sc[0] = __funnelshift_r(c0, c1, sh), sc[1] = __funnelshift_r(c1, c2, sh);
    uint16_t dh;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(dh) : "r"(slot + 144 + skew));
    d = f16_bits_to_f32(dh);
  }
};

// Rows of a multiple of eight blocks, which start on 16-byte boundaries, by TMA: a block then starts equally far into its first granule in every row,
// so that the words move down by a count that the whole warp shares, and nothing is spent on the addresses and predicates of 11 copies a lane:
// some 130 of 500 instructions that 32 rows x 128 k took, and issue is what bounds these rows.
struct TmQ6KT : Q6KUnit {
  struct Ctx { const uint8_t *w; };
  static constexpr int SLOT = 32 * 160, BYTES = 32 * 160, BOXES = 3;  // ql, qh, scales and d
  static constexpr Box BOX[3] = {{80, 0}, {48, 0}, {32, 32}};
  static __host__ __forceinline__ bool fits(const void *w, int K) { return !((uintptr_t)w & 15) && (K >> 8) % 8 == 0; }
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)(K >> 8) * 210; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) {
    const uint32_t x = ((uint32_t)(u >> 1) * 210u) & ~15u, h = u & 1;
    tma_rows(slot, m, bar, x + 64 * h, y);
    tma_rows(slot + 32 * 80, m + 1, bar, x + 128 + 32 * h, y);
    tma_rows(slot + 32 * 128, m + 2, bar, x + 192, y);
  }
  __device__ __forceinline__ TmQ6KT(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &, int, int) {}
  __device__ __forceinline__ void fetch_scales(const Ctx &, int) {}
  template <int FIRST>  // the word of its first granule that a block starts in
  __device__ __forceinline__ void take(uint32_t slot, uint32_t sh, bool second) {
    const uint32_t r = threadIdx.x & 31;
    uint32_t w[20];
    lds_words(slot + 80 * r, w);
#pragma unroll
    for (int i = 0; i < 16; i++) ql[i] = __funnelshift_r(w[FIRST + i], w[FIRST + i + 1], sh);
    uint32_t v[12];
    lds_words(slot + 32 * 80 + 48 * r, v);
#pragma unroll
    for (int i = 0; i < 8; i++) qh[i] = __funnelshift_r(v[FIRST + i], v[FIRST + i + 1], sh);
    const uint32_t at = slot + 32 * 128 + 32 * r, flip = (r >> 2 & 1) << 4;  // (32-byte swizzle)
    uint32_t g[8];
    to_words(lds128(at + flip), g), to_words(lds128(at + (flip ^ 16)), g + 4);
    const uint32_t c0 = second ? g[FIRST + 2] : g[FIRST], c1 = second ? g[FIRST + 3] : g[FIRST + 1], c2 = second ? g[FIRST + 4] : g[FIRST + 2];
    sc[0] = __funnelshift_r(c0, c1, sh), sc[1] = __funnelshift_r(c1, c2, sh);
    d = f16_bits_to_f32((uint16_t)(g[FIRST + 4] >> sh));
  }
  __device__ __forceinline__ void load(uint32_t slot, int u) {
    const uint32_t skew = ((uint32_t)(u >> 1) * 210u) & 15u, sh = (skew & 2u) * 8u;
    const bool second = u & 1;
    if (skew < 8) {
      if (skew < 4) take<0>(slot, sh, second);
      else take<1>(slot, sh, second);
    } else {
      if (skew < 12) take<2>(slot, sh, second);
      else take<3>(slot, sh, second);
    }
  }
};

// ---- Q8_0: a unit is four 34-byte blocks = 136 bytes, which start 0 or 8 bytes into nine granules
struct TmQ80 {
  struct Ctx { const uint8_t *w; };
  static constexpr int SLOT = 32 * 144, BYTES = 32 * 144, BOXES = 1;
  static constexpr Box BOX[1] = {{144, 0}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)(K >> 5) * 34; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) {
    tma_rows(slot, m, bar, (uint32_t)(u * 136 - 8 * (u & 1)), y);
  }
  uint32_t w[34];
  __device__ __forceinline__ TmQ80(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &, int, int) {}
  __device__ __forceinline__ void fetch_scales(const Ctx &, int) {}
  __device__ __forceinline__ void load(uint32_t slot, int u) {
    uint32_t g[36];
    lds_words(slot + (threadIdx.x & 31) * 144, g);
    const bool odd = u & 1;
#pragma unroll
    for (int i = 0; i < 34; i++) w[i] = odd ? g[i + 2] : g[i];
  }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
    const __half2 off = __float2half2_rn(-1152.f);
#pragma unroll
    for (int p = 0; p < 4; p++) {  // block p starts 34 p bytes in: its codes lie on word boundaries for odd p
      const int qw = (34 * p + 2) / 4;
      const uint32_t dw = w[34 * p / 4];
      const __half2 d2 = p & 1 ? __high2half2(bits_h2(dw)) : __low2half2(bits_h2(dw));
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t raw = p & 1 ? w[qw + i] : __funnelshift_r(w[qw + i], w[qw + i + 1], 16);
        const uint32_t v = raw ^ 0x80808080u;
        const uint32_t p01 = __byte_perm(v, 0x64646464u, 0x5140), p23 = __byte_perm(v, 0x64646464u, 0x7362);
        o[2 * i] = h2_bits(__hmul2(__hadd2(bits_h2(p01), off), d2));
        o[2 * i + 1] = h2_bits(__hmul2(__hadd2(bits_h2(p23), off), d2));
      }
      put(p, o);
    }
  }
};

// ---- 4-bit codes in groups of G (a multiple of 64): 64 bytes; scale and zero point of each half's group
struct TmInt4 {
  struct Ctx {
    const uint32_t *codes;
    const float *s, *z;
    int G;
    Div per;  // 64-element steps of a group
  };
  static constexpr int SLOT = 32 * 64, BYTES = 32 * 64, BOXES = 1;
  static constexpr Box BOX[1] = {{64, 64}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)(K >> 1); }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return reinterpret_cast<const uint8_t *>(c.codes); }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) { tma_rows(slot, m, bar, (uint32_t)(u * 64), y); }
  const float *sr, *zr;
  float ns[2], nz[2], s[2], z[2];  // of the next unit (on their way), of this one
  uint32_t q[16];
  __device__ __forceinline__ TmInt4(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &c, int r, int K) { sr = c.s + (size_t)r * (K / c.G), zr = c.z + (size_t)r * (K / c.G); }
  __device__ __forceinline__ void fetch_scales(const Ctx &c, int u) {
    const int g0 = c.per(2 * u), g1 = c.per(2 * u + 1);
    ns[0] = __ldg(sr + g0), ns[1] = __ldg(sr + g1), nz[0] = __ldg(zr + g0), nz[1] = __ldg(zr + g1);
  }
  __device__ __forceinline__ void load(uint32_t slot, int) {
#pragma unroll
    for (int j = 0; j < 4; j++) to_words(lds128(slot + sw64(threadIdx.x & 31, j)), q + 4 * j);
    s[0] = ns[0], s[1] = ns[1], z[0] = nz[0], z[1] = nz[1];
  }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
    // A code byte under the bits of 2^23 is the f32 2^23 + code.  Zero points are whole numbers (every converter's are), so
    // that 2^23 + z is exact and one subtraction gives code - z; anything else takes the two subtractions one by one.
    const float m0 = 8388608.f + z[0], m1 = 8388608.f + z[1];
    const bool whole = __all_sync(0xffffffffu, m0 - 8388608.f == z[0] && m1 - 8388608.f == z[1]);
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const float zz = z[p >> 1], mz = p >> 1 ? m1 : m0;
      const F2 s2 = f2(s[p >> 1], s[p >> 1]);
      uint32_t o[16];
      auto words = [&](F2 first, F2 second, auto two_steps) {
#pragma unroll
        for (int i = 0; i < 4; i++) {  // a code word: nibbles 0 .. 7 in element order
          const uint32_t lo = q[4 * p + i] & 0x0F0F0F0Fu, hi = (q[4 * p + i] >> 4) & 0x0F0F0F0Fu;  // even / odd nibbles
#pragma unroll
          for (int b = 0; b < 4; b++) {
            F2 m = add2(f2_bits(__byte_perm(lo, 0x4B000000u, 0x7650 + b), __byte_perm(hi, 0x4B000000u, 0x7650 + b)), first);
            if (decltype(two_steps)::value) m = add2(m, second);
            o[4 * i + b] = pack2<BF16>(mul2(s2, m));
          }
        }
      };
      if (whole) words(f2(-mz, -mz), f2(0.f, 0.f), std::false_type{});
      else words(f2(-8388608.f, -8388608.f), f2(-zz, -zz), std::true_type{});
      put(p, o);
    }
  }
};

// ---- block-scaled e4m3
struct TmFp8 {
  struct Ctx {
    const uint8_t *w;
    const float *scale;
    int bR, bC;
    Div per;  // 64-element steps of a block
  };
  static constexpr int SLOT = 32 * 128, BYTES = 32 * 128, BOXES = 1;
  static constexpr Box BOX[1] = {{128, 128}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)K; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) { tma_rows(slot, m, bar, (uint32_t)(u * 128), y); }
  const float *sr;
  float ns[2], s[2];
  uint32_t q[32];
  __device__ __forceinline__ TmFp8(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &c, int r, int K) { sr = c.scale + (size_t)(r / c.bR) * (K / c.bC); }
  __device__ __forceinline__ void fetch_scales(const Ctx &c, int u) { ns[0] = __ldg(sr + c.per(2 * u)), ns[1] = __ldg(sr + c.per(2 * u + 1)); }
  __device__ __forceinline__ void load(uint32_t slot, int) {
#pragma unroll
    for (int j = 0; j < 8; j++) to_words(lds128(slot + sw128(threadIdx.x & 31, j)), q + 4 * j);
    s[0] = ns[0], s[1] = ns[1];
  }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const F2 s2 = f2(s[p >> 1], s[p >> 1]);
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t w = q[8 * p + i];
        __half2_raw a = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xFFFFu), __NV_E4M3);
        __half2_raw b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3);
        const float2 fa = __half22float2(__half2(a)), fb = __half22float2(__half2(b));
        o[2 * i] = pack2<BF16>(mul2(f2(fa.x, fa.y), s2));
        o[2 * i + 1] = pack2<BF16>(mul2(f2(fb.x, fb.y), s2));
      }
      put(p, o);
    }
  }
};

// ---- the same for f16 operands, whole blocks of 128 rows and 128 k under one scale.  A code is exact in f16 and one conversion gives
// two of them; the scale, over a power of two that puts the row block's largest at [64, 128) (the epilogue multiplies by it again), is
// rounded to f16 and so is the product: 2^-11 each at most where the bf16 weight has 2^-8.  Five instructions per four weights
// instead of a dozen through f32: 64 pairs over 64 experts of 4096 x 7168 220 -> 205 us (5.6 TB/s of weights), with 128 tokens to an expert
// 712 -> 694 (there the clock falls with the power), error against 64 bits 2.2e-3 -> 1.66e-3, of which the bf16 output is 1.64e-3.
//
// f16 has the range for that while a row block's scales lie within 2^16 of each other: the smallest normal code then gives 2^-16 and is
// as exact as in bf16.  Experts with scales further apart (zeros aside), or with a token that f16 does not hold, are left to a launch with
// bf16 operands, as above, that follows.
struct TmFp8H {
  struct Ctx {
    const uint8_t *w;
    const float *scale;
    int bR;
    Div per;  // units of a block
    int cols; // blocks of a row
  };
  static constexpr int SLOT = 32 * 128, BYTES = 32 * 128, BOXES = 1;
  static constexpr Box BOX[1] = {{128, 128}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)K; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return c.w; }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) { tma_rows(slot, m, bar, (uint32_t)(u * 128), y); }
  static __device__ __forceinline__ int exponent(const Ctx &c, int r) { return fp8_scale_exponent(c.scale + (size_t)(r / c.bR) * c.cols, c.cols); }
  static __device__ __forceinline__ float unscale(const Ctx &c, int r) { return __uint_as_float((uint32_t)(254 - exponent(c, r)) << 23); }
  const float *sr;
  float mult, ns;
  __half2 s2;
  uint32_t q[32];
  __device__ __forceinline__ TmFp8H(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &c, int r, int) {
    sr = c.scale + (size_t)(r / c.bR) * c.cols;
    mult = __uint_as_float((uint32_t)exponent(c, r) << 23);
  }
  __device__ __forceinline__ void fetch_scales(const Ctx &c, int u) { ns = __ldg(sr + c.per(u)) * mult; }
  __device__ __forceinline__ void load(uint32_t slot, int) {
#pragma unroll
    for (int j = 0; j < 8; j++) to_words(lds128(slot + sw128(threadIdx.x & 31, j)), q + 4 * j);
    s2 = __float2half2_rn(ns);
  }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
#pragma unroll
    for (int p = 0; p < 4; p++) {
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t w = q[8 * p + i];
        o[2 * i] = h2_bits(__hmul2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xFFFFu), __NV_E4M3)), s2));
        o[2 * i + 1] = h2_bits(__hmul2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3)), s2));
      }
      put(p, o);
    }
  }
};
template <typename Row> struct Unscales : std::false_type {};  // rows that carry a power of two less: the epilogue multiplies by unscale()
template <> struct Unscales<TmFp8H> : std::true_type {};
template <typename Row> struct HasModes : std::false_type {};  // rows whose experts may be shared out over two launches
template <> struct HasModes<TmFp8H> : std::true_type {};
template <> struct HasModes<TmFp8> : std::true_type {};

// ---- dense 16-bit rows (nothing to expand: pieces are read from the slot as they are stored)
struct TmDense {
  struct Ctx { const uint16_t *w; };
  static constexpr int SLOT = 32 * 256, BYTES = 32 * 256, BOXES = 1;
  static constexpr Box BOX[1] = {{128, 128}};
  static __host__ __device__ __forceinline__ size_t stride(int K) { return (size_t)K * 2; }
  static __host__ __device__ __forceinline__ const uint8_t *base(const Ctx &c) { return reinterpret_cast<const uint8_t *>(c.w); }
  static __device__ __forceinline__ void copy(uint32_t slot, const CUtensorMap *m, uint32_t bar, int u, int y) {
    tma_rows(slot, m, bar, (uint32_t)(u * 256), y);
    tma_rows(slot + 32 * 128, m, bar, (uint32_t)(u * 256 + 128), y);
  }
  uint32_t slot;
  __device__ __forceinline__ TmDense(const Ctx &) {}
  __device__ __forceinline__ void row(const Ctx &, int, int) {}
  __device__ __forceinline__ void fetch_scales(const Ctx &, int) {}
  __device__ __forceinline__ void load(uint32_t slot_, int) { slot = slot_; }
  template <bool BF16, typename Put>
  __device__ __forceinline__ void expand(int, Put &&put) const {
#pragma unroll
    for (int p = 0; p < 4; p++) {
      uint32_t o[16];
#pragma unroll
      for (int j = 0; j < 4; j++) to_words(lds128(slot + 32 * 128 * (p >> 1) + sw128(threadIdx.x & 31, 4 * (p & 1) + j)), o + 4 * j);
      put(p, o);
    }
  }
};
template <typename Row> struct ReadsLate : std::false_type {};  // rows whose slot is read during expand()
template <> struct ReadsLate<TmDense> : std::true_type {};

}  // namespace
}  // namespace lb
