// Batched decode, 9 to 64 activation rows (tokens) of Q4_K and Q6_K: the weights go through TENSOR MEMORY as WHOLE NUMBERS.
//
// What bounds the token tiles on mma.sync (gguf_decode_nt.cu): they expand a weight in registers once per warp and multiply by the legacy
// tensor path, which holds the pipe 8 clocks per 16 x 16 x 8; neither pipe nor issue is half busy, and time grows with the tokens
// (28672 x 4096: 42.6 us with 32, 67.5 with 64).  gemm_tmem.cu expands a weight once for all tokens and lets one tcgen05.mma take 128 x
// 16 x 64, but rounds d sc q - dmin m to 11 bits, which this path does not.  Here the operand is sc q, exact in f16 (Q6_K: f16(sc
// (code - 32)), as the token tiles have it); d, one per row and 256 k, multiplies the block's f32 sums on their way out of tensor memory; and the minimums
// are one more MMA per 128 k into sums of their own: -dmin m as f16 hi and lo against the sub-blocks' sums of x as f16 hi and lo.
//
//   warps 0-15   expanders, as gemm_tmem.cu's: the four warps w, w + 4, .. own rows 32 (w & 3) .. + 31, set w / 4 has every fourth unit of 128 k
//                (sets 0 and 2 the first halves of blocks, 1 and 3 the second).
//   warps 16-17  one lane of each: TMA of the tokens, half a block each; the second one also their sub-blocks' sums.
//   warp  18     MMAs and commits, a block at a time (half a block at a time a pass has the same looks at barriers for half the work).  18 MMAs of 32 columns
//                are 290 clocks of the tensor pipe; beside the expanders' instructions they take some 750 to issue, of 1400 to 1500 a block (with
//                operands in vector registers 900 whatever their columns: same(), tmem_ops.cuh).
//   warps 19-26  drain: row quarter w & 3 and every second chunk of 16 tokens; per block sums += d x D; at a tile's end the minimums'
//                sums are added and the tile leaves, or is left for, or put together from, the runs it is cut into.
//
// Work is the list of (tile of 128 rows, block of 256 k), cut into equal runs, one per CTA; parts of tiles as in gemm_tmem.cu.
#include <cuda.h>

#include "common.cuh"
#include "mma_sync.cuh"
#include "tmem_ops.cuh"
#include "tmem_rows.cuh"
#include "umma.cuh"

namespace lb {
namespace {

constexpr int EXPANDERS = 16, TMA_WARP = 16, MMA_WARP = 18, DRAIN_WARP = 19, DRAINS = 8, THREADS = 27 * 32;
constexpr int NBS = 4;                        // most blocks of tokens on their way (of weights: two)
constexpr int MAX_NT = 64;
// tensor memory: buffers of a block's sums (two, or four where 32 columns are enough), the minimums' sums, the minimums (8 columns per
// half block), the weights
constexpr int P_COL = 2 * MAX_NT, M_COL = 3 * MAX_NT, A_COL = 256;
constexpr int BAR_BYTES = 512;
constexpr int PART_FLOATS = MAX_NT * 128;     // one partial tile: [token][row]

__device__ int g_status;                      // non-zero: a bounded wait gave up (sticky)
__device__ Sync g_sync;                       // a flag per (CTA, drain warp)

struct Args {
  int M, N, K, nt;            // nt: tokens of a tile, a multiple of 16
  int stage_bytes, stages;    // of the tokens
  int bufs;                   // buffers of a block's sums: a power of two
  float *parts;
};
struct Maps {
  CUtensorMap x, sums, w[3];
};

// D[tmem] += A[tmem] x B[smem], with B a tile of 16 k in the 32-byte swizzle
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)6 << 61;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]),
               "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ---- rows: as in tmem_rows.cuh, but whole numbers, d apart
struct ExQ4K : TmQ4K {
  static constexpr bool MINS = true;
  __device__ __forceinline__ ExQ4K(const Ctx &c) : TmQ4K(c) {}
  __device__ __forceinline__ float scale() const { return __low2float(bits_h2(h.x)); }
  template <typename Put>
  __device__ __forceinline__ void whole(int u, Put &&put) const {
    const uint32_t sc = u & 1 ? (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const __half2 s = __half2half2(__uint2half_rn((sc >> (8 * p)) & 63)), c = __hmul2(s, __float2half2_rn(p & 1 ? -64.f : -1024.f));  // exact
      const uint32_t mask = p & 1 ? 0x00F000F0u : 0x000F000Fu, magic = p & 1 ? 0x54005400u : 0x64006400u;
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {  // word i: k = 4 i .. 4 i + 3 in the order 0, 2, 1, 3
        const uint32_t a = q[8 * (p >> 1) + i];
        o[2 * i] = h2_bits(__hfma2(bits_h2(and_or(a, mask, magic)), s, c)), o[2 * i + 1] = h2_bits(__hfma2(bits_h2(and_or(a >> 8, mask, magic)), s, c));
      }
      put(p, o);
    }
  }
  __device__ __forceinline__ void mins(int u, uint32_t (&o)[8]) const {  // -dmin m of the unit's four sub-blocks: hi, lo, hi, nothing
    const float dmin = __high2float(bits_h2(h.x));
    const uint32_t mn = u & 1 ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const float a = -dmin * (float)((mn >> (16 * j)) & 63), b = -dmin * (float)((mn >> (16 * j + 8)) & 63);
      const __half2 hi = __floats2half2_rn(a, b);
      const float2 f = __half22float2(hi);
      o[j] = o[4 + j] = h2_bits(hi), o[2 + j] = h2_bits(__floats2half2_rn(a - f.x, b - f.y)), o[6 + j] = 0u;
    }
  }
};
template <typename Rows>
struct ExQ6K : Rows {
  using Rows::d;
  using Rows::qh;
  using Rows::ql;
  using Rows::sc;
  static constexpr bool MINS = false;
  __device__ __forceinline__ ExQ6K(const typename Rows::Ctx &c) : Rows(c) {}
  __device__ __forceinline__ float scale() const { return d; }
  template <typename Put>
  __device__ __forceinline__ void whole(int, Put &&put) const {
    const __half2 off = __float2half2_rn(-1056.f), off_s = __float2half2_rn(-1152.f);
    const uint32_t s8[2] = {sc[0] ^ 0x80808080u, sc[1] ^ 0x80808080u};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        // scale 2 q + i / 4 of the half as the f16 pair (sc, sc): 1024 + (sc + 128) by PRMT, less 1152
        const __half2 s = __hadd2(bits_h2(__byte_perm(s8[q >> 1], 0x64646464u, 0x4040 + 0x0101 * (2 * (q & 1) + (i >> 2)))), off_s);
        const uint32_t wq = ql[8 * (q & 1) + i] >> (4 * (q >> 1)), wh = qh[i];
        const uint32_t hi2 = q == 0 ? (wh << 4) : q == 1 ? (wh << 2) : q == 2 ? wh : (wh >> 2);
        const uint32_t v = and_or(wq, 0x0F0F0F0Fu, hi2 & 0x30303030u);
        o[2 * i] = h2_bits(__hmul2(__hadd2(bits_h2(__byte_perm(v, 0x64646464u, 0x4240)), off), s));
        o[2 * i + 1] = h2_bits(__hmul2(__hadd2(bits_h2(__byte_perm(v, 0x64646464u, 0x4341)), off), s));
      }
      put(q, o);
    }
  }
};

// ---- tokens: f16 in the order the weights come out in (of every four k: 0, 2, 1, 3), clamped; and per 128 k, for the minimums, the sums of the
// rounded values over its four sub-blocks: hi, hi, lo, nothing.  A warp to each token's block.
template <bool SUMS>
__global__ void __launch_bounds__(256) x_rows_kernel(const float4 *__restrict__ x, uint2 *__restrict__ y, uint4 *__restrict__ sums, int M, int K) {
  pdl_launch_dependents();
  pdl_wait();
  const int nb = K >> 8, rec = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (rec >= M * nb) return;
  const __half2 lim = __float2half2_rn(65504.f);
  auto clamp2 = [&](float a, float b) { return __hmax2(__hmin2(__floats2half2_rn(a, b), lim), __hneg2(lim)); };
  float4 v[2];
#pragma unroll
  for (int j = 0; j < 2; j++) v[j] = __ldg(x + (size_t)rec * 64 + 32 * j + lane);  // (records follow one another as rows do)
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const __half2 h02 = clamp2(v[j].x, v[j].z), h13 = clamp2(v[j].y, v[j].w);
    y[(size_t)rec * 64 + 32 * j + lane] = make_uint2(h2_bits(h02), h2_bits(h13));
    if constexpr (SUMS) {
      const float2 a = __half22float2(h02), c = __half22float2(h13);
      float p = (a.x + a.y) + (c.x + c.y);
      p += __shfl_xor_sync(0xffffffffu, p, 1), p += __shfl_xor_sync(0xffffffffu, p, 2), p += __shfl_xor_sync(0xffffffffu, p, 4);
      const float p1 = __shfl_sync(0xffffffffu, p, 8), p2 = __shfl_sync(0xffffffffu, p, 16), p3 = __shfl_sync(0xffffffffu, p, 24);
      if (lane == 0) {
        const __half2 h0 = clamp2(p, p1), h1 = clamp2(p2, p3);
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        uint4 *o = sums + ((size_t)rec * 2 + j) * 2;
        o[0] = make_uint4(h2_bits(h0), h2_bits(h1), h2_bits(h0), h2_bits(h1));
        o[1] = make_uint4(h2_bits(clamp2(p - f0.x, p1 - f0.y)), h2_bits(clamp2(p2 - f1.x, p3 - f1.y)), 0u, 0u);
      }
    }
  }
}

template <typename Row>
__global__ void __launch_bounds__(THREADS, 1) decode_tmem_kernel(const __grid_constant__ Maps maps, const typename Row::Ctx ctx, const __grid_constant__ Args a,
                                                                float *__restrict__ out) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_sh;
  __shared__ unsigned tag_sh;
  __shared__ float scales[8][128];  // d of a block's rows, by the block's number in the run
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sB = base, sRaw = base + (uint32_t)a.stages * a.stage_bytes, sBar = sRaw + (uint32_t)EXPANDERS * Row::SLOT;
  // full, empty: a block's weights are there, its MMAs have completed; t_full, t_empty: its tokens; d_full, d_empty: its sums are
  // complete, are read out; p_empty: the minimums' sums are; drained: nothing of the MMA warp's is in flight.
  const uint32_t full = sBar, empty = full + 16, d_full = empty + 16, d_empty = d_full + 32, p_empty = d_empty + 32, w_full = p_empty + 8,
                 t_full = w_full + 8 * EXPANDERS, t_empty = t_full + 8 * NBS, drained = t_empty + 8 * NBS;
  const int warp = same((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int nb = a.K >> 8, G = gridDim.x, cta = blockIdx.x, U = (a.N + 127) / 128 * nb;
  auto bound = [&](int j) { return (int)((long long)U * j / G); };
  const int v0 = same(bound(cta)), n = same(bound(cta + 1)) - v0;  // this CTA's run of (tile, block)

  if (threadIdx.x == 0) {
    prefetch_tmap(&maps.x);
    if constexpr (Row::MINS) prefetch_tmap(&maps.sums);
    for (int i = 0; i < Row::BOXES; i++) prefetch_tmap(&maps.w[i]);
    abort_flag = 0;
    for (int i = 0; i < 2; i++) mbar_init(full + 8 * i, 8), mbar_init(empty + 8 * i, 1);
    for (int i = 0; i < a.stages; i++) mbar_init(t_full + 8 * i, 2), mbar_init(t_empty + 8 * i, 1);
    for (int i = 0; i < a.bufs; i++) mbar_init(d_full + 8 * i, 1), mbar_init(d_empty + 8 * i, DRAINS);
    mbar_init(p_empty, DRAINS), mbar_init(drained, 1);
    for (int i = 0; i < EXPANDERS; i++) mbar_init(w_full + 8 * i, 1);
    fence_barrier_init();
  }
  // (every CTA of this grid is resident once all have come by here: the next kernel's wait for room, and for its operands)
  pdl_launch_dependents();
  if (warp == MMA_WARP) alloc512<1>(smem_u32(&tmem_sh));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = same(tmem_sh), bmask = (uint32_t)a.bufs - 1;
  const int blog = a.bufs == 4 ? 2 : 1;
  const uint32_t cols = 2 * MAX_NT >> blog;
  volatile int *abort = &abort_flag;

  if (warp >= TMA_WARP && warp < MMA_WARP) {
    pdl_wait();  // the tokens are the kernel before's
    const int half = warp - TMA_WARP;
    const uint32_t bytes = (uint32_t)a.nt * (Row::MINS && half ? 320u : 256u), tile = (uint32_t)a.nt * 128u;
    int s = 0, par = 1, kb = same(v0 % nb);
    bool wrapped = false;
    for (int i = 0; i < n; i++) {
      const uint32_t bar = t_full + 8 * s, dst = sB + s * a.stage_bytes;
      if (wrapped && !warp_wait(t_empty + 8 * s, par, abort)) break;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, bytes);
        tma_load_2d(dst + 2 * half * tile, &maps.x, bar, kb * 256 + half * 128, 0);
        tma_load_2d(dst + (2 * half + 1) * tile, &maps.x, bar, kb * 256 + half * 128 + 64, 0);
        if (Row::MINS && half) {
          tma_load_2d(dst + 4 * tile, &maps.sums, bar, kb * 32, 0);
          tma_load_2d(dst + 4 * tile + tile / 4, &maps.sums, bar, kb * 32 + 16, 0);
        }
      }
      __syncwarp();
      if (++kb == nb) kb = 0;
      if (++s == a.stages) s = 0, par ^= 1, wrapped = true;
    }
  } else if (warp == MMA_WARP) {
    const uint32_t idesc = idesc_f16(128, 16, false) + ((uint32_t)((a.nt - 16) >> 3) << 17);
    const uint32_t tile = (uint32_t)a.nt * 128u;
    int t = 0, tpar = 0, kb = same(v0 % nb), seg = 0;
    bool first = true;                  // of the tile's blocks in this run
    bool ready = false, room = false;   // the next block's barriers and buffer, looked at before this one's MMAs are issued
    for (int i = 0; i < n; i++) {
      if (i >= a.bufs && !__all_sync(0xffffffffu, room) && !warp_wait(d_empty + 8 * (i & bmask), ((i >> blog) - 1) & 1, abort)) break;
      if (Row::MINS && first && seg > 0 && !warp_wait(p_empty, (seg - 1) & 1, abort)) break;
      if (!__all_sync(0xffffffffu, ready) && !(warp_wait(t_full + 8 * t, tpar, abort) && warp_wait(full + 8 * (i & 1), (i >> 1) & 1, abort))) break;
      tc_fence_after();
      const uint32_t d = tmem + cols * (i & bmask), st = sB + t * a.stage_bytes, tdone = t_empty + 8 * t;
      if (++t == a.stages) t = 0, tpar ^= 1;
      const bool weights = mbar_test_wait(full + 8 * ((i + 1) & 1), ((i + 1) >> 1) & 1), tokens = mbar_test_wait(t_full + 8 * t, tpar);
      room = i + 1 >= a.bufs && mbar_test_wait(d_empty + 8 * ((i + 1) & bmask), (((i + 1) >> blog) - 1) & 1);
      ready = weights && tokens;
      if (elect_one()) {
        const uint32_t am = tmem + A_COL + 128 * (i & 1), mins = tmem + M_COL + 16 * (i & 1);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint64_t b = smem_desc_sw128(st + q * tile);
#pragma unroll
          for (int j = 0; j < 4; j++) mma_ts<1>(d, am + 32 * q + 8 * j, b + 2 * j, idesc, q || j ? 1u : 0u);
        }
        if constexpr (Row::MINS) {
          mma_ts<1>(tmem + P_COL, mins, smem_desc_sw32(st + 4 * tile), idesc, first ? 0u : 1u);
          mma_ts<1>(tmem + P_COL, mins + 8, smem_desc_sw32(st + 4 * tile + tile / 4), idesc, 1u);
        }
        mma_commit(empty + 8 * (i & 1));
        mma_commit(d_full + 8 * (i & bmask));
        mma_commit(tdone);
      }
      __syncwarp();
      first = false;
      if (++kb == nb) kb = 0, first = true, seg++;
    }
    // No MMA, and none of the arrivals that nobody above waits for, may be in flight when the CTA gives its memory back, whichever way the
    // loop ended.
    if (elect_one()) mma_commit(drained);
    __syncwarp();
    for (int i = 0; i < (1 << 16) && !__all_sync(0xffffffffu, mbar_test_wait(drained, 0)); i++) {
    }
  } else if (warp < EXPANDERS) {
    // ================================================================ expanders
    const int set = warp >> 2, quad = warp & 3, half = set & 1;
    const uint32_t slot = sRaw + (uint32_t)warp * Row::SLOT, copied = w_full + 8 * warp, lanes = (uint32_t)(quad * 32) << 16;
    Row rowx(ctx);
    int i = set >> 1, kb = same((v0 + i) % nb), tile = same((v0 + i) / nb);  // this warp's next block: number in the run, in its rows, and the tile
    [[maybe_unused]] int y = 0;
    [[maybe_unused]] const uint8_t *src = nullptr;
    [[maybe_unused]] int rows = 0;
    auto aim = [&]() {
      const int nw = min(tile * 128 + quad * 32, a.N - 1);
      y = nw;
      if constexpr (Row::BOXES == 0) src = Row::base(ctx) + (size_t)nw * Row::stride(a.K), rows = a.N - 1 - nw;
      rowx.row(ctx, min(nw + lane, a.N - 1), a.K);
    };
    auto issue = [&]() {
      if constexpr (Row::BOXES > 0) {
        if (elect_one()) {
          mbar_arrive_expect_tx(copied, Row::BYTES);
          Row::copy(slot, maps.w, copied, 2 * kb + half, y);
        }
      } else {  // (as in gemm_tmem.cu: lanes 10 r + i copy granule i of rows r, r + 3, ..)
        const int r0 = lane / 10, g = lane - 10 * r0;
        const size_t step = Row::stride(a.K);
        const uint8_t *at = src + kb * 210;
        const uint32_t dst = slot + r0 * Row::PITCH + 16 * g;
        const int place = 16 * Row::number(half, g);
        if (lane < 30) {
          if (rows >= 32) {  // (a whole row follows the last one: no copy passes the end of the matrix)
            at += (size_t)r0 * step;
#pragma unroll
            for (int k = 0; k < 11; k++, at += 3 * step)
              if (k < 10 || r0 < 2) cp_async16(dst + 3 * k * Row::PITCH, reinterpret_cast<const uint8_t *>((uintptr_t)at & ~(uintptr_t)15) + place);
          } else {
            const uint8_t *const end = Row::base(ctx) + (size_t)a.N * step;
            for (int k = 0; k < 11; k++)
              if (k < 10 || r0 < 2) {
                const uint8_t *p = reinterpret_cast<const uint8_t *>((uintptr_t)(at + (size_t)min(r0 + 3 * k, rows) * step) & ~(uintptr_t)15) + place;
                if (p + 16 <= end) cp_async16(dst + 3 * k * Row::PITCH, p);
                else if (p < end) cp_async16_part(dst + 3 * k * Row::PITCH, p, (uint32_t)(end - p));
              }
          }
        }
        cp_async_commit();
      }
    };
    const uint32_t acol = tmem + lanes + A_COL + 64 * set;
    if (i < n) aim(), issue();
    bool ok = true;
    for (int round = 0; i < n && ok; round++) {
      if constexpr (Row::BOXES > 0) {
        if (!warp_wait(copied, round & 1, abort)) break;
      } else {
        cp_async_wait<0>();
        __syncwarp();
      }
      const int u = 2 * kb + half, now = i;
      rowx.load(slot, u);
      if constexpr (Row::BOXES > 0) fence_proxy_async();  // the reads above come before the copy that overwrites the slot
      __syncwarp();
      i += 2, kb += 2;
      if (i < n) {
        if (kb >= nb) {
          while (kb >= nb) kb -= nb, tile++;
          aim();
        }
        issue();
      }
      if (round > 0 && !warp_wait(empty + 8 * (set >> 1), (round - 1) & 1, abort)) break;  // the MMAs of the block two before
      tc_fence_after();
      // (the drain is done with the block eight before: the MMAs of the one two before, complete now, have waited for a later one)
      if (half == 0) scales[now & 7][quad * 32 + lane] = rowx.scale();
      if constexpr (Row::MINS) {
        uint32_t m[8];
        rowx.mins(u, m);
        __syncwarp();
        tmem_st8(tmem + lanes + M_COL + 8 * set, m);
      }
      rowx.whole(u, [&](int p, const uint32_t (&o)[16]) {
        __syncwarp();
        tmem_st16(acol + 16 * p, o);
      });
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * (set >> 1));
    }
    if constexpr (Row::BOXES == 0) cp_async_wait<0>();
  } else {
    // ================================================================ drain
    const int dw = warp - DRAIN_WARP, quad = warp & 3, grp = dw >> 2, row = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    pdl_wait();  // `out` and the partial tiles may still be in use by the kernel before
    if (dw == 0 && lane == 0) {
      unsigned epoch;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(epoch) : "l"(&g_sync.epoch) : "memory");
      tag_sh = epoch + 1;
      if (atomicInc(&g_sync.readers, gridDim.x - 1) == gridDim.x - 1) atomicExch(&g_sync.epoch, epoch + 1);  // every CTA has read it
    }
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
    const unsigned tag = tag_sh;
    bool ok = true;
    for (int i = 0; i < n && ok;) {
      const int tile = (v0 + i) / nb, k0 = (v0 + i) - tile * nb, k1 = min(nb, k0 + n - i);
      float acc[2][16];
#pragma unroll
      for (int c = 0; c < 2; c++)
#pragma unroll
        for (int k = 0; k < 16; k++) acc[c][k] = 0.f;
      for (int kb = k0; kb < k1; kb++, i++) {
        if (!warp_wait(d_full + 8 * (i & bmask), (i >> blog) & 1, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const float s = scales[i & 7][row];
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const int c0 = 16 * (2 * c + grp);
          if (c0 < a.nt) {
            uint32_t w[16];
            tmem_ld16(tmem + lanes + cols * (i & bmask) + c0, w);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; k++) acc[c][k] = fmaf(__uint_as_float(w[k]), s, acc[c][k]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty + 8 * (i & bmask));
      }
      if (!ok) break;
      if constexpr (Row::MINS) {  // (complete: committed before the last block's sums)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const int c0 = 16 * (2 * c + grp);
          if (c0 < a.nt) {
            uint32_t w[16];
            tmem_ld16(tmem + lanes + P_COL + c0, w);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; k++) acc[c][k] += __uint_as_float(w[k]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_empty);
      }
      if (k0 > 0) {  // the tile is another run's: leave this part of it
        float *mine = a.parts + (size_t)cta * PART_FLOATS + row;
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const int c0 = 16 * (2 * c + grp);
          if (c0 < a.nt) {
#pragma unroll
            for (int k = 0; k < 16; k++) __stcg(mine + (c0 + k) * 128, acc[c][k]);
          }
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(g_sync.flags + cta * 64 + dw), "r"(tag) : "memory");
        continue;
      }
      if (16 * grp >= a.nt) continue;  // none of the tile's tokens
      if (k1 < nb) {  // other runs hold the rest of it
        int jlast = cta;
        while (jlast + 1 < G && bound(jlast + 1) < (tile + 1) * nb) jlast++;
        for (int j0 = cta + 1; j0 <= jlast && ok; j0 += 32) {  // their flags, a lane to each (no run is empty)
          const int j = min(j0 + lane, jlast), last = min(j0 + 31, jlast);
          ok = wait_flag(g_sync.flags + j * 64 + dw, tag, true, abort);
          if (a.nt <= 32) {  // one chunk to a warp: two parts on their way together
            const float *theirs = a.parts + (size_t)j0 * PART_FLOATS + row + 16 * grp * 128;
            for (int p = j0; p <= last && ok; p += 2, theirs += 2 * PART_FLOATS) {
              float x[2][16];
#pragma unroll
              for (int c = 0; c < 2; c++)
#pragma unroll
                for (int k = 0; k < 16; k++) x[c][k] = p + c <= last ? __ldcg(theirs + (size_t)c * PART_FLOATS + k * 128) : 0.f;
#pragma unroll
              for (int k = 0; k < 16; k++) acc[0][k] = (acc[0][k] + x[0][k]) + x[1][k];
            }
            continue;
          }
          for (int p = j0; p <= last && ok; p++) {
            const float *theirs = a.parts + (size_t)p * PART_FLOATS + row;
            float x[2][16];
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
              for (int k = 0; k < 16; k++) x[c][k] = 16 * (2 * c + grp) < a.nt ? __ldcg(theirs + (16 * (2 * c + grp) + k) * 128) : 0.f;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
              for (int k = 0; k < 16; k++) acc[c][k] += x[c][k];
          }
        }
        if (!ok) break;
      }
      const int col = tile * 128 + row;
      if (col < a.N) {
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int k = 0; k < 16; k++) {
            const int m = 16 * (2 * c + grp) + k;
            if (m < a.M) out[(size_t)m * a.N + col] = acc[c][k];
          }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {  // copies and MMAs still in flight get some time to land before the CTA retires
    __nanosleep(50000);
    if (threadIdx.x == 0) g_status = 1;
  }
  if (warp == MMA_WARP) dealloc512<1>(tmem);
}

size_t align1k(size_t n) { return (n + 1023) & ~(size_t)1023; }

template <typename Row>
int run(const typename Row::Ctx &ctx, const float *x, float *out, int M, int N, int K, void *ws, size_t ws_bytes, cudaStream_t st) {
  const size_t x_bytes = align1k((size_t)M * K * 2), sum_bytes = Row::MINS ? align1k((size_t)M * (K / 128) * 32) : 0;
  const int nb = K >> 8, U = (N + 127) / 128 * nb;
  int G = sm_count() < MAX_GRID ? sm_count() : MAX_GRID;
  if (U < 2 * G) G = U / 2 > 0 ? U / 2 : 1;  // (a run of one block is mostly start and end)
  if (ws_bytes < x_bytes + sum_bytes + (size_t)G * PART_FLOATS * 4) return 0;
  const EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(LB200_E_DEVICE, "light_b200: cuTensorMapEncodeTiled is not available from the driver");
  Args a = {};
  a.M = M, a.N = N, a.K = K, a.nt = (M + 15) / 16 * 16, a.bufs = a.nt <= 32 ? 4 : 2;
  a.stage_bytes = (a.nt * (Row::MINS ? 576 : 512) + 1023) & ~1023;
  const int fixed = EXPANDERS * Row::SLOT + BAR_BYTES + 1024 + 5120;  // (the last: static shared memory)
  a.stages = (SMEM_MAX - fixed) / a.stage_bytes;
  if (a.stages > NBS) a.stages = NBS;
  if (a.stages < 2) return 0;
  const int smem = fixed - 5120 + a.stages * a.stage_bytes;
  char *const w8 = (char *)ws;
  a.parts = (float *)(w8 + x_bytes + sum_bytes);
  Maps tm = {};
  const cuuint32_t estr[2] = {1, 1};
  auto map = [&](CUtensorMap *m, CUtensorMapDataType dt, const void *p, size_t width, size_t height, size_t pitch, int bw, int bh, CUtensorMapSwizzle sw) {
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)height}, strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
    return enc(m, dt, 2, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  bool ok = map(&tm.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w8, K, M, (size_t)K * 2, 64, a.nt, CU_TENSOR_MAP_SWIZZLE_128B);
  if (Row::MINS) ok = ok && map(&tm.sums, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w8 + x_bytes, K / 8, M, (size_t)K / 4, 16, a.nt, CU_TENSOR_MAP_SWIZZLE_32B);
  if constexpr (Row::BOXES > 0)
    for (int i = 0; i < Row::BOXES; i++)
      ok = ok && map(&tm.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, Row::base(ctx), Row::stride(K), N, Row::stride(K), Row::BOX[i].bytes, 32,
                     swizzle_of(Row::BOX[i].swizzle));
  if (!ok) return fail(LB200_E_SHAPE, "light_b200: cuTensorMapEncodeTiled failed");
  launch_early(x_rows_kernel<Row::MINS>, dim3((unsigned)((M * nb + 7) / 8)), dim3(256), st, (const float4 *)x, (uint2 *)w8, (uint4 *)(w8 + x_bytes), M, K);
  if (int rc = launched("decode: activations to f16")) return rc;
  auto kern = decode_tmem_kernel<Row>;
  static DeviceOnce attr;
  cudaError_t e = attr.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX - 5120); });
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode (tmem): %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)G), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at, cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kern, tm, ctx, a, out);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode (tmem): %s", cudaGetErrorString(e));
  if (int rc = launched("decode (whole numbers through tensor memory)")) return rc;
  return 1;
}

}  // namespace

// Where this beats the kernels that take the call otherwise (us per call of a chain with a cold L2, those / here).  What it costs beside its
// blocks is the exchange of cut tiles and some 10 us of start and end, so the rules go by the list of (tile, block) and the runs it is cut into.
//   Q4_K, 9 to 16 rows: lists of four blocks or more to an SM, which the token tiles have: 4096 x 5120 14.3 / 13.6, 4096 x 14336 23.0 / 20.5, 28672 x 4096
//     32.8 / 28.1 (even from 20 to 32 Mi weights; K = 1024 loses, 28672 x 1024 9.8 / 11.9).  Shorter ones are the cluster kernel's (K split over a
//     cluster, no pass over x): 4096 x 4096 8.9 / 12.8, 4096 x 4352 10.8 / 12.9, 3584 x 4864 11.2 / 13.5, 3072 x 5632 10.9 / 13.4, 2048 x 8192 13.0 / 14.3,
//     unless the matrix is so tall that a tile is cut into four parts at most: 5120 x 3328 14.8 / 12.7, 6144 x 2816 15.7 / 12.2, 8192 x 2048 12.2 / 12.0.
//   Q4_K, 17 to 32: from 16 Mi weights on: 28672 x 4096 42.6 / 30.9, 6144 x 4096 18.6 / 14.7, 8192 x 2048 16.6 / 12.6, 1024 x 16384 26.6 / 19.1,
//     4096 x 4096 12.8 / 13.1; below, a tile is cut into too many parts (4096 x 2048 9.3 / 9.8, 1024 x 4096 9.3 / 10.7).
//   33 to 64, where a part is a chunk more to each warp: not where a tile is cut into more than eight parts of few blocks: Q4_K 2048 x 8192 18.5 / 21.4, 1024 x
//     8192 17.3 / 18.2, 1024 x 20480 24.4 / 31.5, 2048 x 10240 21.3 / 23.5, but 2048 x 2048 11.9 / 8.8, 1024 x 4096 14.9 / 11.7, 4096 x 2048 12.0 / 9.5,
//     2048 x 4096 13.6 / 12.3, 2560 x 6656 20.6 / 18.8, 1536 x 16384 26.9 / 24.5, 28672 x 4096 65.2 / 33.2, 4096 x 14336 40.8 / 27.8.
//     Q6_K 2048 x 8192 19.0 / 21.4, 2048 x 12288 24.2 / 24.6, but 1024 x 4096 14.8 / 11.0, 2048 x 2048 11.6 / 8.1, 2048 x 4096 13.6 / 12.0, 2560 x 6656 21.9 / 20.4, 2048 x 16384 30.7 /
//     27.4, 4096 x 14336 43.2 / 26.5, 128256 x 4096 307 / 170 (4096 x 4096 17.1 / 15.6).
// And where the token tiles' runs are all alike (decode_nt_equal_run) they stay ahead of this kernel, whose hand-overs then weigh more:
//   Q6_K, 9 to 16 (12 rows): whole tiles 12800 x 512 5.9 / 6.1; runs of two, from 250 blocks on 1792 x 4608 10.3 / 11.6 (1536 x 4608, 216 blocks, 11.5 / 9.2); runs of three or four on up to 138
//     CTAs 4096 x 3072 10.9 / 13.5, 2304 x 7168 13.4 / 15.7, 4096 x 4096 12.0 / 12.8 (140 CTAs: 2560 x 7168 17.0 / 16.0); beyond 592 blocks rows of 2, 4 or 12: 32768 x 1024 13.9 / 16.1, 12288 x
//     3072 18.5 / 20.7 (3072 x 8192 18.0 / 15.6).
//   33 to 64: whole tiles of three or four blocks: Q4_K 64 rows 15360 x 768 9.7 / 11.4, 16000 x 1024 12.3 / 13.3, Q6_K 16000 x 1024 13.6 / 15.0 (two: Q4_K 16384 x 512 1.17 times as fast here).
//   Rows of one block on fewer tiles than SMs: Q4_K 8192 x 256, 33 rows 5.0 / 5.6.
//   Q6_K, 17 to 32: 1024 x 3584 10.7 / 7.9, 2048 x 2048 10.7 / 6.9, 2048 x 5632 19.0 / 14.3, 4096 x 14336 31.1 / 21.9, 128256 x 4096 186 / 156.  9 to 16, but for
//     tiles in more than nine parts (2048 x 5632 16.2 / 14.1, 2048 x 7168 14.5 / 15.6): 4096 x 1024 8.0 / 6.2, 2048 x 2048 8.5 / 6.8, 1024 x 4096 9.3 / 8.0, 2048 x 4096
//     10.8 / 8.9, 3072 x 9216 19.0 / 18.3, 4096 x 10240 22.2 / 17.8.
int gguf_decode_tmem(int type, const float *x, const void *w, float *out, int M, int N, int K, void *ws, size_t ws_bytes, cudaStream_t st) {
  static const int min_m = knob("LIGHT_B200_DECODE_TMEM_MIN_M", 9);
  const bool q4 = type == LB200_Q4_K;
  const long long size = (long long)N * K;
  if ((!q4 && type != LB200_Q6_K) || M < min_m || M > MAX_NT || K % 256 || !ws || N < 128 || size >> 8 > 1ll << 30 || ((uintptr_t)x & 15)) return 0;
  const long long tiles = (N + 127) / 128, U = tiles * (K >> 8), sms = sm_count();
  const long long runs = U < 2 * sms ? U / 2 : sms;  // (as run() has them)
  if (size < (q4 && M <= 32 ? 16ll : 2ll) << 20) return 0;  // (smaller matrices were not compared, nor below 16 Mi the cluster kernel's, which needs no workspace)
  if (q4 && M <= 16 && U < 4 * sms && 4 * tiles < sms) return 0;
  if (!q4 && M <= 16 && runs > 9 * tiles) return 0;
  if (M > 32 && U < (q4 ? 5 : 6) * sms && runs > 8 * tiles) return 0;
  const int nb = K >> 8, equal = decode_nt_equal_run(U, nb);
  if (!q4 && M <= 16 && equal >= 2 && (nb <= equal || (equal == 2 ? U >= 250 : U <= 138 * equal) || (U > 4 * sms && nb <= 16 && nb % 8))) return 0;
  if (M > 32 && equal >= 3 && nb <= equal && U <= 4 * sms) return 0;
  if (nb == 1 && tiles <= sms) return 0;
  if (q4 && !((uintptr_t)w & 15)) return run<ExQ4K>({(const uint8_t *)w}, x, out, M, N, K, ws, ws_bytes, st);
  if (!q4 && TmQ6KT::fits(w, K)) return run<ExQ6K<TmQ6KT>>({(const uint8_t *)w}, x, out, M, N, K, ws, ws_bytes, st);
  if (!q4 && !((uintptr_t)w & 3) && (K >> 8) % 2 == 0) return run<ExQ6K<TmQ6K>>({(const uint8_t *)w}, x, out, M, N, K, ws, ws_bytes, st);
  return 0;
}

int decode_tmem_status() {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, g_status, sizeof(int));
  return e == cudaSuccess ? v : -(int)e;
}

}  // namespace lb
