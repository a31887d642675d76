// Dequantize-and-multiply for many activation rows, plain and grouped (MoE), with the expanded weights handed to
// tcgen05.mma through TENSOR MEMORY: D (128 weight rows x NT tokens) += A (weights, TMEM) x B (tokens, shared memory).
//
// What bounds it.  A kernel that stages both operands in shared memory moves 40 KB through the SM's 128 B/clk port per
// 256 x 256 x 16 of work (the operand reads of two MMAs, the TMA writes of the tokens and the expander's writes of the
// weights): 320 clocks for 256 clocks of tensor time, 441 measured.  Here weights never touch shared memory after
// they arrive packed (a thread owns a weight row = a TMEM lane and stores 64 expanded values with one tcgen05.st), and in
// the paired form (CG = 2) two SMs share each token tile, which leaves 8 KB per 256 x 256 x 16 and SM: half the port.
// Tokens are the N side, so a tile holds any multiple of 16 (32 when paired) of them: short prompts and the ragged
// token counts of experts cost what they are, not the next multiple of 128.  Weight rows are the M side and always full.
//
//   warps 0-7    expanders.  Warps w and w + 4 own rows 32 (w & 3) .. + 31 (the TMEM lanes a warp can reach) and take
//                turns at the K chunks: packed rows arrive by cp.async in the warp's own slots, are read into registers,
//                and leave as 32 TMEM columns per 64 k (eight stages).
//   warp  8      one lane: TMA of the token tiles.
//   warp  9      one lane: MMAs and commits; in the second CTA of a pair: forwards "my half is ready" to the first.
//   warps 10-13  epilogue: TMEM -> registers -> output rows (a warp's lanes hold 32 consecutive columns of a token's row:
//                full lines without a transpose), while the next tile's MMAs run (token tiles up to 128 use two accumulators).
//
// Work is the list of (tile, K chunk) pairs, cut into equal runs, one per CTA (pair): stream-K.  A segment that does not
// start its tile writes a partial tile and raises its flag, which it does first; the segment that starts the tile owns it
// and adds the partials in run order.  In a grouped launch the units are weighted by their token count, so that runs are
// equal in time.  Every wait is bounded; on giving up the status word is set, TMEM is freed and the CTA retires.
#include <cuda.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "mma_sync.cuh"
#include "row_expand.cuh"
#include "umma.cuh"

namespace lb {
namespace {

using namespace umma;

constexpr int TMA_WARP = 8, MMA_WARP = 9, THREADS = 14 * 32;
constexpr int NAS = 4;                        // TMEM stages of expanded weights, 64 columns (128 k) each
constexpr int A_COL = 256;                    // columns 0-255: accumulators, 256-511: weight stages
constexpr int MAX_E = 1024;                   // experts whose prefix sums fit the shared tables
constexpr int MAX_GRID = 160;
constexpr int PART_FLOATS = 256 * 128;        // one partial tile: [token][row]
constexpr int SMEM_MAX = 227 * 1024 - 1024;   // dynamic; the static part (prefix tables, flags) is accounted below

__device__ int g_status;                      // non-zero: a bounded wait gave up (sticky)
__device__ unsigned int g_flags[MAX_GRID * 4];  // per epilogue warp: raised by the writer of a partial tile, lowered by its one reader

// Per row format: k per chunk (one copy of a warp's 32 rows), its 16-byte granules per row, the slot pitch (an odd
// number of granules spreads the rows over the banks), and the load units (Row::load_*) that make up a chunk.
template <typename Row> struct Fmt;
template <> struct Fmt<Q4KRow> { static constexpr int KU = 256, GR = 9, PITCH = 144, LOADS = 1; };
template <> struct Fmt<Q6KRow> { static constexpr int KU = 256, GR = 14, PITCH = 240, LOADS = 2; };
template <> struct Fmt<Q80Row> { static constexpr int KU = 256, GR = 17, PITCH = 272, LOADS = 2; };
template <> struct Fmt<Int4Row> { static constexpr int KU = 256, GR = 8, PITCH = 144, LOADS = 1; };
template <> struct Fmt<Fp8Row> { static constexpr int KU = 128, GR = 8, PITCH = 144, LOADS = 1; };
template <> struct Fmt<DenseRow> { static constexpr int KU = 128, GR = 16, PITCH = 272, LOADS = 2; };

struct Args {
  const int32_t *offsets;   // grouped: expert e owns rows offsets[e] .. offsets[e + 1] of the (gathered) tokens; null: one matrix
  const int64_t *pairs;     // grouped: token row i goes to output row pairs[i] ...
  const float *topkw;       // ... scaled by its routing weight (or null)
  long long size_m;
  int E, M, N, K;
  int nt_max;               // most tokens of a tile
  int box;                  // token rows of one TMA box
  int stage_bytes, nbs;     // of the token ring (a stage: 128 k), per CTA
  int wmin;                 // grouped: a unit's weight is max(tokens of its tile, wmin)
  float *parts;
};

struct Tile {
  int expert, n0, m0, m_end, nt;
};

// ------------------------------------------------------------------------------------ PTX forms this file adds
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) { return map_to_rank(addr, rank); }
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
// A whole warp waits, together: every lane looks and all branches are on votes, so the warp never diverges here (what
// follows are .aligned instructions and values the compiler keeps in the warp's uniform registers).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort) {
  if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 1;; i++) {
    if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
    if ((i & 63u) == 0) {
      if (__any_sync(0xffffffffu, *abort != 0)) return false;
      if (__any_sync(0xffffffffu, global_ns() - t0 > 1000000000ull)) break;
      __nanosleep(32);
    }
  }
  *abort = 1;
  return false;
}
__device__ __forceinline__ void st_if(bool p, float *o, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}\n" ::"l"(o), "f"(v), "r"((int)p) : "memory");
}
__device__ __forceinline__ void st_if(bool p, __nv_bfloat16 *o, float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.b16 [%0], %1;\n\t}\n" ::"l"(o), "h"(*reinterpret_cast<const uint16_t *>(&b)), "r"((int)p)
               : "memory");
}
template <int CG>
__device__ __forceinline__ void alloc512(uint32_t smem_dst) {
  if constexpr (CG == 1) {
    tmem_alloc(smem_dst, 512);
    tmem_relinquish();
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_dst) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void dealloc512(uint32_t taddr) {
  if constexpr (CG == 1) tmem_dealloc(taddr, 512);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(taddr) : "memory");
}
// D[tmem] (+)= A[tmem] x B[smem]; with CG = 2 each CTA of the pair holds half of the rows of A and D and half of the
// columns (tokens) of B at the same addresses, and the first CTA issues for both
template <int CG>
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar) {  // CG = 2: on this barrier of both CTAs
  if constexpr (CG == 1) mma_commit(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ bool wait_flag(const unsigned *flag, volatile int *abort) {  // whole warp
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 1;; i++) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(flag) : "memory");
    if (__all_sync(0xffffffffu, v != 0)) return true;
    if ((i & 15u) == 0) {
      if (__any_sync(0xffffffffu, *abort != 0)) return false;
      if (__any_sync(0xffffffffu, global_ns() - t0 > 1000000000ull)) break;
      __nanosleep(64);
    }
  }
  *abort = 1;
  return false;
}

// ------------------------------------------------------------------------------------ work list
// Experts with their token tiles: preT[e] tiles and preW[e] weighted units before expert e.  Within an expert the token
// tiles of one row tile follow one another, so that its packed weights are read from HBM once and from L2 after that.
template <int CG>
struct Work {
  const Args &a;
  const int *preT;
  const long long *preW;
  int nb, nrt;
  __device__ __forceinline__ int count(int e) const { return a.offsets ? a.offsets[e + 1] - a.offsets[e] : a.M; }
  __device__ __forceinline__ int first(int e) const { return a.offsets ? a.offsets[e] : 0; }
  __device__ __forceinline__ void geo(int cnt, int &ntt, int &nt) const {
    ntt = (cnt + a.nt_max - 1) / a.nt_max;
    nt = ntt ? ((cnt + ntt - 1) / ntt + 16 * CG - 1) / (16 * CG) * (16 * CG) : 0;
  }
  __device__ __forceinline__ int weight(int nt) const { return a.offsets ? max(nt, a.wmin) : 1; }
  __device__ __forceinline__ Tile tile(int t) const {
    int lo = 0, hi = a.E - 1;  // the expert with preT[e] <= t < preT[e + 1]
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (preT[mid + 1] <= t) lo = mid + 1;
      else hi = mid;
    }
    Tile T;
    int ntt;
    const int cnt = count(lo);
    geo(cnt, ntt, T.nt);
    const int r = t - preT[lo], rt = r / ntt, tt = r - rt * ntt;
    T.expert = lo, T.n0 = rt * 128 * CG, T.m0 = first(lo) + tt * T.nt, T.m_end = min(first(lo) + cnt, T.m0 + T.nt);
    return T;
  }
  // first unit (tile-major) of run j of G
  __device__ __forceinline__ long long bound(int j, int G) const {
    const long long W = preW[a.E], w = W * j / G;
    if (j >= G) return (long long)preT[a.E] * nb;
    int lo = 0, hi = a.E - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (preW[mid + 1] <= w) lo = mid + 1;
      else hi = mid;
    }
    int ntt, nt;
    geo(count(lo), ntt, nt);
    return (long long)preT[lo] * nb + (w - preW[lo]) / weight(nt);
  }
};

template <typename Row>
__device__ __forceinline__ const uint8_t *row_ptr(const Row &r) { return reinterpret_cast<const uint8_t *>(r.row); }
template <typename Row> struct HasAux : std::false_type {};
template <> struct HasAux<Int4Row> : std::true_type {};
template <> struct HasAux<Fp8Row> : std::true_type {};

// ------------------------------------------------------------------------------------ kernel
template <typename Row, bool BF16, typename OutT, int CG, int NSLOT>
__global__ void __launch_bounds__(THREADS, 1) gemm_tmem_kernel(const __grid_constant__ CUtensorMap tmap, const typename Row::Ctx ctx,
                                                              const __grid_constant__ Args a, OutT *__restrict__ out) {
  using F = Fmt<Row>;
  constexpr int SPC = F::KU / 64, SPL = SPC / F::LOADS;  // 64-k steps per chunk and per load unit
  extern __shared__ unsigned char smem_raw[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_sh;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char *gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t ring_bytes = (uint32_t)a.nbs * a.stage_bytes;
  const uint32_t sB = base, sRaw = base + ring_bytes, sBar = sRaw + 8u * NSLOT * 32 * F::PITCH;
  const uint32_t a_full = sBar, a_empty = a_full + 8 * NAS, peer_full = a_empty + 8 * NAS, d_full = peer_full + 8 * NAS, d_empty = d_full + 16,
                 b_full = d_empty + 16, b_empty = b_full + 8 * 16, drained = b_empty + 8 * 16;
  long long *preW = reinterpret_cast<long long *>(gen + (sBar - base) + 512);
  int *preT = reinterpret_cast<int *>(preW + a.E + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CG == 2 ? (int)cluster_ctarank() : 0;
  const Work<CG> wk{a, preT, preW, a.K / F::KU, (a.N + 128 * CG - 1) / (128 * CG)};
  const int nb = wk.nb;
  const int G = gridDim.x / CG, cta = blockIdx.x / CG;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < NAS; i++) mbar_init(a_full + 8 * i, 4), mbar_init(a_empty + 8 * i, 1), mbar_init(peer_full + 8 * i, 1);
    for (int i = 0; i < 2; i++) mbar_init(d_full + 8 * i, 1), mbar_init(d_empty + 8 * i, 4 * CG);
    mbar_init(drained, 1);
    for (int i = 0; i < a.nbs; i++) mbar_init(b_full + 8 * i, 1), mbar_init(b_empty + 8 * i, 1);
    fence_barrier_init();
  }
  for (int e = threadIdx.x; e < a.E; e += THREADS) {
    int ntt, nt;
    wk.geo(wk.count(e), ntt, nt);
    preT[e + 1] = ntt * wk.nrt;
    preW[e + 1] = (long long)ntt * wk.nrt * nb * wk.weight(nt);
  }
  if (warp == MMA_WARP) alloc512<CG>(smem_u32(&tmem_sh));
  __syncthreads();
  if (warp == 0) {  // inclusive prefix sums, 32 experts at a time
    int ct = 0;
    long long cw = 0;
    for (int e0 = 0; e0 < a.E; e0 += 32) {
      int t = e0 + lane < a.E ? preT[e0 + lane + 1] : 0;
      long long w = e0 + lane < a.E ? preW[e0 + lane + 1] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int tt = __shfl_up_sync(0xffffffffu, t, d);
        const long long ww = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) t += tt, w += ww;
      }
      if (e0 + lane < a.E) preT[e0 + lane + 1] = ct + t, preW[e0 + lane + 1] = cw + w;
      ct += __shfl_sync(0xffffffffu, t, 31), cw += __shfl_sync(0xffffffffu, w, 31);
    }
    if (lane == 0) preT[0] = 0, preW[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem = tmem_sh;
  volatile int *abort = &abort_flag;
  const long long pos0 = wk.bound(cta, G), pos1 = wk.bound(cta + 1, G);
  const int n = (int)(pos1 - pos0);  // units of this run

  if (warp == TMA_WARP) {
    if (lane == 0) {
      prefetch_tmap(&tmap);
      int bt = 0, ph = 1, issued = 0;
      for (long long pos = pos0; pos < pos1 && !*abort;) {
        const int t = (int)(pos / nb), u0 = (int)(pos - (long long)t * nb), u1 = (int)min((long long)nb, u0 + (pos1 - pos));
        const Tile T = wk.tile(t);
        const int rows = T.nt / CG, boxes = (rows + a.box - 1) / a.box, y0 = T.m0 + rank * rows;
        const uint32_t bytes = (uint32_t)(boxes * a.box) * 128u;
        for (int k = u0 * SPC; k < u1 * SPC; k += 2) {
          if (issued >= a.nbs && !mbar_wait(b_empty + 8 * bt, ph, abort)) break;
          mbar_arrive_expect_tx(b_full + 8 * bt, 2 * bytes);
          for (int i = 0; i < 2 * boxes; i++) {
            const int h = i & 1, bx = i >> 1;
            tma_load_2d(sB + bt * a.stage_bytes + h * (a.stage_bytes / 2) + bx * a.box * 128, &tmap, b_full + 8 * bt, (k + h) * 64, y0 + bx * a.box);
          }
          issued++;
          if (++bt == a.nbs) bt = 0, ph ^= 1;
        }
        pos += u1 - u0;
      }
      if (*abort)  // the loads still in flight get a bounded time to land before the CTA retires
        for (int k = issued > a.nbs ? issued - a.nbs : 0; k < issued; k++)
          for (int i = 0; i < (1 << 14) && !mbar_test_wait(b_full + 8 * (k % a.nbs), (k / a.nbs) & 1); i++) {
          }
    }
  } else if (warp == MMA_WARP) {
    // The whole warp runs the loop and one elected lane issues.  A pass costs about 700 clocks of instruction latency
    // (three barrier looks, fence, first MMA, two commits) whatever it issues, so a stage is 128 k: eight MMAs of 128 clocks;
    // with 64 k per pass the tensor pipe stood at half its rate.  The next stage's barriers are looked at before this
    // stage's turn ends.
    const bool leader = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    int s = 0, par = 0, bt = 0, bph = 0, seg = 0;
    bool ok = true, wide_before = false;
    auto look = [&]() {
      const bool x = mbar_test_wait(a_full + 8 * s, par), y = mbar_test_wait(b_full + 8 * bt, bph);
      return x && y && (CG == 1 || rank != 0 || mbar_test_wait(peer_full + 8 * s, par));
    };
    for (long long pos = pos0; pos < pos1 && ok; seg++) {
      const int t = (int)(pos / nb), u0 = (int)(pos - (long long)t * nb), u1 = (int)min((long long)nb, u0 + (pos1 - pos));
      const int nt = __shfl_sync(0xffffffffu, wk.tile(t).nt, 0);
      const bool wide = nt > 128;
      if (rank == 0) {  // the accumulators this segment overwrites must have been read out
        if (seg >= 2 && !warp_wait(d_empty + 8 * (seg & 1), ((seg - 2) >> 1) & 1, abort)) break;
        if (seg >= 1 && (wide || wide_before) && !warp_wait(d_empty + 8 * ((seg - 1) & 1), ((seg - 1) >> 1) & 1, abort)) break;
      }
      wide_before = wide;
      const uint32_t d = tm + (wide ? 0 : 128 * (seg & 1));
      const uint32_t idesc = idesc_f16(128 * CG, 16, BF16) + ((uint32_t)((nt - 16) >> 3) << 17);
      const int stages = (u1 - u0) * (SPC / 2);
      uint32_t acc = 0;
      bool ready = look();
      for (int k = 0; k < stages; k++) {
        if (!__all_sync(0xffffffffu, ready)) {
          ok = warp_wait(a_full + 8 * s, par, abort) && warp_wait(b_full + 8 * bt, bph, abort);
          if (CG == 2 && rank == 0) ok = ok && warp_wait(peer_full + 8 * s, par, abort);
          if (!ok) break;
        }
        tc_fence_after();
        if (CG == 1 || rank == 0) {
          const uint64_t b0 = smem_desc_sw128(sB + bt * a.stage_bytes), b1 = b0 + (uint64_t)(a.stage_bytes >> 5);
          const uint32_t am = tm + A_COL + 64 * (s & (NAS - 1));
          if (leader) {
            mma_ts<CG>(d, am, b0, idesc, acc);
#pragma unroll
            for (int j = 1; j < 4; j++) mma_ts<CG>(d, am + 8 * j, b0 + 2 * j, idesc, 1u);
#pragma unroll
            for (int j = 0; j < 4; j++) mma_ts<CG>(d, am + 32 + 8 * j, b1 + 2 * j, idesc, 1u);
            commit<CG>(a_empty + 8 * s);
            commit<CG>(b_empty + 8 * bt);
          }
          acc = 1;
        } else {  // the pair's second CTA: its operands are ready, tell the one that issues
          tc_fence_before();
          if (leader) mbar_arrive_remote(mapa(peer_full + 8 * s, 0));
        }
        if (++bt == a.nbs) bt = 0, bph ^= 1;
        if (++s == NAS) s = 0, par ^= 1;
        __syncwarp();
        if (k + 1 < stages) ready = look();
      }
      if (ok && rank == 0 && leader) commit<CG>(d_full + 8 * (seg & 1));
      __syncwarp();
      pos += u1 - u0;
    }
    if (rank == 0) {  // no MMA may be in flight when tensor memory is given back, whichever way the loop ended
      if (leader) commit<CG>(drained);
      __syncwarp();
      for (int i = 0; i < (1 << 16) && !__all_sync(0xffffffffu, mbar_test_wait(drained, 0)); i++) {
      }
    }
  } else if (warp < 8) {
    // ================================================================ expanders
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t wslot = sRaw + (uint32_t)warp * NSLOT * 32 * F::PITCH;
    const size_t stride = Row::row_stride(ctx, a.K);
    const int rofs = 128 * rank + quad * 32;  // the warp's first row within the tile
    struct Cursor {
      int c, u, t;  // chunk of the run, chunk within the tile, tile
    };
    auto at = [&](int c) {
      const long long p = pos0 + c;
      Cursor q;
      q.c = c, q.t = (int)(p / nb), q.u = (int)(p - (long long)q.t * nb);
      return q;
    };
    // ---- the copies run ahead of the expansion by NSLOT chunks of this warp
    Cursor ic = at(half);
    const uint8_t *ibase = nullptr, *ilim = nullptr;
    uint32_t roff[F::GR];
    constexpr bool SKEWED = std::is_same<Row, Q6KRow>::value;
    auto aim = [&]() {
      const Tile T = wk.tile(ic.t);
      const int nw = min(T.n0 + rofs, a.N - 1);
      Row r0;
      r0.init(ctx, T.expert, nw, a.N, a.K);
      ibase = row_ptr(r0);
      if constexpr (SKEWED) ilim = r0.raw_end();
#pragma unroll
      for (int i = 0; i < F::GR; i++) {
        const int q = lane + 32 * i, rr = q / F::GR, piece = q - rr * F::GR;
        roff[i] = (uint32_t)(min(T.n0 + rofs + rr, a.N - 1) - nw) * (uint32_t)stride + (SKEWED ? 0 : piece * 16);
      }
    };
    if (ic.c < n) aim();
    int islot = 0;
    constexpr int CBYTES = SKEWED ? 210 : std::is_same<Row, Q4KRow>::value ? 144 : std::is_same<Row, Q80Row>::value ? 272 : std::is_same<Row, DenseRow>::value ? 256 : 128;
    auto issue = [&]() {  // always closes a commit group
      if (ic.c < n) {
        const uint8_t *src = ibase + (size_t)ic.u * CBYTES;
        const uint32_t dst = wslot + islot * (32 * F::PITCH);
#pragma unroll
        for (int i = 0; i < F::GR; i++) {
          const int q = lane + 32 * i, rr = q / F::GR, piece = q - rr * F::GR;
          const uint32_t d = dst + (F::PITCH == F::GR * 16 ? (uint32_t)q * 16u : (uint32_t)(rr * F::PITCH + piece * 16));
          if constexpr (SKEWED) {  // the 16-byte granules that cover the block
            const uint8_t *s = reinterpret_cast<const uint8_t *>((uintptr_t)(src + roff[i]) & ~(uintptr_t)15) + piece * 16;
            if (s + 16 <= ilim) cp_async16(d, s);
            else if (s < ilim) cp_async16_part(d, s, (uint32_t)(ilim - s));
          } else {
            cp_async16(d, src + roff[i]);
          }
        }
        islot = islot + 1 == NSLOT ? 0 : islot + 1;
        ic.c += 2, ic.u += 2;
        if (ic.u >= nb && ic.c < n) {
          while (ic.u >= nb) ic.u -= nb, ic.t++;
          aim();
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < NSLOT; i++) issue();

    // ---- expansion
    Cursor cc = at(half);
    Row cur;
    auto init_row = [&]() {
      const Tile T = wk.tile(cc.t);
      cur.init(ctx, T.expert, min(T.n0 + rofs + lane, a.N - 1), a.N, a.K);
    };
    auto advance = [&]() {
      cc.c += 2, cc.u += 2;
      if (cc.u >= nb && cc.c < n) {
        while (cc.u >= nb) cc.u -= nb, cc.t++;
        init_row();
      }
    };
    if (cc.c < n) init_row();
    if constexpr (HasAux<Row>::value) {
      if (cc.c < n) cur.aux = cur.fetch_aux(cc.u);
    }
    int slot = 0, pending = -1;
    bool ok = true;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    auto deliver = [&]() {  // the stage stored last is complete: hand it to the MMA warp
      if (pending >= 0) {
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + 8 * pending);
        pending = -1;
      }
    };
    for (int c = half; c < n && ok; c += 2) {
      cp_async_wait<NSLOT - 1>();
      __syncwarp();
      const uint32_t rs = wslot + slot * (32 * F::PITCH) + lane * F::PITCH;
#pragma unroll
      for (int l = 0; l < F::LOADS; l++) {
        if constexpr (HasAux<Row>::value || std::is_same<Row, DenseRow>::value) cur.load_codes(rs + 128 * l);
        else cur.load_smem(rs, cc.u * F::LOADS + l);
        [[maybe_unused]] const Row here = cur;  // (registers; the pointers move on below)
        if (l == F::LOADS - 1) {
          __syncwarp();
          issue();  // into the slot just read
          advance();
        }
        if constexpr (HasAux<Row>::value) {  // the next chunk's scales arrive while this one is expanded
          if (cc.c < n) cur.aux = cur.fetch_aux(cc.u);
        }
#pragma unroll
        for (int j = 0; j < SPL; j++) {
          const int it = c * SPC + l * SPL + j, s = (it >> 1) % NAS;
          uint32_t o[32];
          here.template emit<BF16>(j, [&](int ch, const uint4 &v) { o[4 * ch] = v.x, o[4 * ch + 1] = v.y, o[4 * ch + 2] = v.z, o[4 * ch + 3] = v.w; });
          if (!((l * SPL + j) & 1)) {  // a new stage: hand over the one before, wait until this one's MMAs have completed
            deliver();
            if (it >= 2 * NAS) {
              if (!warp_wait(a_empty + 8 * s, ((it / (2 * NAS)) - 1) & 1, abort)) {
                ok = false;
                break;
              }
              tc_fence_after();
            }
          }
          __syncwarp();
          tmem_st32(tmem + lanes + A_COL + 64 * s + 32 * (it & 1), o);
          if ((l * SPL + j) & 1) pending = s;
        }
        if (!ok) break;
      }
      slot = slot + 1 == NSLOT ? 0 : slot + 1;
    }
    deliver();
    cp_async_wait<0>();
  } else {
    // ================================================================ epilogue
    const int quad = warp & 3, row = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    float *const mine = a.parts + (size_t)blockIdx.x * PART_FLOATS + row;
    int seg = 0;
    for (long long pos = pos0; pos < pos1; seg++) {
      const int t = (int)(pos / nb), u0 = (int)(pos - (long long)t * nb), u1 = (int)min((long long)nb, u0 + (pos1 - pos));
      const Tile T = wk.tile(t);
      pos += u1 - u0;
      if (!warp_wait(d_full + 8 * (seg & 1), (seg >> 1) & 1, abort)) break;
      tc_fence_after();
      const uint32_t d = tmem + lanes + (T.nt > 128 ? 0 : 128 * (seg & 1));
      const bool owner = u0 == 0, whole = owner && u1 == nb;
      int jlast = cta;
      bool ok = true;
      if (owner && !whole) {  // the runs that hold the rest of this tile
        const long long tile_end = (long long)(t + 1) * nb;
        long long b = pos1;
        while (jlast + 1 < G && b < tile_end) {
          const long long b1 = wk.bound(++jlast + 1, G);
          if (b1 > b && !wait_flag(g_flags + (jlast * CG + rank) * 4 + quad, abort)) ok = false;
          b = b1;
        }
      }
      const int ncol = T.m_end - T.m0, col = T.n0 + 128 * rank + row;
      const bool live = col < a.N;
#pragma unroll 1
      for (int c0 = 0; c0 < T.nt; c0 += 32) {
        uint32_t v[32];
        __syncwarp();
        if (c0 + 32 <= T.nt) {
          tmem_ld32(d + c0, v);
        } else {
          uint32_t h[16];
          tmem_ld16(d + c0, h);
#pragma unroll
          for (int i = 0; i < 16; i++) v[i] = h[i], v[16 + i] = 0u;
        }
        tmem_ld_wait();
        if (c0 + 32 >= T.nt) {  // the last of it is in registers: the accumulator is free
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (CG == 1) mbar_arrive(d_empty + 8 * (seg & 1));
            else mbar_arrive_remote(mapa(d_empty + 8 * (seg & 1), 0));
          }
        }
        if (!owner) {  // (columns past the tile's tokens are written and read too: the slot has room for 256)
#pragma unroll
          for (int i = 0; i < 32; i++) __stcg(mine + (c0 + i) * 128, __uint_as_float(v[i]));
          continue;
        }
        for (int j = cta + 1; j <= jlast && ok; j++) {
          if (a.offsets && wk.bound(j, G) == wk.bound(j + 1, G)) continue;  // an empty run wrote nothing
          const float *theirs = a.parts + (size_t)(j * CG + rank) * PART_FLOATS + row + c0 * 128;
          float p[32];
#pragma unroll
          for (int i = 0; i < 32; i++) p[i] = __ldcg(theirs + i * 128);
#pragma unroll
          for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) + p[i]);
        }
        if (!a.offsets) {  // consecutive output rows
          OutT *o = out + (size_t)(T.m0 + c0) * a.N + col;
          if (c0 + 32 <= ncol) {
#pragma unroll
            for (int i = 0; i < 32; i++, o += a.N) st_if(live, o, __uint_as_float(v[i]));
          } else {
#pragma unroll
            for (int i = 0; i < 32; i++, o += a.N) st_if(live && c0 + i < ncol, o, __uint_as_float(v[i]));
          }
        } else {
          int prow = -1;  // output row and weight of token c0 + lane
          float pw = 1.f;
          if (c0 + lane < ncol) {
            const long long p = a.pairs[T.m0 + c0 + lane];
            if (p >= 0 && p < a.size_m) {
              prow = (int)p;
              if (a.topkw) pw = a.topkw[p];
            }
          }
          OutT *o = out + col;
#pragma unroll
          for (int i0 = 0; i0 < 32; i0 += 8) {
            int m[8];
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; i++) m[i] = __shfl_sync(0xffffffffu, prow, i0 + i), f[i] = __shfl_sync(0xffffffffu, pw, i0 + i) * __uint_as_float(v[i0 + i]);
#pragma unroll
            for (int i = 0; i < 8; i++) st_if(live && m[i] >= 0, o + (long long)m[i] * a.N, f[i]);
          }
        }
      }
      __syncwarp();
      if (!owner) {  // this warp's rows of the partial tile are written: raise its flag
        __threadfence();
        __syncwarp();
        if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(g_flags + blockIdx.x * 4 + quad), "r"(1u) : "memory");
      } else if (!whole) {  // the partials have been read: lower the flags for the next launch
        for (int j = cta + 1 + lane; j <= jlast; j += 32) g_flags[(j * CG + rank) * 4 + quad] = 0u;
      }
    }
  }
  __syncwarp();
  if (abort_flag && threadIdx.x == 0) g_status = 1;
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync();  // nobody leaves while the peer may still signal its barriers
  if (warp == MMA_WARP) dealloc512<CG>(tmem);
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static const EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeTiledFn)p : (EncodeTiledFn) nullptr;
  }();
  return fn;
}
int knob(const char *name, int otherwise) {
  const char *e = getenv(name);
  return e ? atoi(e) : otherwise;
}

template <typename Row> constexpr int narrow_slots() { return Fmt<Row>::PITCH > 144 ? 2 : 4; }

template <typename Row, bool BF16, typename OutT, int CG, int NSLOT>
int run(const typename Row::Ctx &ctx, const TmemCall &c, Args a, int nt_max, cudaStream_t st) {
  using F = Fmt<Row>;
  // token ring: what shared memory the weight slots leave, up to eight stages of 64 k
  a.nt_max = nt_max;
  const int rows = nt_max / CG;
  a.box = c.offsets ? 32 : rows;
  a.stage_bytes = (rows + a.box - 1) / a.box * a.box * 256;
  const int fixed = 8 * NSLOT * 32 * F::PITCH + 512 + (a.E + 1) * 12 + 16 + 1024;
  a.nbs = (SMEM_MAX - fixed) / a.stage_bytes;
  if (a.nbs > 8) a.nbs = 8;
  if (a.nbs < 2) return 0;
  int G = sm_count() / CG;
  if (G * CG > MAX_GRID) G = MAX_GRID / CG;
  if (!c.offsets) {
    const int ntt = (int)((c.M + nt_max - 1) / nt_max);
    const long long U = (long long)ntt * ((c.N + 128 * CG - 1) / (128 * CG)) * (c.K / F::KU), least = c.min_run_k / F::KU;
    if (U / least < G) G = (int)(U / least > 0 ? U / least : 1);
  }
  if (c.parts_bytes < (size_t)G * CG * PART_FLOATS * 4) return 0;
  a.parts = (float *)c.parts;
  const EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(LB200_E_DEVICE, "light_b200: cuTensorMapEncodeTiled is not available from the driver");
  CUtensorMap tm;
  const cuuint64_t dims[2] = {(cuuint64_t)c.K, (cuuint64_t)c.M};
  const cuuint64_t strides[1] = {(cuuint64_t)c.K * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)a.box}, estr[2] = {1, 1};
  const CUresult r = enc(&tm, BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(c.x16), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(LB200_E_SHAPE, "light_b200: cuTensorMapEncodeTiled failed (%d)", (int)r);
  auto kern = gemm_tmem_kernel<Row, BF16, OutT, CG, NSLOT>;
  const int smem = a.nbs * a.stage_bytes + fixed;
  static DeviceOnce attr;
  cudaError_t e = attr.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX); });
  if (e != cudaSuccess) return fail((int)e, "light_b200: gemm (tmem): %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(G * CG));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CG, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
  cfg.attrs = at, cfg.numAttrs = CG > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, tm, ctx, a, (OutT *)c.out);
  if (e != cudaSuccess) return fail((int)e, "light_b200: gemm (tmem): %s", cudaGetErrorString(e));
  if (int rc = launched("gemm (weights through tensor memory)")) return rc;
  return 1;
}

template <typename Row, bool BF16, typename OutT>
int pick(const typename Row::Ctx &ctx, const TmemCall &c, cudaStream_t st) {
  if (c.K % Fmt<Row>::KU || c.E > MAX_E) return 0;
  Args a = {};
  a.offsets = c.offsets, a.pairs = c.pairs, a.topkw = c.topkw, a.size_m = c.size_m;
  a.E = c.offsets ? c.E : 1, a.M = (int)c.M, a.N = c.N, a.K = c.K;
  static const int k_cg = knob("LIGHT_B200_TMEM_CG", 0), k_nt = knob("LIGHT_B200_TMEM_NT", 0), k_wmin = knob("LIGHT_B200_TMEM_WMIN", 96);
  a.wmin = k_wmin;
  // the token tile: at most 256, all tiles of a matrix alike
  const int cap = k_nt ? k_nt : 256;
  int cg = k_cg ? k_cg : c.mean_tokens > 192 ? 2 : 1;
  int nt = cap;
  if (!c.offsets) {
    const int ntt = (int)((c.M + cap - 1) / cap);
    nt = (int)((c.M + ntt - 1) / ntt + 16 * cg - 1) / (16 * cg) * (16 * cg);
  }
  if (cg == 2) return run<Row, BF16, OutT, 2, 1>(ctx, c, a, nt, st);
  if (nt <= 64) return run<Row, BF16, OutT, 1, narrow_slots<Row>()>(ctx, c, a, nt, st);
  return run<Row, BF16, OutT, 1, 1>(ctx, c, a, nt, st);
}

}  // namespace

size_t gemm_tmem_parts_bytes() { return (size_t)MAX_GRID * PART_FLOATS * 4; }

int gemm_tmem(const TmemCall &c, cudaStream_t st) {
  switch (c.kind) {
    case TmemCall::Q4K: return pick<Q4KRow, false, float>(GgufCtx{(const uint8_t *)c.w}, c, st);
    case TmemCall::Q6K: return pick<Q6KRow, false, float>(GgufCtx{(const uint8_t *)c.w}, c, st);
    case TmemCall::Q80: return pick<Q80Row, false, float>(GgufCtx{(const uint8_t *)c.w}, c, st);
    case TmemCall::INT4:
      if (c.bf16) return pick<Int4Row, true, __nv_bfloat16>(Int4Ctx{(const uint32_t *)c.w, c.s, c.z, c.G}, c, st);
      return pick<Int4Row, false, float>(Int4Ctx{(const uint32_t *)c.w, c.s, c.z, c.G}, c, st);
    case TmemCall::FP8:
      if (c.bf16) return pick<Fp8Row, true, __nv_bfloat16>(Fp8Ctx{(const uint8_t *)c.w, c.s, c.bR, c.bC}, c, st);
      return pick<Fp8Row, false, float>(Fp8Ctx{(const uint8_t *)c.w, c.s, c.bR, c.bC}, c, st);
    case TmemCall::DENSE: return pick<DenseRow, true, __nv_bfloat16>(DenseCtx{(const uint16_t *)c.w}, c, st);
  }
  return 0;
}

int gemm_tmem_status() {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, g_status, sizeof(int));
  return e == cudaSuccess ? v : -(int)e;
}

}  // namespace lb
