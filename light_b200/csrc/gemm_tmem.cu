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
//   warps 0-15   expanders.  The four warps w, w + 4, .. own rows 32 (w & 3) .. + 31 (the TMEM lanes a warp can reach) and
//                take turns at the units of 128 k: a unit's packed rows arrive by cp.async in the warp's own slot, go into
//                registers (the slot then takes the next copy) and leave as 64 TMEM columns.  Expansion is a chain of
//                short dependent instructions: two warps per row quarter instead of four ran it at 4 to 8 clocks each
//                and set the pace wherever a tile had few tokens (4-bit rows at 2048 tokens: 1092 against 1335 TFLOP/s).
//   warps 16-17  one lane of each: TMA of the token tiles, 64 of a unit's 128 k to each warp, one box to a unit.  (One lane for
//                both halves, in boxes of 16 or 32 tokens where groups are ragged, chosen by its number instead of elected so that
//                operands went through vector registers: 240 clocks to a box, 470 to 730 per unit, and the MMAs of a tile of few
//                tokens waited for those: 64 bf16 pairs over 64 experts of 4096 x 7168 247 -> 220 us, with 128 tokens to an expert
//                744 -> 704, Q4_K experts of 1536 x 2048 with 5 tokens each 109 -> 95.)
//   warp  18     MMAs and commits; in the second CTA of a pair: forwards "my half is ready" to the first.
//   warps 19-22  epilogue, while the next tile's MMAs run (token tiles up to 128 use two accumulators; beyond, the MMAs wait until the
//                last chunk is out of tensor memory): TMEM -> registers -> a [token][row] strip of the warp's own in shared memory
//                -> a box of 16 tokens, or 16 bytes a lane where tokens go to rows of their own.  (One strip for the four warps, two
//                barriers and a bulk copy per token: 1600 clocks for 32 tokens; Q4_K 28672 x 4096, 2048 tokens 388 -> 375 us, a
//                4-bit layer of 4096 tokens 1830 -> 1786.)  The run's last segment is finished by the expanders too, five warps to
//                a row quarter, each 16 tokens at a time.
//
// Work is the list of (tile, K chunk) pairs, cut into equal runs, one per CTA (pair): stream-K.  A segment that does not
// start its tile writes a partial tile and sets its flags to the launch's tag, which it does first; the segment that starts the
// tile owns it and adds the partials in run order.  In a grouped launch the units are weighted by their token count, so that runs are
// equal in time.  Every wait is bounded; on giving up the status word is set, TMEM is freed and the CTA retires.
#include <cuda.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "mma_sync.cuh"
#include "tmem_ops.cuh"
#include "tmem_rows.cuh"
#include "umma.cuh"

namespace lb {
namespace {

constexpr int EXPANDERS = 16, TMA_WARP = 16, MMA_WARP = 18, EPI_WARP = 19, THREADS = 23 * 32;
constexpr int KU = 128;                       // k of a unit: one TMEM stage, one stage of the token ring
constexpr int NAS = 4;                        // stages of expanded weights: 128 k, 64 TMEM columns each
constexpr int NBS = 12;                       // most stages of the token ring, 128 k each
constexpr int A_COL = 256;                    // columns 0-255: accumulators, 256-511: weight stages
constexpr int MAX_E = 1024;                   // experts whose prefix sums fit the shared tables
constexpr int BAR_BYTES = 640;                // barriers
constexpr int MAX_ROWS = 128;                 // most token rows of a stage (one SM's)
constexpr int PART_FLOATS = 256 * 128;        // one partial tile: [token][row]

__device__ int g_status;                      // non-zero: a bounded wait gave up (sticky)
__device__ Sync g_sync;  // of the launches without one of their own; a flag per (CTA, row quarter, 16-token chunk)

struct Args {
  const int32_t *offsets;   // grouped: expert e owns rows offsets[e] .. offsets[e + 1] of the (gathered) tokens; null: one matrix
  const int64_t *pairs;     // grouped: token row i goes to output row pairs[i] ...
  const float *topkw;       // ... scaled by its routing weight (or null)
  const float *factor;      // f16 tokens over a power of two each: token row i is to be multiplied by factor[i] (null: as they are)
  const int32_t *modes;     // see TmemCall
  int mode;                 // with modes: of the experts that are this launch's
  const uint4 *tokens;      // with factor: see TmemCall
  uint4 *x16;
  int topk, row_per_pair;
  long long size_m;
  int E, M, N, K;
  int nt_max;               // most tokens of a tile
  int stage_bytes, nbs;     // of the token ring, per CTA
  int wmin;                 // grouped: a unit's weight is max(tokens of its tile, wmin)
  struct Sync *sync;
  float *parts;
};

struct Tile {
  int expert, n0, m0, m_end, nt;
};

__device__ __forceinline__ void st_if(bool p, float *o, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}\n" ::"l"(o), "f"(v), "r"((int)p) : "memory");
}
__device__ __forceinline__ void st_if(bool p, __nv_bfloat16 *o, float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.b16 [%0], %1;\n\t}\n" ::"l"(o), "h"(*reinterpret_cast<const uint16_t *>(&b)), "r"((int)p)
               : "memory");
}
// ------------------------------------------------------------------------------------ work list
// Experts with their token tiles: preT[e] tiles and preW[e] weighted units before expert e.  Within an expert the token
// tiles of one row tile follow one another, so that its packed weights are read from HBM once and from L2 after that.
template <int CG, bool MODES>  // MODES: some experts may be another launch's
struct Work {
  const Args &a;
  const int *preT, *preW, *counts;  // counts (MODES): of the experts that are this launch's, with MODE_APART
  int nb, nrt;
  __device__ __forceinline__ int count_of(int e) const { return a.offsets ? a.offsets[e + 1] - a.offsets[e] : a.M; }
  __device__ __forceinline__ int count(int e) const { return MODES ? counts[e] & (MODE_APART - 1) : count_of(e); }
  __device__ __forceinline__ int first(int e) const { return a.offsets ? a.offsets[e] : 0; }
  __device__ __forceinline__ void geo(int cnt, int &ntt, int &nt) const {
    ntt = (cnt + a.nt_max - 1) / a.nt_max;
    nt = ntt ? ((cnt + ntt - 1) / ntt + 16 * CG - 1) / (16 * CG) * (16 * CG) : 0;
  }
  __device__ __forceinline__ int weight(int nt) const { return a.offsets ? max(nt, a.wmin) / 16 : 1; }
  __device__ __forceinline__ int expert_of(const int *pre, int v) const {  // the expert with pre[e] <= v < pre[e + 1]
    int lo = 0, hi = a.E - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (pre[mid + 1] <= v) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  }
  // A walk over the list: the search once, then one tile after the other.
  struct Walk {
    int t, e, rt, tt, ntt, nt, first, cnt;
  };
  __device__ __forceinline__ Walk walk(int t) const {
    Walk w;
    w.t = t, w.e = expert_of(preT, t), w.cnt = count(w.e), w.first = first(w.e);
    geo(w.cnt, w.ntt, w.nt);
    const int r = t - preT[w.e];
    w.rt = w.ntt ? r / w.ntt : 0, w.tt = r - w.rt * w.ntt;
    return w;
  }
  __device__ __forceinline__ void next(Walk &w, int stride) const {
    if (stride > 1) {
      if (w.t + stride < preT[a.E]) w = walk(w.t + stride);
      return;
    }
    w.t++;
    if (++w.tt < w.ntt) return;
    w.tt = 0;
    if (++w.rt < nrt) return;
    w.rt = 0;
    if (MODES && a.modes && a.mode) {  // (few experts of many: no walk from one to the next)
      if (w.t < preT[a.E]) w = walk(w.t);
      return;
    }
    do w.e++;
    while (w.e < a.E && count(w.e) == 0);
    if (w.e >= a.E) return;  // (the list's end)
    w.cnt = count(w.e), w.first = first(w.e);
    geo(w.cnt, w.ntt, w.nt);
  }
  __device__ __forceinline__ Tile tile(const Walk &w) const {
    Tile T;
    T.expert = w.e, T.nt = w.nt, T.n0 = w.rt * 128 * CG, T.m0 = w.first + w.tt * w.nt, T.m_end = min(w.first + w.cnt, T.m0 + w.nt);
    return T;
  }
  // first unit (tile-major) of run j of G
  __device__ __forceinline__ int bound(int j, int G) const {
    if (j >= G) return preT[a.E] * nb;
    const int W = preW[a.E], q = W / G, w = q * j + min(j, W - q * G);
    if (!a.offsets) return w;
    const int e = expert_of(preW, w);
    int ntt, nt;
    geo(count(e), ntt, nt);
    return preT[e] * nb + (w - preW[e]) / weight(nt);
  }
};

// The rows of experts that are left to the bf16 launch, as they are: nothing in this launch makes use of them.
__device__ __noinline__ void copy_rows(const Args &a) {
  const int lane = threadIdx.x & 31, pieces = a.K >> 3;
  for (int e = 0; e < a.E; e += 32) {
    unsigned left = __ballot_sync(0xffffffffu, e + lane < a.E && (a.modes[min(e + lane, a.E - 1)] & MODE_BF16));
    while (left) {
      const int f = e + __ffs(left) - 1;
      left &= left - 1;
      for (int i = a.offsets[f] + (int)blockIdx.x; i < a.offsets[f + 1]; i += gridDim.x) {
        const long long p = a.pairs[i];
        const bool ok = p >= 0 && p < a.size_m;
        const uint4 *src = a.tokens + (ok ? (size_t)(a.row_per_pair ? p : p / a.topk) * pieces : 0);
        for (int k = threadIdx.x; k < pieces; k += THREADS) a.x16[(size_t)i * pieces + k] = ok ? __ldg(src + k) : make_uint4(0, 0, 0, 0);
      }
    }
  }
}

// ------------------------------------------------------------------------------------ kernel
template <typename OutT>
constexpr uint32_t STRIP = 32 * 128 * sizeof(OutT);  // 32 tokens of 128 output columns
template <typename OutT>
constexpr int STRIPS = 2 * STRIP<OutT>;

struct Maps {
  CUtensorMap x[MAX_ROWS / 16], w[3];  // tokens, by the rows of a box (16, 32, ..); the weight rows, per box of the format
  CUtensorMap out;                     // one matrix: 16 tokens of 32 output columns
};

template <typename Row, bool BF16, typename OutT, int CG>
__global__ void __launch_bounds__(THREADS, 1) gemm_tmem_kernel(const __grid_constant__ Maps maps, const typename Row::Ctx ctx,
                                                              const __grid_constant__ Args a, OutT *__restrict__ out) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ int abort_flag;
  __shared__ uint32_t tmem_sh;
  __shared__ unsigned tag_sh;  // this launch's tag, there once `tagged` is complete
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char *gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sB = base, sRaw = base + (uint32_t)a.nbs * a.stage_bytes, sStrip = sRaw + (uint32_t)EXPANDERS * Row::SLOT, sBar = sStrip + STRIPS<OutT>;
  // full[s]: a stage's weights are there (four warps; in the first CTA of a pair also: the other CTA's weights and tokens);
  // empty[s]: its MMAs have completed.  t_full, t_empty: the token ring's, which runs further ahead: a token tile takes a TMA
  // latency to refill, and with only four stages that, not the tensor core, set the pace of narrow tiles.
  const uint32_t full = sBar, empty = full + 8 * NAS, d_full = empty + 8 * NAS, d_empty = d_full + 16, drained = d_empty + 16, w_full = drained + 8,
                 t_full = w_full + 8 * EXPANDERS, t_empty = t_full + 8 * NBS, tagged = t_empty + 8 * NBS;
  int *preW = reinterpret_cast<int *>(gen + (sBar - base) + BAR_BYTES), *preT = preW + a.E + 1;
  [[maybe_unused]] int *const counts = preT + a.E + 1;
  const int warp = same((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = CG == 2 ? same((int)cluster_ctarank()) : 0;
  const Work<CG, HasModes<Row>::value> wk{a, preT, preW, counts, a.K / KU, (a.N + 128 * CG - 1) / (128 * CG)};
  const int nb = wk.nb;
  const int G = gridDim.x / CG, cta = blockIdx.x / CG;

  if (threadIdx.x == 0) {
    if (!a.offsets) prefetch_tmap(&maps.x[a.nt_max / CG / 16 - 1]);
    if constexpr (Row::BOXES > 0) prefetch_tmap(&maps.w[0]);
    if constexpr (Row::BOXES > 1) prefetch_tmap(&maps.w[1]);
    if constexpr (Row::BOXES > 2) prefetch_tmap(&maps.w[2]);
    abort_flag = 0;
    for (int i = 0; i < NAS; i++) mbar_init(full + 8 * i, CG == 2 && rank == 0 ? 5 : 4), mbar_init(empty + 8 * i, 1);
    for (int i = 0; i < a.nbs; i++) mbar_init(t_full + 8 * i, 2), mbar_init(t_empty + 8 * i, 1);
    for (int i = 0; i < 2; i++) mbar_init(d_full + 8 * i, 1), mbar_init(d_empty + 8 * i, 4 * CG);
    mbar_init(drained, 1), mbar_init(tagged, 1);
    for (int i = 0; i < EXPANDERS; i++) mbar_init(w_full + 8 * i, 1);
    fence_barrier_init();
  }
  // (every CTA of this grid is resident once all have come by here: the next kernel's wait for room, and for its operands)
  pdl_launch_dependents();
  if (a.offsets) pdl_wait();
  [[maybe_unused]] int others = 0;
  if constexpr (HasModes<Row>::value) {
    bool any = false;
    for (int e = threadIdx.x; e < a.E; e += THREADS) {
      const int cnt = wk.count_of(e), m = a.modes ? a.modes[e] : a.mode;
      counts[e] = (m & MODE_BF16) == a.mode ? cnt | (m & MODE_APART) : 0;
      any |= cnt > 0 && (m & MODE_BF16) == a.mode, others |= m & MODE_BF16;
    }
    if (a.modes && a.mode && !__syncthreads_or(any)) return;  // (mostly: no expert is left to the bf16 launch)
  }
  for (int e = threadIdx.x; e < a.E; e += THREADS) {
    int ntt, nt;
    wk.geo(wk.count(e), ntt, nt);
    preT[e + 1] = ntt * wk.nrt;
    preW[e + 1] = ntt * wk.nrt * nb * wk.weight(nt);
  }
  if (warp == MMA_WARP) alloc512<CG>(smem_u32(&tmem_sh));
  if constexpr (Unscales<Row>::value) others = __syncthreads_or(others);
  else __syncthreads();
  if (Unscales<Row>::value && others) copy_rows(a);
  if (warp == 0) {  // inclusive prefix sums, 32 experts at a time
    int ct = 0, cw = 0;
    for (int e0 = 0; e0 < a.E; e0 += 32) {
      int t = e0 + lane < a.E ? preT[e0 + lane + 1] : 0;
      int w = e0 + lane < a.E ? preW[e0 + lane + 1] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int tt = __shfl_up_sync(0xffffffffu, t, d);
        const int ww = __shfl_up_sync(0xffffffffu, w, d);
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
  const uint32_t tmem = same(tmem_sh);
  volatile int *abort = &abort_flag;
  // This CTA (pair)'s run: n units from unit v0 of tile tf on, then tile tf + stride, ...  Where there are plenty of tiles a grouped
  // launch deals them out in turn instead: the tiles in flight are then neighbours, of a few experts whose tokens
  // stay in L2.  (Contiguous runs, one far from the other, read the tokens of 74 experts at once, more than L2 holds, and
  // from HBM again for every row tile.)
  const int total = same(preT[a.E]);
  const bool dealt = a.offsets && total >= 16 * G;
  const int pos0 = dealt ? cta * nb : same(wk.bound(cta, G)), tf = same(pos0 / nb), v0 = pos0 - tf * nb, stride = dealt ? G : 1;
  const int n = dealt ? same(total > cta ? (total - 1 - cta) / G + 1 : 0) * nb : same(wk.bound(cta + 1, G)) - pos0;
  const int v1 = v0 + n;

  if (warp >= TMA_WARP && warp < MMA_WARP) {
    pdl_wait();  // the tokens may be the kernel before's; the weights are not
    const int half = warp - TMA_WARP;
    const uint32_t first = sB + half * (a.stage_bytes / 2);
    uint32_t dst = first;
    int bt = 0, par = 1;
    bool wrapped = false, ok = true;
    auto W = wk.walk(tf);
    for (int v = v0; v < v1 && ok; wk.next(W, stride)) {
      const int u0 = same(v % nb), u1 = min(nb, u0 + (v1 - v));
      const Tile T = wk.tile(W);
      const int rows = same(T.nt / CG), y = same(T.m0) + rank * rows;
      const CUtensorMap *const map = &maps.x[rows / 16 - 1];
      int x = u0 * 128 + half * 64;
      for (int u = u0; u < u1; u++, x += 128) {
        const uint32_t bar = t_full + 8 * bt;
        if (wrapped && !warp_wait(t_empty + 8 * bt, par, abort)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(bar, (uint32_t)rows * 128u);
          tma_load_2d(dst, map, bar, x, y);
        }
        __syncwarp();
        dst += a.stage_bytes;
        if (++bt == a.nbs) bt = 0, par ^= 1, wrapped = true, dst = first;
      }
      v += u1 - u0;
    }
  } else if (warp == MMA_WARP) {
    // The whole warp runs the loop and one elected lane issues.  A pass is a chain of some 60 instructions that share their
    // scheduler with the expanders: with 64 k and two or three barriers per pass it took 700 clocks and the tensor pipe
    // stood at half its rate.  Hence 128 k to a stage, and the look at the next stage's barriers issued
    // before this stage's MMAs.  (128 x 16 x 128 in 8 MMAs and two commits: 110 clocks alone, 290 beside the expanders.)
    const bool leader = elect_one();
    int s = 0, par = 0, bt = 0, bpar = 0, seg = 0;
    bool ok = true, wide_before = false;
    auto W = wk.walk(tf);
    for (int v = v0; v < v1 && ok; seg++, wk.next(W, stride)) {
      const int u0 = same(v % nb), u1 = min(nb, u0 + (v1 - v));
      const int nt = same(W.nt);
      const bool wide = nt > 128;
      if (rank == 0) {  // the accumulators this segment overwrites must have been read out
        if (seg >= 2 && !warp_wait(d_empty + 8 * (seg & 1), ((seg - 2) >> 1) & 1, abort)) break;
        if (seg >= 1 && (wide || wide_before) && !warp_wait(d_empty + 8 * ((seg - 1) & 1), ((seg - 1) >> 1) & 1, abort)) break;
      }
      wide_before = wide;
      const uint32_t d = tmem + (wide ? 0 : 128 * (seg & 1));
      const uint32_t idesc = idesc_f16(128 * CG, 16, BF16) + ((uint32_t)((nt - 16) >> 3) << 17);
      const int stages = u1 - u0;
      uint32_t acc = 0;
      bool ready = mbar_test_wait(full + 8 * s, par), tokens = mbar_test_wait(t_full + 8 * bt, bpar);
      for (int k = 0; k < stages; k++) {
        if (!__all_sync(0xffffffffu, ready && tokens) && !(warp_wait(t_full + 8 * bt, bpar, abort) && warp_wait(full + 8 * s, par, abort))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t b0 = smem_desc_sw128(sB + bt * a.stage_bytes), b1 = b0 + (uint64_t)(a.stage_bytes >> 5);
        const uint32_t am = tmem + A_COL + 64 * s, done = empty + 8 * s, fwd = full + 8 * s, tdone = t_empty + 8 * bt;
        if (++s == NAS) s = 0, par ^= 1;
        if (++bt == a.nbs) bt = 0, bpar ^= 1;
        ready = mbar_test_wait(full + 8 * s, par), tokens = mbar_test_wait(t_full + 8 * bt, bpar);
        if (CG == 1 || rank == 0) {
          if (leader) {
            mma_ts<CG>(d, am, b0, idesc, acc);
#pragma unroll
            for (int j = 1; j < 4; j++) mma_ts<CG>(d, am + 8 * j, b0 + 2 * j, idesc, 1u);
#pragma unroll
            for (int j = 0; j < 4; j++) mma_ts<CG>(d, am + 32 + 8 * j, b1 + 2 * j, idesc, 1u);
            commit<CG>(done);
            commit<CG>(tdone);
          }
          acc = 1;
        } else {  // the pair's second CTA: its operands are ready, tell the one that issues
          tc_fence_before();
          if (leader) mbar_arrive_remote(mapa(fwd, 0));
        }
        __syncwarp();
      }
      if (ok && rank == 0 && leader) commit<CG>(d_full + 8 * (seg & 1));
      __syncwarp();
      v += u1 - u0;
    }
    // No MMA may be in flight when tensor memory is given back, whichever way the loop ended, nor an arrival on a barrier of the pair's second CTA when that
    // one leaves: each waits for its own.
    if (rank == 0 && leader) commit<CG>(drained);
    __syncwarp();
    for (int i = 0; i < (1 << 16) && !__all_sync(0xffffffffu, mbar_test_wait(drained, 0)); i++) {
    }
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;
    auto sync = [&]() { return a.sync ? a.sync : &g_sync; };  // (looked up where it is used: held, it cost the expanders registers)
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    // Columns c0 .. c0 + 31 of the accumulator at `d` into registers (a tile's last chunk may hold 16).
    auto take = [&](uint32_t d, int c0, int nt, uint32_t (&v)[32]) {
      __syncwarp();
      if (c0 + 32 <= nt) {
        tmem_ld32(d + c0, v);
        tmem_ld_wait();
      } else {
        uint32_t h[16];
        tmem_ld16(d + c0, h);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = h[i], v[16 + i] = 0u;
      }
    };
    // Sixteen columns of a partial tile (those past the tile's tokens are written and read too); then, once all of a warp's
    // chunks first, first + step, .. < nt are on their way, their flags.
    auto put_part = [&](int c0, const uint32_t *v) {
      float *mine = a.parts + (size_t)blockIdx.x * PART_FLOATS + row + c0 * 128;
#pragma unroll
      for (int i = 0; i < 16; i++) __stcg(mine + i * 128, __uint_as_float(v[i]));
    };
    auto raise_flags = [&](int first, int step, int nt, unsigned tag) {
      __threadfence();
      __syncwarp();
      const int c0 = first + lane * step;
      if (c0 < nt) asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(sync()->flags + (blockIdx.x * 4 + quad) * 16 + (c0 >> 4)), "r"(tag) : "memory");
    };
    // Rows over powers of two (Unscales): what a row block's sums are to be multiplied by (the warp's rows of the tile), negative where some token's
    // factor times its routing weight may leave f32's range, so that they are multiplied by one after the other; a token row's factor.
    [[maybe_unused]] auto unscale = [&](const Tile &T) {
      if constexpr (Unscales<Row>::value)
        return copysignf(Row::unscale(ctx, T.expert * a.N + min(T.n0 + 128 * rank + quad * 32, a.N - 1)), counts[T.expert] & MODE_APART ? -1.f : 1.f);
      else
        return 1.f;
    };
    [[maybe_unused]] auto factor = [&](const Tile &T, int c0) { return T.m0 + c0 + lane < T.m_end ? a.factor[T.m0 + c0 + lane] : 1.f; };
    // Output row (-1: none) and routing weight, with the row's factor if `joint`, of token c0 + lane of a tile.
    auto route = [&](const Tile &T, int c0, [[maybe_unused]] bool joint, int &prow, float &pw) {
      prow = -1, pw = 1.f;
      if (T.m0 + c0 + lane < T.m_end) {
        prow = T.m0 + c0 + lane;
        if (a.offsets) {
          const long long p = a.pairs[prow];
          prow = p >= 0 && p < a.size_m ? (int)p : -1;
          if (prow >= 0 && a.topkw) pw = a.topkw[p];
        }
      }
      if constexpr (Unscales<Row>::value)
        if (joint) pw *= factor(T, c0);
    };
    // The run's last segment, 16 tokens at a time: chunks first, first + step, ...  `shared`: five warps of this row quarter take
    // turns (only where K is long enough that an expander cannot get here before the segment before the last but one is
    // complete: the barrier's phase parity tells those two apart from one another, not from earlier ones).  What a chunk
    // costs is latency (flags, partial sums, stores): the flags of all runs that hold a part of the tile are polled at
    // once, a lane to each, and the partial sums of two runs are on their way together.
    const bool shared = nb >= 8;
    auto finish_last = [&](int first, int step) {
      const int seg = (v1 - 1) / nb, t = tf + seg * stride, u0 = seg ? 0 : v0, u1 = v1 - seg * nb;
      const Tile T = wk.tile(wk.walk(t));
      if (first >= T.nt) return;
      const bool owner = u0 == 0;
      int jlast = cta;  // the runs that hold the rest of this tile
      if (owner && u1 < nb)
        while (jlast + 1 < G && wk.bound(jlast + 1, G) < (t + 1) * nb) jlast++;
      const int col = T.n0 + 128 * rank + row;
      const bool live = col < a.N;
      const float scale = unscale(T);
      if (!warp_wait(d_full + 8 * (seg & 1), (seg >> 1) & 1, abort) || !warp_wait(tagged, 0, abort)) return;
      tc_fence_after();
      const unsigned tag = tag_sh;
      const uint32_t d = tmem + lanes + (T.nt > 128 ? 0 : 128 * (seg & 1));
      if (jlast > cta) {  // all parts of this warp's chunks: (run, chunk) pairs, a lane to each
        const int chunks = (T.nt - first + step - 1) / step;
        for (int i0 = 0; i0 < (jlast - cta) * chunks; i0 += 32) {
          const int i = i0 + lane, j = min(cta + 1 + i / chunks, jlast), c0 = first + (i % chunks) * step;
          const bool has = i < (jlast - cta) * chunks && wk.bound(j, G) < wk.bound(j + 1, G);  // (an empty run writes nothing)
          if (!wait_flag(sync()->flags + ((j * CG + rank) * 4 + quad) * 16 + (c0 >> 4), tag, has, abort)) return;
        }
      }
#pragma unroll 1
      for (int c0 = first; c0 < T.nt; c0 += step) {
        uint32_t v[16];
        __syncwarp();
        tmem_ld16(d + c0, v);
        tmem_ld_wait();
        if (!owner) {
          put_part(c0, v);
          continue;
        }
        for (int j0 = cta + 1; j0 <= jlast; j0 += 32) {
          const int j = j0 + lane;
          const bool has = j <= jlast && wk.bound(j, G) < wk.bound(j + 1, G);
          unsigned left = __ballot_sync(0xffffffffu, has);
          const float *theirs = a.parts + row + c0 * 128 + (size_t)rank * PART_FLOATS;
          while (left) {
            const int ja = j0 + __ffs(left) - 1;
            left &= left - 1;
            const int jb = left ? j0 + __ffs(left) - 1 : -1;
            left &= left - 1;
            float p[16], q[16];
#pragma unroll
            for (int i = 0; i < 16; i++) p[i] = __ldcg(theirs + (size_t)ja * CG * PART_FLOATS + i * 128);
            if (jb >= 0) {
#pragma unroll
              for (int i = 0; i < 16; i++) q[i] = __ldcg(theirs + (size_t)jb * CG * PART_FLOATS + i * 128);
            }
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) + p[i]);
            if (jb >= 0) {
#pragma unroll
              for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) + q[i]);
            }
          }
        }
        if (!a.offsets) {  // consecutive output rows
          OutT *o = out + (size_t)(T.m0 + c0) * a.N + col;
          const int ncol = T.m_end - T.m0 - c0;
#pragma unroll
          for (int i = 0; i < 16; i++, o += a.N) st_if(live && i < ncol, o, __uint_as_float(v[i]));
        } else {
          int prow;
          float pw;
          route(T, c0, scale > 0.f, prow, pw);
          [[maybe_unused]] const float power = scale < 0.f ? factor(T, c0) : 1.f;
          OutT *o = out + col;
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const int m = __shfl_sync(0xffffffffu, prow, i);
            const float y = Unscales<Row>::value ? __uint_as_float(v[i]) * fabsf(scale) : __uint_as_float(v[i]);
            float f = __shfl_sync(0xffffffffu, pw, i) * y;
            if constexpr (Unscales<Row>::value) f *= __shfl_sync(0xffffffffu, power, i);
            st_if(live && m >= 0, o + (long long)m * a.N, f);
          }
        }
      }
      if (!owner) raise_flags(first, step, T.nt, tag);
    };

    if (warp < EXPANDERS) {
      // ================================================================ expanders
      const int set = warp >> 2;
      const uint32_t slot = sRaw + (uint32_t)warp * Row::SLOT, copied = w_full + 8 * warp;
      const int rofs = 128 * rank + quad * 32;  // the warp's first row within the tile
      if constexpr (std::is_same<Row, TmDense>::value) pdl_wait();  // (a dense weight may have been expanded just now)
      // this warp's next unit: number in the run, in the tile, and the tile
      int c = set, t = tf + (v0 + c) / nb * stride, u = (v0 + c) % nb;  // (a walk's state would cost these warps registers: they search)
      Row rowx(ctx);
      [[maybe_unused]] int y = 0;                 // TMA: the warp's first row among all experts' rows
      [[maybe_unused]] const uint8_t *src = nullptr;  // row copies: its address, and the rows of the matrix after it
      [[maybe_unused]] int rows = 0;
      auto aim = [&]() {
        const Tile T = wk.tile(wk.walk(t));
        const int nw = min(T.n0 + rofs, a.N - 1);
        const size_t r0 = (size_t)T.expert * a.N;
        y = same((int)(r0 + nw));
        if constexpr (Row::BOXES == 0) src = Row::base(ctx) + (r0 + nw) * Row::stride(a.K), rows = a.N - 1 - nw;
        rowx.row(ctx, (int)r0 + min(nw + lane, a.N - 1), a.K);
      };
      auto issue = [&]() {
        if constexpr (Row::BOXES > 0) {
          if (elect_one()) {
            mbar_arrive_expect_tx(copied, Row::BYTES);
            Row::copy(slot, maps.w, copied, u, y);
          }
        } else {
          // Lanes 10 r + i copy granule i of rows r, r + 3, ..: the granule's place in the block is the lane's own, and the
          // next row is one addition away.
          const int r0 = lane / 10, i = lane - 10 * r0;
          const size_t step = Row::stride(a.K);
          const uint8_t *at = src + (u >> 1) * 210;
          const uint32_t dst = slot + r0 * Row::PITCH + 16 * i;
          const int place = 16 * Row::number(u & 1, i);
          if (lane < 30) {
            if (rows >= 32) {  // (a whole row follows the last one: no copy passes the end of the matrix)
              at += (size_t)r0 * step;
#pragma unroll
              for (int k = 0; k < 11; k++, at += 3 * step)
                if (k < 10 || r0 < 2) cp_async16(dst + 3 * k * Row::PITCH, reinterpret_cast<const uint8_t *>((uintptr_t)at & ~(uintptr_t)15) + place);
            } else {
              const uint8_t *const end = Row::base(ctx) + (size_t)a.E * a.N * step;
              for (int k = 0; k < 11; k++)
                if (k < 10 || r0 < 2) {
                  const uint8_t *g = reinterpret_cast<const uint8_t *>((uintptr_t)(at + (size_t)min(r0 + 3 * k, rows) * step) & ~(uintptr_t)15) + place;
                  if (g + 16 <= end) cp_async16(dst + 3 * k * Row::PITCH, g);
                  else if (g < end) cp_async16_part(dst + 3 * k * Row::PITCH, g, (uint32_t)(end - g));
                }
            }
          }
          cp_async_commit();
        }
      };
      const uint32_t acol = tmem + lanes + A_COL + 64 * set;  // (four sets, four stages: always the same one)
      if (c < n) {
        aim();
        issue();
        rowx.fetch_scales(ctx, u);
      }
      bool ok = true;
      for (int round = 0; c < n && ok; round++) {
        if constexpr (Row::BOXES > 0) {
          if (!warp_wait(copied, round & 1, abort)) break;
        } else {
          cp_async_wait<0>();
          __syncwarp();
        }
        rowx.load(slot, u);
        const int now = u;
        auto next = [&]() {  // everything of this unit is in registers: on to the next one
          if constexpr (Row::BOXES > 0) fence_proxy_async();  // the reads above come before the copy that overwrites the slot
          __syncwarp();
          c += EXPANDERS / 4, u += EXPANDERS / 4;
          if (c < n) {
            if (u >= nb) {
              while (u >= nb) u -= nb, t += stride;
              aim();
            }
            issue();
            rowx.fetch_scales(ctx, u);
          }
        };
        if constexpr (!ReadsLate<Row>::value) next();
        rowx.template expand<BF16>(now, [&](int p, const uint32_t (&o)[16]) {
          if (p == 0 && round > 0) {  // the stage's MMAs of the round before
            ok = warp_wait(empty + 8 * set, (round - 1) & 1, abort);
            tc_fence_after();
          }
          __syncwarp();
          if (ok) tmem_st16(acol + 16 * p, o);
        });
        if constexpr (ReadsLate<Row>::value) next();
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * set);
      }
      if constexpr (Row::BOXES == 0) cp_async_wait<0>();
      __syncwarp();
      pdl_wait();
      if (ok && n > 0 && shared) finish_last(16 * (1 + set), 80);
    } else {
      // ================================================================ epilogue
      pdl_wait();  // `out` and the partial tiles may still be in use by the kernel before
      if (warp == EPI_WARP && lane == 0) {
        unsigned epoch;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(epoch) : "l"(&sync()->epoch) : "memory");
        tag_sh = epoch + 1;
        mbar_arrive(tagged);
        if (atomicInc(&sync()->readers, gridDim.x - 1) == gridDim.x - 1) atomicExch(&sync()->epoch, epoch + 1);  // every CTA has read it
      }
      __syncwarp();
      warp_wait(tagged, 0, abort);
      constexpr uint32_t SB = STRIP<OutT> / 4;  // of one warp
      const uint32_t strip = sStrip + 2 * SB * quad;
      const bool bulk = ((size_t)a.N * sizeof(OutT)) % 16 == 0 && ((uintptr_t)out & 15) == 0;
      int seg = 0, chunk = 0;
      auto W = wk.walk(tf);
      for (int v = v0; v < v1; seg++, wk.next(W, stride)) {
        const int u0 = v % nb, u1 = min(nb, u0 + (v1 - v));
        const Tile T = wk.tile(W);
        v += u1 - u0;
        if (v >= v1) {
          finish_last(0, shared ? 80 : 16);
          break;
        }
        const float scale = unscale(T);
        if (!warp_wait(d_full + 8 * (seg & 1), (seg >> 1) & 1, abort)) break;
        tc_fence_after();
        const uint32_t d = tmem + lanes + (T.nt > 128 ? 0 : 128 * (seg & 1));
        const int n0 = T.n0 + 128 * rank + 32 * quad;  // the warp's first output column (beyond N: no rows of the matrix here)
#pragma unroll 1
        for (int c0 = 0; c0 < T.nt; c0 += 32, chunk++) {
          uint32_t v[32];
          take(d, c0, T.nt, v);
          if (c0 + 32 >= T.nt) {  // the last of it is in registers: the accumulator is free
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if constexpr (CG == 1) mbar_arrive(d_empty + 8 * (seg & 1));
              else mbar_arrive_remote(mapa(d_empty + 8 * (seg & 1), 0));
            }
          }
          if (u0 > 0) {
            put_part(c0, v);
            if (c0 + 16 < T.nt) put_part(c0 + 16, v + 16);
            if (c0 + 32 >= T.nt) raise_flags(0, 16, T.nt, tag_sh);
            continue;
          }
          int prow;
          float pw;
          route(T, c0, scale > 0.f, prow, pw);
          if constexpr (Unscales<Row>::value) {
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * fabsf(scale));
          }
          if (a.topkw || a.factor) {
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, pw, i));
          }
          if constexpr (Unscales<Row>::value) {
            if (scale < 0.f) {
              const float power = factor(T, c0);
#pragma unroll
              for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, power, i));
            }
          }
          if (bulk) {  // through a strip of the warp's own: [32 tokens][32 rows], no other warp to wait for
            const uint32_t buf = strip + (chunk & 1) * SB;
            asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");  // this lane's copies from this strip, if any (every lane closes a group per chunk)
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 32; i++) {
              if constexpr (sizeof(OutT) == 4) {
                asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(buf + (uint32_t)(i * 32 + lane) * 4u), "r"(v[i]) : "memory");
              } else {
                const __nv_bfloat16 h = __float2bfloat16_rn(__uint_as_float(v[i]));
                asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(buf + (uint32_t)(i * 32 + lane) * 2u), "h"(*reinterpret_cast<const uint16_t *>(&h)) : "memory");
              }
            }
            if (!a.offsets) {
              fence_proxy_async();
              __syncwarp();
#pragma unroll
              for (int j = 0; j < 2; j++)  // (16 tokens each: a tile's last chunk may hold no more, and what follows is the next tile's)
                if (n0 < a.N && T.m0 + c0 + 16 * j < T.m_end && elect_one())
                  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(&maps.out), "r"(buf + j * (SB / 2)), "r"(n0),
                               "r"(T.m0 + c0 + 16 * j)
                               : "memory");
              asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
            } else {
              constexpr int LPT = 2 * (int)sizeof(OutT);  // lanes to a token, 16 bytes each
              const int seg16 = lane % LPT, n = n0 + seg16 * (32 / LPT);
              __syncwarp();
#pragma unroll
              for (int i = lane / LPT; i < 32; i += 32 / LPT) {
                const int m = __shfl_sync(0xffffffffu, prow, i);
                const uint4 q = lds128(buf + (uint32_t)(i * LPT + seg16) * 16u);
                if (m >= 0 && n < a.N) *reinterpret_cast<uint4 *>(out + (long long)m * a.N + n) = q;
              }
            }
          } else {
            OutT *o = out + n0 + lane;
#pragma unroll
            for (int i = 0; i < 32; i++) {
              const int m = __shfl_sync(0xffffffffu, prow, i);
              st_if(n0 + lane < a.N && m >= 0, o + (long long)m * a.N, __uint_as_float(v[i]));
            }
          }
        }
      }
      asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {  // copies still in flight get some time to land before the CTA retires
    __nanosleep(50000);
    if (threadIdx.x == 0) g_status = 1;
  }
  if constexpr (CG == 2) cluster_sync();  // nobody leaves while the peer may still signal its barriers
  if (warp == MMA_WARP) dealloc512<CG>(tmem);
}

// ------------------------------------------------------------------------------------ host
template <typename Row, typename OutT>
constexpr int fixed_smem(int E) { return EXPANDERS * Row::SLOT + STRIPS<OutT> + BAR_BYTES + (E + 1) * 12 + 16 + 1024; }

template <typename Row, bool BF16, typename OutT, int CG>
int run(const typename Row::Ctx &ctx, const TmemCall &c, Args a, int nt_max, cudaStream_t st) {
  if (nt_max < 16 * CG || nt_max % (16 * CG) || nt_max > MAX_ROWS * CG) return 0;  // (the tensor maps and the kernel's own rounding of tiles go by sixteens)
  a.nt_max = nt_max;
  const int rows = nt_max / CG;
  a.stage_bytes = rows * 256;
  a.nbs = (SMEM_MAX - fixed_smem<Row, OutT>(a.E)) / a.stage_bytes;
  if (a.nbs > NBS) a.nbs = NBS;
  if (a.nbs < 3) return 0;
  const int smem = a.nbs * a.stage_bytes + fixed_smem<Row, OutT>(a.E);
  if (smem > SMEM_MAX) return 0;
  int G = sm_count() / CG;
  if (G * CG > MAX_GRID) G = MAX_GRID / CG;
  if (!c.offsets) {
    const int ntt = (int)((c.M + nt_max - 1) / nt_max);
    const long long nb = c.K / KU, tiles = (long long)ntt * ((c.N + 128 * CG - 1) / (128 * CG)), least = c.min_run_k < KU ? 1 : c.min_run_k / KU;
    if (tiles * nb >= 1ll << 27) return 0;
    // Tiles shorter than two runs are whole ones while there is an SM for each.  Cut by their length alone those below one run went several to a CTA, and others
    // ended within a tile: 4-bit 3072 x 768, 16 rows 8.5 -> 5.0 us (token tiles 6.7), Q8_0 4096 x 256, 8 rows 6.8 -> 4.5, Q4_K 2048 x 1536, 100 rows 11.7 -> 8.8.
    const long long runs = tiles <= G && nb < 2 * least ? tiles : tiles * nb / least;
    if (runs < G) G = (int)(runs > 0 ? runs : 1);
  }
  if (c.parts_bytes < (size_t)G * CG * PART_FLOATS * 4) return 0;
  a.parts = (float *)c.parts, a.sync = (Sync *)c.sync;
  const EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(LB200_E_DEVICE, "light_b200: cuTensorMapEncodeTiled is not available from the driver");
  Maps tm = {};
  const cuuint64_t dims[2] = {(cuuint64_t)c.K, (cuuint64_t)c.M};
  const cuuint64_t strides[1] = {(cuuint64_t)c.K * 2};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = CUDA_SUCCESS;
  for (int i = c.offsets ? 16 : rows; i <= rows && r == CUDA_SUCCESS; i += 16) {  // (one matrix: all its tiles are alike)
    const cuuint32_t box[2] = {64, (cuuint32_t)i};
    r = enc(&tm.x[i / 16 - 1], BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(c.x16), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (!c.offsets && ((size_t)c.N * sizeof(OutT)) % 16 == 0 && ((uintptr_t)c.out & 15) == 0 && r == CUDA_SUCCESS) {  // (as the kernel has it: else plain stores)
    const cuuint64_t odims[2] = {(cuuint64_t)c.N, (cuuint64_t)c.M}, ostr[1] = {(cuuint64_t)c.N * sizeof(OutT)};
    const cuuint32_t obox[2] = {32, 16};
    r = enc(&tm.out, sizeof(OutT) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c.out, odims, ostr, obox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if constexpr (Row::BOXES > 0) {
    const cuuint64_t wdims[2] = {(cuuint64_t)Row::stride(c.K), (cuuint64_t)a.E * c.N}, wstr[1] = {wdims[0]};
    for (int i = 0; i < Row::BOXES && r == CUDA_SUCCESS; i++) {
      const cuuint32_t wbox[2] = {(cuuint32_t)Row::BOX[i].bytes, 32};
      const CUtensorMapSwizzle sw = swizzle_of(Row::BOX[i].swizzle);
      r = enc(&tm.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(Row::base(ctx)), wdims, wstr, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
  }
  if (r != CUDA_SUCCESS) return fail(LB200_E_SHAPE, "light_b200: cuTensorMapEncodeTiled failed (%d)", (int)r);
  auto kern = gemm_tmem_kernel<Row, BF16, OutT, CG>;
  static DeviceOnce attr;
  cudaError_t e = attr.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX); });
  if (e != cudaSuccess) return fail((int)e, "light_b200: gemm (tmem): %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(G * CG));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CG, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
  cfg.attrs = at, cfg.numAttrs = CG > 1 ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kern, tm, ctx, a, (OutT *)c.out);
  if (e != cudaSuccess) return fail((int)e, "light_b200: gemm (tmem): %s", cudaGetErrorString(e));
  if (int rc = launched("gemm (weights through tensor memory)")) return rc;
  return 1;
}

template <typename Row, bool BF16, typename OutT>
int pick(const typename Row::Ctx &ctx, const TmemCall &c, cudaStream_t st) {
  if (c.K % KU || c.E > MAX_E || (c.offsets && (c.M / 16 + c.E) * ((c.N + 127) / 128) * (c.K / KU) >= 1ll << 31)) return 0;
  Args a = {};
  a.offsets = c.offsets, a.pairs = c.pairs, a.topkw = c.topkw, a.factor = c.factor, a.modes = c.modes, a.mode = c.factor ? 0 : MODE_BF16, a.size_m = c.size_m;
  a.tokens = c.tokens, a.x16 = (uint4 *)const_cast<void *>(c.x16), a.topk = c.topk, a.row_per_pair = c.row_per_pair;
  a.E = c.offsets ? c.E : 1, a.M = (int)c.M, a.N = c.N, a.K = c.K;
  static const int k_cg = knob("LIGHT_B200_TMEM_CG", 0), k_nt = knob("LIGHT_B200_TMEM_NT", 0), k_wmin = knob("LIGHT_B200_TMEM_WMIN", 128), k_pair = knob("LIGHT_B200_TMEM_PAIR", 0);
  a.wmin = k_wmin < 16 ? 16 : k_wmin > 1024 ? 1024 : k_wmin;
  // The token tile: at most 256 (two SMs; less where the weight slots leave less room), all tiles of a matrix alike.  One SM
  // alone takes up to 128, with two accumulators.
  int rows = (SMEM_MAX - fixed_smem<Row, OutT>(a.E)) / (3 * 256) / 16 * 16;
  if (rows > 128) rows = 128;
  // Two SMs to a tile halve the token traffic and the number of times a weight is expanded, one SM has the shorter chain of
  // hand-overs.  Measured crossing: 32 units per SM (333 tokens, 4096 x 4096: 21.6 us alone, 22.9 in pairs; 4096 x 14336: 46
  // against 40); grouped, 64 tokens per expert on average (64 experts of 2048 x 2048, 64 tokens: 95 against 88 us).
  const bool big = c.offsets ? c.mean_tokens >= (k_pair ? k_pair : 64)
                             : c.M > 128 && (long long)((c.N + 127) / 128) * ((c.M + 127) / 128) * (c.K / KU) >= (k_pair ? k_pair : 32) * sm_count();
  const int cg = (k_cg ? k_cg >= 2 : big) ? 2 : 1;
  int cap = rows * cg;
  if (k_nt && k_nt < cap) cap = k_nt < 16 * cg ? 16 * cg : k_nt / (16 * cg) * (16 * cg);
  int nt = cap;
  if (!c.offsets) {
    const int ntt = (int)((c.M + cap - 1) / cap);
    nt = (int)((c.M + ntt - 1) / ntt + 16 * cg - 1) / (16 * cg) * (16 * cg);
  }
  if (cg == 2) return run<Row, BF16, OutT, 2>(ctx, c, a, nt, st);
  return run<Row, BF16, OutT, 1>(ctx, c, a, nt, st);
}

}  // namespace

size_t gemm_tmem_sync_bytes() { return (sizeof(Sync) + 1023) & ~(size_t)1023; }
size_t gemm_tmem_parts_bytes() { return (size_t)MAX_GRID * PART_FLOATS * 4; }

int gemm_tmem(const TmemCall &c, cudaStream_t st) {
  switch (c.kind) {
    case TmemCall::Q4K: return pick<TmQ4K, false, float>({(const uint8_t *)c.w}, c, st);
    case TmemCall::Q6K:
      if (TmQ6KT::fits(c.w, c.K)) return pick<TmQ6KT, false, float>({(const uint8_t *)c.w}, c, st);
      return pick<TmQ6K, false, float>({(const uint8_t *)c.w}, c, st);
    case TmemCall::Q80: return pick<TmQ80, false, float>({(const uint8_t *)c.w}, c, st);
    case TmemCall::INT4: {
      const TmInt4::Ctx x{(const uint32_t *)c.w, c.s, c.z, c.G, Div::of(c.G / 64)};
      if (c.out_bf16) return pick<TmInt4, false, __nv_bfloat16>(x, c, st);
      return c.bf16 ? pick<TmInt4, true, __nv_bfloat16>(x, c, st) : pick<TmInt4, false, float>(x, c, st);
    }
    case TmemCall::FP8: {
      if (c.factor && c.modes) {
        if (c.bR % 128 || c.bC % KU || c.N % c.bR) return 0;
        return pick<TmFp8H, false, __nv_bfloat16>({(const uint8_t *)c.w, c.s, c.bR, Div::of(c.bC / KU), c.K / c.bC}, c, st);
      }
      const TmFp8::Ctx x{(const uint8_t *)c.w, c.s, c.bR, c.bC, Div::of(c.bC / 64)};
      return c.bf16 ? pick<TmFp8, true, __nv_bfloat16>(x, c, st) : pick<TmFp8, false, float>(x, c, st);
    }
    case TmemCall::DENSE: return pick<TmDense, true, __nv_bfloat16>({(const uint16_t *)c.w}, c, st);
  }
  return 0;
}

int gemm_tmem_status() {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, g_status, sizeof(int));
  return e == cudaSuccess ? v : -(int)e;
}

}  // namespace lb
