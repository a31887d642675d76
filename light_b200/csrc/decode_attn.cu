// Decode-step attention against a fixed-capacity KV cache whose length lives on the device: the
// counterparts of the reference's ops.KVAppend, ops.DecodeAttention and ops.IncrementI64
// (ops/decode_attn.go:13-205, kernels/cuda/decode_attn.go:44-133, kernels/cuda/src/decode_attn.cu:1-161).
//
// The reference runs three launches per layer (append; split-K partials into a scratch tensor, one block
// per 32 keys of the CAPACITY; combine).  Here one launch does all of it: a thread-block cluster of up to
// eight CTAs serves one (batch, KV head); the cluster divides the VALID keys [start, n) evenly (n is read
// on the device), every warp walks its keys with an online softmax for all query heads of the group (one
// lane owns D / 32 consecutive dims, so a key or value row is one coalesced warp load), the warps' and
// then the CTAs' partial (max, sum, sum p v) meet in shared and distributed shared memory, and CTA r
// writes slice r of the output.  No scratch tensor, no atomics, the same launch at every position.  With
// k_new / v_new given, the new row is read from there by the warp that owns position `pos` and copied
// into the cache by rank 0, so the append needs no launch of its own.
#include "common.cuh"
#include "mma_sync.cuh"
#include "umma.cuh"

namespace lb {
namespace {

constexpr int DA_WARPS = 16, DA_THREADS = DA_WARPS * 32;
constexpr int DA_MAX_G = 16;  // query heads per KV head, the reference's limit (decode_attn.cu:11)

__device__ unsigned int g_attn_status = 0;  // bit 0: a position outside [0, Cap) was seen (and clamped)

struct AttnArgs {
  const void *q, *k_new, *v_new;
  void *kbuf, *vbuf, *out;
  const long long *pos;
  int B, NH, KH, Cap, window;
  float scale;
  double rope_k;  // 0: no rotation; else -2 log2(base) / D, so that base^(-2 i / D) = 2^(i rope_k)
};

// cos and sin of pos * base^(-2 i / D): the angle in f64 (an f32 angle of a few hundred radians is already
// off by 1e-5), reduced to [-pi, pi] there, then the f32 functions.  Out of line: its registers are not the
// attention loop's.
__device__ __noinline__ float2 rope_cos_sin(long long pos, int i, double rope_k) {
  const double theta = (double)pos * exp2((double)i * rope_k);
  const double r = theta - 6.283185307179586476925 * rint(theta * 0.15915494309189533577);
  float sn, c;
  sincosf((float)r, &sn, &c);
  return make_float2(c, sn);
}

// PER consecutive elements of a row, as floats; 2 to 64 bytes per lane, naturally aligned
template <int PER>
__device__ __forceinline__ void load_row(const float *p, float (&f)[PER]) {
  if constexpr (PER >= 4) {
#pragma unroll
    for (int i = 0; i < PER / 4; i++) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(p) + i);
      f[4 * i] = v.x, f[4 * i + 1] = v.y, f[4 * i + 2] = v.z, f[4 * i + 3] = v.w;
    }
  } else if constexpr (PER == 2) {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
    f[0] = v.x, f[1] = v.y;
  } else {
    f[0] = __ldg(p);
  }
}
template <int PER>
__device__ __forceinline__ void load_row(const __nv_bfloat16 *p, float (&f)[PER]) {
  if constexpr (PER >= 8) {
#pragma unroll
    for (int i = 0; i < PER / 8; i++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + i);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int c = 0; c < 4; c++) f[8 * i + 2 * c] = __uint_as_float(w[c] << 16), f[8 * i + 2 * c + 1] = __uint_as_float(w[c] & 0xFFFF0000u);
    }
  } else if constexpr (PER == 4) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
    f[0] = __uint_as_float(v.x << 16), f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16), f[3] = __uint_as_float(v.y & 0xFFFF0000u);
  } else if constexpr (PER == 2) {
    const uint32_t v = __ldg(reinterpret_cast<const uint32_t *>(p));
    f[0] = __uint_as_float(v << 16), f[1] = __uint_as_float(v & 0xFFFF0000u);
  } else {
    f[0] = __bfloat162float(*p);
  }
}

// The CTAs of a cluster: rank r writes elements r (g D) / KS .. of the group's output from all ranks' (max, sum, sum p v).  BASE2:
// the maxima are in units of log2 e.
template <typename T, bool BASE2>
__device__ __forceinline__ void cluster_combine(const AttnArgs &a, const float *cpart, int g, int D, int ROW, int KS, int rank, int b, int kh, int threads) {
  const int tot = g * D, e0 = tot * rank / KS, e1 = tot * (rank + 1) / KS;
  const uint32_t cbase = (uint32_t)__cvta_generic_to_shared(cpart);
  for (int idx = e0 + threadIdx.x; idx < e1; idx += threads) {
    const int h = idx / D, d = idx - h * D;
    const uint32_t ra = cbase + (uint32_t)(h * ROW) * 4u;
    float M = -INFINITY, L = 0.f, A = 0.f;
    if (KS > 1) {
      float mr[8], lr[8], ar[8];  // all remote loads at once
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const uint32_t peer = umma::map_to_rank(ra, (uint32_t)(r < KS ? r : 0));
        mr[r] = umma::ld_cluster_f32(peer), lr[r] = umma::ld_cluster_f32(peer + 4u), ar[r] = umma::ld_cluster_f32(peer + 8u + (uint32_t)d * 4u);
      }
#pragma unroll
      for (int r = 0; r < 8; r++)
        if (r < KS) M = fmaxf(M, mr[r]);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        if (r < KS && mr[r] > -INFINITY) {  // a rank without keys holds (-inf, 0, 0)
          const float e = BASE2 ? exp2f(mr[r] - M) : __expf(mr[r] - M);
          L = fmaf(e, lr[r], L), A = fmaf(e, ar[r], A);
        }
      }
    } else {
      L = cpart[h * ROW + 1], A = cpart[h * ROW + 2 + d];
    }
    st_act(static_cast<T *>(a.out), ((long long)b * a.NH + (long long)kh * g + h) * D + d, A / L);
  }
  if (KS > 1) umma::cluster_sync();  // nobody leaves while a peer still reads its partials
}

// The position: read before the wait as a hint and once more after it, so never from a line that the first read left in L1.
__device__ __forceinline__ long long load_pos(const long long *p) {
  long long v;
  asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}

template <int PER, int GH_>
struct AttnCfg {
  static constexpr int D = PER * 32;
  static constexpr int GH = GH_;                                        // query heads per pass over the keys
  static constexpr int U = PER >= 16 ? 1 : PER == 8 ? 2 : 4;           // keys per batch of a warp (two batches in flight)
  static constexpr int ROW = D + 2;                                     // max, sum, D dims
  static constexpr int WPART = DA_WARPS * GH * ROW;                     // floats: per-warp partials of a pass
  static size_t smem(int g) { return (size_t)(WPART + g * ROW) * sizeof(float); }
};

template <typename T, int PER, int GH_>
__global__ void __launch_bounds__(DA_THREADS, 1) decode_attn_kernel(AttnArgs a) {
  using Cfg = AttnCfg<PER, GH_>;
  constexpr int D = Cfg::D, GH = Cfg::GH, U = Cfg::U, ROW = Cfg::ROW;
  constexpr int NV = GH * U;  // dot products per batch of keys
  constexpr int SH = NV >= 32 ? 0 : NV == 16 ? 1 : NV == 8 ? 2 : NV == 4 ? 3 : NV == 2 ? 4 : 5;
  extern __shared__ __align__(16) float sm[];  // [warp][head of the pass][ROW] then [head][ROW] of this CTA
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.y, rank = blockIdx.y, bkh = blockIdx.x;
  const int g = a.NH / a.KH, b = bkh / a.KH, kh = bkh - b * a.KH;
  float *wpart = sm, *cpart = sm + Cfg::WPART;
  __shared__ float trig[D];  // cos, sin of the rotation's D / 2 angles
  {
    // The cached rows of this CTA on their way to L2 while the launch before still runs.  Only a hint: the position may be
    // one short here, and every row is read after the wait.
    const long long p = load_pos(a.pos);
    const int n = (int)(p < 0 ? 0 : p < a.Cap ? p + 1 : a.Cap), s0 = a.window > 0 ? max(0, n - a.window) : 0, ch = (n - s0 + KS - 1) / KS;
    const int f = s0 + rank * ch, e = min(n, f + ch);
    const char *kp = static_cast<const char *>(a.kbuf) + ((size_t)bkh * a.Cap + f) * D * sizeof(T), *vp = static_cast<const char *>(a.vbuf) + ((size_t)bkh * a.Cap + f) * D * sizeof(T);
    const int lines = min((e - f) * (int)(D * sizeof(T)) / 128, 4 * DA_THREADS);
    for (int i = threadIdx.x; i < lines; i += DA_THREADS)
      asm volatile("prefetch.global.L2 [%0];\n\tprefetch.global.L2 [%1];\n" ::"l"(kp + (size_t)i * 128), "l"(vp + (size_t)i * 128));
  }
  pdl_wait();  // q, k_new, v_new are the previous launch's output, and so may be pos
  long long pos = load_pos(a.pos);
  // A position outside the cache: reported, nothing is appended (as kv_append_kernel), and the launch attends
  // over the cached rows of the clamped range, so that append-inside stays equal to append-then-attend.
  const bool in_range = pos >= 0 && pos < a.Cap;
  if (!in_range) {
    if (threadIdx.x == 0) atomicOr(&g_attn_status, 1u);
    pos = pos < 0 ? 0 : a.Cap - 1;
  }
  const int n = (int)pos + 1;
  const int start = a.window > 0 ? max(0, n - a.window) : 0;
  const int chunk = (n - start + KS - 1) / KS;
  const int j0 = start + rank * chunk, j1 = min(n, j0 + chunk);
  const T *Kb = static_cast<const T *>(a.kbuf) + (size_t)bkh * a.Cap * D + lane * PER;
  const T *Vb = static_cast<const T *>(a.vbuf) + (size_t)bkh * a.Cap * D + lane * PER;
  const T *kn = a.k_new && in_range ? static_cast<const T *>(a.k_new) + (size_t)bkh * D + lane * PER : nullptr;
  const T *vn = a.k_new && in_range ? static_cast<const T *>(a.v_new) + (size_t)bkh * D + lane * PER : nullptr;
  // rotary embedding of q and of the new key at position pos (rotate-half pairing: dim i with i + D / 2,
  // which is lane ^ 16 here); cached keys were rotated when they were appended
  const bool roped = a.rope_k != 0.0;
  float rc[PER], rs[PER];
  if (roped) {  // each angle once per CTA (a chain of f64 operations): four in a row per lane took 2 us
    for (int i = threadIdx.x; i < D / 2; i += DA_THREADS) {
      const float2 cs = rope_cos_sin(pos, i, a.rope_k);
      trig[i] = cs.x, trig[D / 2 + i] = cs.y;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int i = (lane * PER + p) & (D / 2 - 1);
      rc[p] = trig[i], rs[p] = trig[D / 2 + i];
    }
  }
  auto rotate = [&](float (&v)[PER]) {
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const float o = __shfl_xor_sync(0xffffffffu, v[p], 16);
      v[p] = lane < 16 ? v[p] * rc[p] - o * rs[p] : o * rs[p] + v[p] * rc[p];
    }
  };
  if (kn && rank == 0 && threadIdx.x < D) {  // the append: readers of position pos take the row from k_new
    const T *ks = static_cast<const T *>(a.k_new) + (size_t)bkh * D;
    const size_t dst = ((size_t)bkh * a.Cap + (size_t)pos) * D + threadIdx.x;
    if (roped) {
      const int i = threadIdx.x & (D / 2 - 1);
      const float2 cs = make_float2(trig[i], trig[D / 2 + i]);
      const float x0 = ld_act(ks, i), x1 = ld_act(ks, i + D / 2);
      st_act(static_cast<T *>(a.kbuf), (long long)dst, (int)threadIdx.x < D / 2 ? x0 * cs.x - x1 * cs.y : x0 * cs.y + x1 * cs.x);
    } else {
      static_cast<T *>(a.kbuf)[dst] = ks[threadIdx.x];
    }
    static_cast<T *>(a.vbuf)[dst] = static_cast<const T *>(a.v_new)[(size_t)bkh * D + threadIdx.x];
  }

  for (int h0 = 0; h0 < g; h0 += GH) {
    const int gh = min(GH, g - h0);
    float qf[GH][PER], acc[GH][PER], m[GH], l[GH];
    float m_own = -INFINITY;  // m[head of the value this lane owns in the reduce-scatter]
#pragma unroll
    for (int h = 0; h < GH; h++) {
      m[h] = -INFINITY, l[h] = 0.f;
#pragma unroll
      for (int p = 0; p < PER; p++) acc[h][p] = 0.f, qf[h][p] = 0.f;
      if (h < gh) load_row<PER>(static_cast<const T *>(a.q) + ((size_t)b * a.NH + (size_t)kh * g + h0 + h) * D + lane * PER, qf[h]);
      if (roped) rotate(qf[h]);
    }
    float kf[U][PER], vf[U][PER];
    auto fetch = [&](int j, float (&kk)[U][PER], float (&vv)[U][PER]) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (j + u < j1) {
          const bool fresh = kn && j + u == (int)pos;
          load_row<PER>(fresh ? kn : Kb + (size_t)(j + u) * D, kk[u]);
          load_row<PER>(fresh ? vn : Vb + (size_t)(j + u) * D, vv[u]);
          if (fresh && roped) rotate(kk[u]);
        } else {
#pragma unroll
          for (int p = 0; p < PER; p++) kk[u][p] = 0.f, vv[u][p] = 0.f;
        }
      }
    };
    if (j0 + warp * U < j1) fetch(j0 + warp * U, kf, vf);
    for (int j = j0 + warp * U; j < j1; j += DA_WARPS * U) {
      float kx[U][PER], vx[U][PER];  // the next batch is requested before this one is used
      if (j + DA_WARPS * U < j1) fetch(j + DA_WARPS * U, kx, vx);
      if constexpr (NV <= 32) {
        // The GH x U dot products of this batch are summed over the lanes by a reduce-scatter: at every
        // step a lane hands half of its partial sums to its partner and keeps the other half, so that
        // value i (head i / U, key i % U) ends up, complete, in lanes [i << SH, (i + 1) << SH) -- NV + 1
        // shuffles instead of 5 NV -- and the exponentials are computed once, by the owners.
        float v[NV];
#pragma unroll
        for (int h = 0; h < GH; h++)
#pragma unroll
          for (int u = 0; u < U; u++) {
            float d = 0.f;
#pragma unroll
            for (int p = 0; p < PER; p++) d = fmaf(qf[h][p], kf[u][p], d);
            v[h * U + u] = d;
          }
        int cnt = NV;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
          if (cnt > 1) {
            const int half = cnt / 2;
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < half; i++) {
              const float send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
              v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
            cnt = half;
          } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
          }
        }
        const int own = lane >> SH;  // this lane's value: head own / U, key own % U
        const float s_own = j + (own % U) < j1 ? v[0] * a.scale : -INFINITY;
        float bm = s_own;            // maximum over the batch's keys of the own head
#pragma unroll
        for (int off = 1 << SH; off < (U << SH); off <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, off));
        m_own = fmaxf(m_own, bm);
        const float e_own = __expf(s_own - m_own);  // -inf for a missing key: 0
#pragma unroll
        for (int h = 0; h < GH; h++) {
          const float mx = fmaxf(m[h], __shfl_sync(0xffffffffu, bm, (h * U) << SH));
          const float corr = __expf(m[h] - mx);  // m = -inf on the first batch: 0
          m[h] = mx;
          l[h] *= corr;
#pragma unroll
          for (int p = 0; p < PER; p++) acc[h][p] *= corr;
#pragma unroll
          for (int u = 0; u < U; u++) {
            const float e = __shfl_sync(0xffffffffu, e_own, (h * U + u) << SH);
            l[h] += e;
#pragma unroll
            for (int p = 0; p < PER; p++) acc[h][p] = fmaf(e, vf[u][p], acc[h][p]);
          }
        }
      } else {
#pragma unroll
        for (int h = 0; h < GH; h++) {
          if (h < gh) {
            float s[U], mx = m[h];
  #pragma unroll
            for (int u = 0; u < U; u++) {
              float d = 0.f;
  #pragma unroll
              for (int p = 0; p < PER; p++) d = fmaf(qf[h][p], kf[u][p], d);
              s[u] = j + u < j1 ? warp_sum(d) * a.scale : -INFINITY;
              mx = fmaxf(mx, s[u]);
            }
            const float corr = __expf(m[h] - mx);  // m = -inf on the first batch: 0
            m[h] = mx;
            l[h] *= corr;
  #pragma unroll
            for (int p = 0; p < PER; p++) acc[h][p] *= corr;
  #pragma unroll
            for (int u = 0; u < U; u++) {
              const float e = __expf(s[u] - mx);  // -inf for a missing key: 0
              l[h] += e;
  #pragma unroll
              for (int p = 0; p < PER; p++) acc[h][p] = fmaf(e, vf[u][p], acc[h][p]);
            }
          }
        }
      }
      if (j + DA_WARPS * U < j1) {
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int p = 0; p < PER; p++) kf[u][p] = kx[u][p], vf[u][p] = vx[u][p];
      }
    }
    // ---- the warps of this CTA
#pragma unroll
    for (int h = 0; h < GH; h++) {
      if (h < gh) {
        float *row = wpart + (warp * GH + h) * ROW;
        if (lane == 0) row[0] = m[h], row[1] = l[h];
#pragma unroll
        for (int p = 0; p < PER; p++) row[2 + lane * PER + p] = acc[h][p];
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < gh * D; idx += DA_THREADS) {
      const int h = idx / D, d = idx - h * D;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < DA_WARPS; w++) M = fmaxf(M, wpart[(w * GH + h) * ROW]);
      float L = 0.f, A = 0.f;
      if (M > -INFINITY) {
#pragma unroll
        for (int w = 0; w < DA_WARPS; w++) {
          const float *row = wpart + (w * GH + h) * ROW;
          const float e = __expf(row[0] - M);
          L = fmaf(e, row[1], L), A = fmaf(e, row[2 + d], A);
        }
      }
      float *dst = cpart + (h0 + h) * ROW;
      dst[2 + d] = A;
      if (d == 0) dst[0] = M, dst[1] = L;
    }
    __syncthreads();
  }
  if (KS > 1) umma::cluster_sync();
  cluster_combine<T, false>(a, cpart, g, D, ROW, KS, rank, b, kh, DA_THREADS);
}

// ------------------------------------------------------------------------------------ f32 caches, heads of 64 or 128
// One lane per 1/32 of a row (the first kernel) spends 17 shuffles and 25 exponentials' worth of latency on four keys: 6 us of a 12.4 us
// launch for 1024 positions, and a third of the memory rate on long caches.  Here the keys come in tiles of 64 through shared memory
// (16-byte asynchronous copies, a ring of S tiles: the bytes in flight; one bulk copy per padded row took 2.8 us a tile), and a lane owns a KEY: a quarter of its dot products with all the group's heads
// (K rows are padded by 16 bytes, so 32 keys lie on 32 banks; the queries are broadcasts), one warp per head then turns the tile's
// scores into weights, and a lane owns D / 32 dims of the values, a warp eight keys.  Three CTA barriers a tile, no shuffle per key.
//   * What depends on the position alone (angles, L2 hints) runs before the wait, the first tiles, the queries and the position itself
//     are requested together after it; the position may have moved by then, and everything is planned again if it has.
//   * The new key and value are written into the last tile in shared memory, where the cache's row would have landed: the same bits.
// About 14 shared-memory cycles per key of 128 f32 dims and four heads against 40 that its bytes take from HBM: 8 sequences of 8192
// keys, 8 KV heads of 128 under 32 heads 196 -> 108 us (5.0 TB/s); one of 1024 keys, where the chain of latencies is all, 16.0 -> 7.5 us.
constexpr int FT_WARPS = 8, FT_THREADS = FT_WARPS * 32, FT_KEYS = 64;

template <int D, int GH>
struct F32Cfg {
  static constexpr int S = GH == 16 || (D == 64 && GH == 8) ? 2 : 3;  // tiles in the ring: what 227 KB (two CTAs of D = 64) hold beside the scores
  static constexpr int KP = D * 4 + 16, KB = FT_KEYS * KP, STAGE = KB + FT_KEYS * D * 4, ROW = D + 2;
  static constexpr int QS = S * STAGE, PART = QS + GH * D * 4, PS = PART + 4 * GH * FT_KEYS * 4, CP = PS + FT_KEYS * GH * 4, MISC = CP + GH * ROW * 4;
  // MISC: max, sum, correction [GH] each | angles [D]
  static constexpr int TRIG = MISC + 3 * GH * 4, SMEM = TRIG + D * 4;
};

template <int D, int GH>
__global__ void __launch_bounds__(FT_THREADS, D == 64 ? 2 : 1) decode_attn_f32_kernel(AttnArgs a) {
  using C = F32Cfg<D, GH>;
  constexpr int S = C::S, DQ = D / 4, PV = D / 32, HW = (GH + FT_WARPS - 1) / FT_WARPS;
  constexpr int QP = (GH * D / 2 + FT_THREADS - 1) / FT_THREADS;  // (q[i], q[i + D / 2]) pairs per thread
  extern __shared__ __align__(128) unsigned char fsm[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int KS = gridDim.y, rank = blockIdx.y, bkh = blockIdx.x, g = a.NH / a.KH, b = bkh / a.KH, kh = bkh - b * a.KH;
  const uint32_t base = umma::smem_u32(fsm);
  float *qs = reinterpret_cast<float *>(fsm + C::QS), *part = reinterpret_cast<float *>(fsm + C::PART), *ps = reinterpret_cast<float *>(fsm + C::PS);
  float *cpart = reinterpret_cast<float *>(fsm + C::CP), *ms = reinterpret_cast<float *>(fsm + C::MISC), *ls = ms + GH, *cs = ls + GH;
  float *trig = reinterpret_cast<float *>(fsm + C::TRIG);
  const float *kc = static_cast<const float *>(a.kbuf) + (size_t)bkh * a.Cap * D, *vc = static_cast<const float *>(a.vbuf) + (size_t)bkh * a.Cap * D;
  const bool roped = a.rope_k != 0.0;

  int pos, j0, n;  // this CTA's keys: j0 .. j0 + n
  bool in_range, fresh;  // fresh: the last of them is the new one, which the cache does not hold yet
  auto plan = [&](long long p) {
    // a position outside the cache: nothing is appended (as kv_append_kernel), and the launch attends over the clamped range
    in_range = p >= 0 && p < a.Cap;
    pos = (int)(p < 0 ? 0ll : p < a.Cap ? p : (long long)a.Cap - 1);
    const int start = a.window > 0 ? max(0, pos + 1 - a.window) : 0, end = pos + 1, ch = (end - start + KS - 1) / KS;
    j0 = start + rank * ch, n = max(0, min(end, j0 + ch) - j0);
    fresh = a.k_new && in_range && n > 0 && j0 + n == end;
  };
  auto angles = [&]() {
    for (int i = tid; i < D / 2; i += FT_THREADS) {
      const float2 v = rope_cos_sin(pos, i, a.rope_k);
      trig[i] = v.x, trig[D / 2 + i] = v.y;
    }
  };
  const long long seen = load_pos(a.pos);
  plan(seen);
  {
    const char *kp = reinterpret_cast<const char *>(kc + (size_t)j0 * D), *vp = reinterpret_cast<const char *>(vc + (size_t)j0 * D);
    const int lines = min(n * (D * 4 / 128), 8 * FT_THREADS);
    for (int i = tid; i < lines; i += FT_THREADS)
      asm volatile("prefetch.global.L2 [%0];\n\tprefetch.global.L2 [%1];\n" ::"l"(kp + (size_t)i * 128), "l"(vp + (size_t)i * 128));
  }
  if (roped) angles();
  __syncthreads();
  pdl_wait();  // q, k_new, v_new are the previous launch's output; so may be the cache's last rows and the position
  auto issue = [&](int t) {  // tile t into slot t % S: always one commit group
    const int cnt = min(FT_KEYS, n - (fresh ? 1 : 0) - t * FT_KEYS);  // 0 for a tile of the new key alone
    const uint32_t dst = base + (t % S) * C::STAGE;
    const size_t row = (size_t)(j0 + t * FT_KEYS) * D;
    constexpr int PIECES = D / 4;  // of 16 bytes per row
    for (int i = tid; i < cnt * PIECES; i += FT_THREADS) {
      const int r = i / PIECES, c = i % PIECES;
      cp_async16(dst + r * C::KP + c * 16, kc + row + (size_t)i * 4);
      cp_async16(dst + C::KB + i * 16, vc + row + (size_t)i * 4);
    }
    cp_async_commit();
  };
  auto fill = [&]() {
#pragma unroll 1
    for (int t = 0; t < S - 1; t++) issue(t);
  };
  fill();
  const long long now = load_pos(a.pos);
  float2 qv[QP], kv = make_float2(0.f, 0.f), vv = kv;
#pragma unroll
  for (int i = 0; i < QP; i++) {
    const int idx = tid + i * FT_THREADS, h = idx / (D / 2), d = idx % (D / 2);
    const float *q = static_cast<const float *>(a.q) + ((size_t)b * a.NH + (size_t)kh * g + h) * D + d;
    qv[i] = h < g ? make_float2(q[0], q[D / 2]) : make_float2(0.f, 0.f);
  }
  if (a.k_new && tid < D / 2) {
    const float *k = static_cast<const float *>(a.k_new) + (size_t)bkh * D + tid, *v = static_cast<const float *>(a.v_new) + (size_t)bkh * D + tid;
    kv = make_float2(k[0], k[D / 2]), vv = make_float2(v[0], v[D / 2]);
  }
  if (now != seen) {  // the position moved while the launch before ran (the same in every thread)
    cp_async_wait<0>();
    __syncthreads();
    plan(now);
    if (roped) angles();
    __syncthreads();
    fill();
  }
  auto rot = [&](float2 v, int d) { return roped ? make_float2(v.x * trig[d] - v.y * trig[D / 2 + d], v.x * trig[D / 2 + d] + v.y * trig[d]) : v; };
#pragma unroll
  for (int i = 0; i < QP; i++) {
    const int idx = tid + i * FT_THREADS, h = idx / (D / 2), d = idx % (D / 2);
    if (h < GH) {
      const float2 v = rot(qv[i], d);
      qs[h * D + d] = v.x, qs[h * D + d + D / 2] = v.y;
    }
  }
  if (tid < D / 2) kv = rot(kv, tid);
  __syncthreads();

  float acc[GH][PV], m[HW], l[HW];  // m, l: of heads warp, warp + 8
#pragma unroll
  for (int h = 0; h < GH; h++)
#pragma unroll
    for (int i = 0; i < PV; i++) acc[h][i] = 0.f;
#pragma unroll
  for (int i = 0; i < HW; i++) m[i] = -INFINITY, l[i] = 0.f;
  const int tiles = (n + FT_KEYS - 1) / FT_KEYS, qd = warp >> 1, key = (warp & 1) * 32 + lane;
  for (int t = 0; t < tiles; t++) {
    const int cnt = min(FT_KEYS, n - t * FT_KEYS);
    unsigned char *kt = fsm + (t % S) * C::STAGE, *vt = kt + C::KB;
    if (fresh && t == tiles - 1) {  // the slot is free, and no copy touches this row
      if (tid < D / 2) {
        float *k = reinterpret_cast<float *>(kt + (cnt - 1) * C::KP) + tid, *v = reinterpret_cast<float *>(vt + (cnt - 1) * (D * 4)) + tid;
        k[0] = kv.x, k[D / 2] = kv.y, v[0] = vv.x, v[D / 2] = vv.y;
      }
    }
    cp_async_wait<S - 2>();
    __syncthreads();     // the tile is in place, and every warp is done with the one before it
    issue(t + S - 1);    // into that one's slot
    if (key < cnt || (warp & 1) * 32 < cnt) {  // a quarter of a key's products with every head (rows past cnt hold what they held)
      float d[GH];
#pragma unroll
      for (int h = 0; h < GH; h++) d[h] = 0.f;
#pragma unroll
      for (int i = 0; i < DQ / 4; i++) {
        const float4 k = *reinterpret_cast<const float4 *>(kt + key * C::KP + (qd * DQ + 4 * i) * 4);
#pragma unroll
        for (int h = 0; h < GH; h++) {
          const float4 q = *reinterpret_cast<const float4 *>(qs + h * D + qd * DQ + 4 * i);
          d[h] = fmaf(q.x, k.x, fmaf(q.y, k.y, fmaf(q.z, k.z, fmaf(q.w, k.w, d[h]))));
        }
      }
#pragma unroll
      for (int h = 0; h < GH; h++) part[(qd * GH + h) * FT_KEYS + key] = d[h];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < HW; i++) {
      const int h = warp + FT_WARPS * i;
      if (h < GH) {
        float v[2], mx = m[i];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const float *p = part + h * FT_KEYS + lane + 32 * u;
          v[u] = lane + 32 * u < cnt ? ((p[0] + p[GH * FT_KEYS]) + (p[2 * GH * FT_KEYS] + p[3 * GH * FT_KEYS])) * a.scale : -INFINITY;
          mx = fmaxf(mx, v[u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float corr = __expf(m[i] - mx), e0 = __expf(v[0] - mx), e1 = __expf(v[1] - mx);  // m = -inf at first: 0
        m[i] = mx;
        l[i] = fmaf(l[i], corr, e0 + e1);  // each lane its own keys' part
        ps[lane * GH + h] = e0, ps[(lane + 32) * GH + h] = e1;
        if (lane == 0) cs[h] = corr;
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < GH; h++) {
      const float c = cs[h];
#pragma unroll
      for (int i = 0; i < PV; i++) acc[h][i] *= c;
    }
    auto add = [&](int k) {
      float v[PV];
      if constexpr (PV == 4) {
        const float4 x = *reinterpret_cast<const float4 *>(vt + k * (D * 4) + lane * 16);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
      } else {
        const float2 x = *reinterpret_cast<const float2 *>(vt + k * (D * 4) + lane * 8);
        v[0] = x.x, v[1] = x.y;
      }
      float p[GH];
      if constexpr (GH >= 4) {
#pragma unroll
        for (int h = 0; h < GH; h += 4) {
          const float4 x = *reinterpret_cast<const float4 *>(ps + k * GH + h);
          p[h] = x.x, p[h + 1] = x.y, p[h + 2] = x.z, p[h + 3] = x.w;
        }
      } else {
#pragma unroll
        for (int h = 0; h < GH; h++) p[h] = ps[k * GH + h];
      }
#pragma unroll
      for (int h = 0; h < GH; h++)
#pragma unroll
        for (int i = 0; i < PV; i++) acc[h][i] = fmaf(p[h], v[i], acc[h][i]);
    };
    if (warp * 8 + 8 <= cnt) {
#pragma unroll
      for (int k = 0; k < 8; k++) add(warp * 8 + k);
    } else {
      for (int k = warp * 8; k < cnt; k++) add(k);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---- the warps' values over the (drained) ring, the heads' maxima and sums
  float *wpart = reinterpret_cast<float *>(fsm);
#pragma unroll
  for (int h = 0; h < GH; h++)
#pragma unroll
    for (int i = 0; i < PV; i++) wpart[(warp * GH + h) * D + lane * PV + i] = acc[h][i];
#pragma unroll
  for (int i = 0; i < HW; i++) {
    const float sum = warp_sum(l[i]);
    if (lane == 0 && warp + FT_WARPS * i < GH) ms[warp + FT_WARPS * i] = m[i], ls[warp + FT_WARPS * i] = sum;
  }
  __syncthreads();
  for (int idx = tid; idx < g * D; idx += FT_THREADS) {
    const int h = idx / D, d = idx - h * D;
    float A = 0.f;
#pragma unroll
    for (int w = 0; w < FT_WARPS; w++) A += wpart[(w * GH + h) * D + d];
    cpart[h * C::ROW + 2 + d] = A;
    if (d == 0) cpart[h * C::ROW] = ms[h], cpart[h * C::ROW + 1] = ls[h];
  }
  if (fresh && tid < D / 2) {  // the append: nothing of this launch reads the row from the cache
    const size_t dst = ((size_t)bkh * a.Cap + (size_t)pos) * D + tid;
    float *k = static_cast<float *>(a.kbuf) + dst, *v = static_cast<float *>(a.vbuf) + dst;
    k[0] = kv.x, k[D / 2] = kv.y, v[0] = vv.x, v[D / 2] = vv.y;
  }
  if (tid == 0 && !in_range) atomicOr(&g_attn_status, 1u);
  __syncthreads();
  if (KS > 1) umma::cluster_sync();
  cluster_combine<float, false>(a, cpart, g, D, C::ROW, KS, rank, b, kh, FT_THREADS);
}

// ------------------------------------------------------------------------------------ bf16 caches on the tensor cores
// The kernel above spends about 60 instructions of a warp per key (unpacking, 2 D FMAs per head and key over 32 lanes, the
// reduce-scatter), which bounds a bf16 cache at 1.2 TB/s (8 sequences, 8192 keys, 8 KV heads of 128: 231 us).  Here a warp takes
// 16 keys at a time through mma.sync (bf16 x bf16 -> f32), straight from global memory to fragments, about 13 instructions
// per key, and what remains is the memory.
//   * S = Q K^T: the query heads are the rows.  Rotated q is f32 and is split into bf16 hi + lo: up to eight heads, rows 0-7
//     hold hi and rows 8-15 lo of the same heads and one MMA does both; up to sixteen, two MMAs.  Relative error 2^-17.
//   * O += P V the same way: p split into hi + lo; the S fragment of a lane IS its P fragment (no exchange).
//   * The order of the dims inside a contraction is free as long as both sides agree, so a lane's K fragments are 32
//     consecutive bytes of its key (one 256-bit load feeds two MMAs), and the assignment of dims to V's columns gives a lane
//     32 consecutive bytes of each of its four keys; pairs of keys are interleaved by PRMT.
//   * Loads for the next 16 keys are issued as soon as the registers are free: K behind the QK MMAs, V behind the PV MMAs.
// Four warps to a CTA, two or three CTAs per SM, a cluster of up to eight CTAs along the keys.
constexpr int MA_WARPS = 4, MA_THREADS = MA_WARPS * 32;
constexpr int mma_ctas(int D) { return D == 64 ? 3 : 2; }  // CTAs per SM: what the registers allow

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack_rest(float a, float b, uint32_t hi) {  // what rounding to bf16 left, as bf16
  return pack_bf16(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u));
}
// W words (8 or 4) of a cached row: read once, so no room in L1
template <int W>
__device__ __forceinline__ void ld_stream(const void *p, uint32_t (&v)[W]) {
  if constexpr (W == 8)
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
  else
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
}

// One head's partial result of a warp, the 16 keys from j0 on and every MA_WARPS-th 16 after them, in f32 from end to end, into `row`
// (max in units of log2 e, sum, sum p v).  For caches that hold infinities: the hi and lo parts of a split operand multiply those to
// infinities of either sign, or to NaN, where the product itself is an infinity, or a score of -inf whose key counts for nothing.
template <int D>
__device__ __noinline__ void attend_plain(const __nv_bfloat16 *q, const __nv_bfloat16 *K, const __nv_bfloat16 *V, const __nv_bfloat16 *fresh, int pos_new,
                                          const float *trig, float sc, int j0, int j1, float *row) {
  constexpr int P = D / 32;
  const int lane = threadIdx.x & 31;
  float qf[P], acc[P], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < P; i++) {
    const int d = lane * P + i, e = d & (D / 2 - 1);
    const float x0 = __bfloat162float(q[e]), x1 = __bfloat162float(q[e + D / 2]);
    const float cs = trig ? trig[e] : 1.f, sn = trig ? trig[D / 2 + e] : 0.f;
    qf[i] = !trig ? __bfloat162float(q[d]) : d < D / 2 ? x0 * cs - x1 * sn : x0 * sn + x1 * cs, acc[i] = 0.f;
  }
  for (int i0 = 0, j = j0; j < j1; j = ++i0 % 16 ? j + 1 : j + 1 + 16 * (MA_WARPS - 1)) {
    const __nv_bfloat16 *k = j == pos_new ? fresh : K + (size_t)j * D, *v = j == pos_new ? fresh + D : V + (size_t)j * D;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < P; i++) s = fmaf(qf[i], __bfloat162float(k[lane * P + i]), s);
    s = warp_sum(s) * sc;
    if (s == -INFINITY) continue;
    const float mx = fmaxf(m, s), corr = exp2f(m - mx), e = exp2f(s - mx);
    m = mx, l = fmaf(l, corr, e);
#pragma unroll
    for (int i = 0; i < P; i++) acc[i] = fmaf(e, __bfloat162float(v[lane * P + i]), acc[i] * corr);
  }
  if (lane == 0) row[0] = m, row[1] = l;
#pragma unroll
  for (int i = 0; i < P; i++) row[2 + lane * P + i] = acc[i];
}

template <int D, bool G16>
__global__ void __launch_bounds__(MA_THREADS, mma_ctas(D)) decode_attn_mma_kernel(AttnArgs a) {
  constexpr int KL = D / 64;        // 32-byte loads of a key row per lane; each feeds two 16-dim steps
  constexpr int NT = D / 8;         // column tiles of O, and consecutive dims of a V row per lane
  constexpr int VW = NT / 2;        // words of a V row per lane
  constexpr int HMAX = G16 ? 16 : 8, ROW = D + 2;
  extern __shared__ __align__(16) float sm[];
  float *qs = sm;                                    // [HMAX][D] rotated q; later the warps' partial results [warp][HMAX][ROW]
  float *cpart = sm + MA_WARPS * HMAX * ROW;         // [HMAX][ROW] of this CTA
  float *trig = cpart + HMAX * ROW;                  // cos, sin of D / 2 angles
  uint32_t *fresh = reinterpret_cast<uint32_t *>(trig + D);  // the new key and value, bf16
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const int KS = gridDim.y, rank = blockIdx.y, bkh = blockIdx.x;
  const int g = a.NH / a.KH, b = bkh / a.KH, kh = bkh - b * a.KH;
  pdl_wait();
  long long pos = load_pos(a.pos);
  const bool in_range = pos >= 0 && pos < a.Cap;
  if (!in_range) {
    if (threadIdx.x == 0) atomicOr(&g_attn_status, 1u);
    pos = pos < 0 ? 0 : a.Cap - 1;
  }
  const int n = (int)pos + 1, start = a.window > 0 ? max(0, n - a.window) : 0;
  const int chunk = ((n - start + KS - 1) / KS + 15) & ~15;
  const int j0 = min(n, start + rank * chunk), j1 = min(n, j0 + chunk);
  const bool append = a.k_new && in_range;
  const __nv_bfloat16 *Kb = static_cast<const __nv_bfloat16 *>(a.kbuf) + (size_t)bkh * a.Cap * D;
  const __nv_bfloat16 *Vb = static_cast<const __nv_bfloat16 *>(a.vbuf) + (size_t)bkh * a.Cap * D;

  // ---- this warp's first keys are on their way while the query is prepared
  uint32_t kf[2][KL][8], vf[4][VW];
  auto fetch_k = [&](int j) {
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const __nv_bfloat16 *p = Kb + (size_t)min(j + 8 * t + r, n - 1) * D + c * 16;
#pragma unroll
      for (int i = 0; i < KL; i++) ld_stream<8>(p + 64 * i, kf[t][i]);
    }
  };
  auto fetch_v = [&](int j) {
#pragma unroll
    for (int k = 0; k < 4; k++) ld_stream<VW>(Vb + (size_t)min(j + 2 * c + (k & 1) + 8 * (k >> 1), n - 1) * D + r * NT, vf[k]);
  };
  int j = j0 + warp * 16;
  if (j < j1) fetch_k(j), fetch_v(j);

  const bool roped = a.rope_k != 0.0;
  if (roped) {
    for (int i = threadIdx.x; i < D / 2; i += MA_THREADS) {
      const float2 cs = rope_cos_sin(pos, i, a.rope_k);
      trig[i] = cs.x, trig[D / 2 + i] = cs.y;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < g * (D / 2); i += MA_THREADS) {
    const int h = i / (D / 2), d = i - h * (D / 2);
    const __nv_bfloat16 *q = static_cast<const __nv_bfloat16 *>(a.q) + ((size_t)b * a.NH + (size_t)kh * g + h) * D;
    const float x0 = __bfloat162float(q[d]), x1 = __bfloat162float(q[d + D / 2]);
    const float cs = roped ? trig[d] : 1.f, sn = roped ? trig[D / 2 + d] : 0.f;
    qs[h * D + d] = x0 * cs - x1 * sn, qs[h * D + d + D / 2] = x0 * sn + x1 * cs;
  }
  if (append && threadIdx.x < D / 2) {  // the new row: the cache gets it from rank 0, this CTA reads it from shared memory
    const __nv_bfloat16 *kn = static_cast<const __nv_bfloat16 *>(a.k_new) + (size_t)bkh * D, *vn = static_cast<const __nv_bfloat16 *>(a.v_new) + (size_t)bkh * D;
    const int d = threadIdx.x;
    const float x0 = __bfloat162float(kn[d]), x1 = __bfloat162float(kn[d + D / 2]), cs = roped ? trig[d] : 1.f, sn = roped ? trig[D / 2 + d] : 0.f;
    __nv_bfloat16 *fk = reinterpret_cast<__nv_bfloat16 *>(fresh), *fv = fk + D;
    fk[d] = roped ? __float2bfloat16_rn(x0 * cs - x1 * sn) : kn[d], fk[d + D / 2] = roped ? __float2bfloat16_rn(x0 * sn + x1 * cs) : kn[d + D / 2];
    fv[d] = vn[d], fv[d + D / 2] = vn[d + D / 2];
    if (rank == 0) {
      const size_t dst = ((size_t)bkh * a.Cap + (size_t)pos) * D + d;
      static_cast<__nv_bfloat16 *>(a.kbuf)[dst] = fk[d], static_cast<__nv_bfloat16 *>(a.kbuf)[dst + D / 2] = fk[d + D / 2];
      static_cast<__nv_bfloat16 *>(a.vbuf)[dst] = fv[d], static_cast<__nv_bfloat16 *>(a.vbuf)[dst + D / 2] = fv[d + D / 2];
    }
  }
  __syncthreads();

  // ---- Q fragments: step s covers, for column c, dims 64 (s / 4) + 16 c + 4 (s % 4) .. + 3 of every key (its two registers)
  uint32_t qh[D / 16][2], ql[D / 16][2], qh8[G16 ? D / 16 : 1][2], ql8[G16 ? D / 16 : 1][2];
#pragma unroll
  for (int s = 0; s < D / 16; s++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int d = 64 * (s >> 2) + 16 * c + 4 * (s & 3) + 2 * e;
      const float x0 = r < g ? qs[r * D + d] : 0.f, x1 = r < g ? qs[r * D + d + 1] : 0.f;
      qh[s][e] = pack_bf16(x0, x1), ql[s][e] = pack_rest(x0, x1, qh[s][e]);
      if constexpr (G16) {
        const float y0 = r + 8 < g ? qs[(r + 8) * D + d] : 0.f, y1 = r + 8 < g ? qs[(r + 8) * D + d + 1] : 0.f;
        qh8[s][e] = pack_bf16(y0, y1), ql8[s][e] = pack_rest(y0, y1, qh8[s][e]);
      }
    }
  __syncthreads();  // qs is reused for the partial results

  const float sc = a.scale * 1.4426950408889634f;  // scores in units of log2 e
  float m[G16 ? 2 : 1], l[G16 ? 2 : 1], o[NT][4];
#pragma unroll
  for (int i = 0; i < (G16 ? 2 : 1); i++) m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[t][e] = 0.f;

  for (; j < j1; j += MA_WARPS * 16) {
    if (append && j <= (int)pos && (int)pos < j + 16) {  // (pos is the last key: these loads cannot have its new row)
      const int x = (int)pos - j;
#pragma unroll
      for (int t = 0; t < 2; t++)
        if (x == 8 * t + r) {
#pragma unroll
          for (int i = 0; i < KL; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) kf[t][i][e] = fresh[32 * i + 8 * c + e];
        }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int y = 2 * c + (k & 1) + 8 * (k >> 1);
        if (y >= x) {  // (rows past it were read from its place, which holds anything: their weight is 0, so they must be finite)
#pragma unroll
          for (int e = 0; e < VW; e++) vf[k][e] = y == x ? fresh[D / 2 + VW * r + e] : 0u;
        }
      }
    }
    float s[2][4] = {};
#pragma unroll
    for (int st = 0; st < D / 16; st++)
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const uint32_t b0 = kf[t][st >> 2][2 * (st & 3)], b1 = kf[t][st >> 2][2 * (st & 3) + 1];
        if constexpr (G16) {
          mma_bf16(s[t], qh[st][0], qh8[st][0], qh[st][1], qh8[st][1], b0, b1);
          mma_bf16(s[t], ql[st][0], ql8[st][0], ql[st][1], ql8[st][1], b0, b1);
        } else {
          mma_bf16(s[t], qh[st][0], ql[st][0], qh[st][1], ql[st][1], b0, b1);
        }
      }
    const int jn = j + MA_WARPS * 16;
    if (jn < j1) fetch_k(jn);
    uint32_t ph[2][2], pl[2][2];  // [tile][row half]: P as A fragments
    float mx[G16 ? 2 : 1];
#pragma unroll
    for (int i = 0; i < (G16 ? 2 : 1); i++) {
      float v[4];
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const float x = G16 ? s[t][2 * i + e] : s[t][e] + s[t][2 + e];
          v[2 * t + e] = j + 8 * t + 2 * c + e < j1 ? x * sc : -INFINITY;
        }
      mx[i] = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(m[i], fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2)));
      float p[4];
#pragma unroll
      for (int e = 0; e < 4; e++) p[e] = exp2f(v[e] - mx[i]);  // (a block holds a key: mx is finite)
      const float corr = exp2f(m[i] - mx[i]);
      l[i] = l[i] * corr + ((p[0] + p[1]) + (p[2] + p[3]));
#pragma unroll
      for (int t = 0; t < 2; t++) ph[t][i] = pack_bf16(p[2 * t], p[2 * t + 1]), pl[t][i] = pack_rest(p[2 * t], p[2 * t + 1], ph[t][i]);
    }
    bool same = mx[0] == m[0];
    if constexpr (G16) same = same && mx[1] == m[1];
    if (!__all_sync(0xffffffffu, same)) {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const float c0 = exp2f(m[0] - mx[0]), c1 = G16 ? exp2f(m[G16 ? 1 : 0] - mx[G16 ? 1 : 0]) : c0;
        o[t][0] *= c0, o[t][1] *= c0, o[t][2] *= c1, o[t][3] *= c1;
      }
    }
#pragma unroll
    for (int i = 0; i < (G16 ? 2 : 1); i++) m[i] = mx[i];
#pragma unroll
    for (int t = 0; t < NT; t++) {  // column r of tile t is dim NT r + t
      const uint32_t sel = t & 1 ? 0x7632u : 0x5410u;
      const uint32_t b0 = __byte_perm(vf[0][t >> 1], vf[1][t >> 1], sel), b1 = __byte_perm(vf[2][t >> 1], vf[3][t >> 1], sel);
      if constexpr (G16) {
        mma_bf16(o[t], ph[0][0], ph[0][1], ph[1][0], ph[1][1], b0, b1);
        mma_bf16(o[t], pl[0][0], pl[0][1], pl[1][0], pl[1][1], b0, b1);
      } else {
        mma_bf16(o[t], ph[0][0], pl[0][0], ph[1][0], pl[1][0], b0, b1);
      }
    }
    if (jn < j1) fetch_v(jn);
  }
  // ---- the warps of this CTA: O fragment element (row r, column 2 c + e of tile t) is dim NT (2 c + e) + t
  float *mine = sm + warp * HMAX * ROW;
#pragma unroll
  for (int i = 0; i < (G16 ? 2 : 1); i++) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1), l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    float *row = mine + (r + 8 * i) * ROW;
    if (c == 0) row[0] = m[i], row[1] = l[i];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) row[2 + NT * (2 * c + e) + t] = G16 ? o[t][2 * i + e] : o[t][e] + o[t][2 + e];
  }
  float sum = 0.f;
#pragma unroll
  for (int t = 0; t < NT; t++) sum += (o[t][0] + o[t][1]) + (o[t][2] + o[t][3]);
#pragma unroll
  for (int i = 0; i < (G16 ? 2 : 1); i++) sum += l[i];
  if (__any_sync(0xffffffffu, sum != sum)) {  // NaN: of infinities met by hi and lo, or truly; the warp's keys once more tell which
    __syncwarp();
    for (int h = 0; h < g; h++)
      attend_plain<D>(static_cast<const __nv_bfloat16 *>(a.q) + ((size_t)b * a.NH + (size_t)kh * g + h) * D, Kb, Vb, reinterpret_cast<const __nv_bfloat16 *>(fresh),
                      append ? (int)pos : -1, roped ? trig : nullptr, sc, j0 + warp * 16, j1, mine + h * ROW);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < g * D; idx += MA_THREADS) {
    const int h = idx / D, d = idx - h * D;
    float M = -INFINITY, L = 0.f, A = 0.f;
#pragma unroll
    for (int w = 0; w < MA_WARPS; w++) M = fmaxf(M, sm[(w * HMAX + h) * ROW]);
    if (M > -INFINITY) {
#pragma unroll
      for (int w = 0; w < MA_WARPS; w++) {
        const float *row = sm + (w * HMAX + h) * ROW;
        const float e = exp2f(row[0] - M);
        L = fmaf(e, row[1], L), A = fmaf(e, row[2 + d], A);
      }
    }
    cpart[h * ROW + 2 + d] = A;
    if (d == 0) cpart[h * ROW] = M, cpart[h * ROW + 1] = L;
  }
  if (KS > 1) umma::cluster_sync();
  else __syncthreads();
  cluster_combine<__nv_bfloat16, true>(a, cpart, g, D, ROW, KS, rank, b, kh, MA_THREADS);
}

template <typename T>
__global__ void kv_append_kernel(const T *__restrict__ k, const T *__restrict__ v, T *__restrict__ kbuf, T *__restrict__ vbuf,
                                 const long long *__restrict__ pos, long long n, int D, int Cap) {
  pdl_launch_dependents();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long p = pos[0];
  if (p < 0 || p >= Cap) {
    if (i == 0) atomicOr(&g_attn_status, 1u);
    return;
  }
  const long long bh = i / D;
  const long long dst = (bh * Cap + p) * D + (i - bh * D);
  kbuf[dst] = k[i];
  vbuf[dst] = v[i];
}

__global__ void inc_i64_kernel(long long *p, int n) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] += 1;
}

template <typename K, typename... Args>
cudaError_t launch_chain(K kern, dim3 grid, dim3 block, size_t smem, unsigned cluster_y, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1, attr[1].val.clusterDim.y = cluster_y, attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster_y > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <typename T, int PER, int GH>
int launch_attn(const AttnArgs &a, int ks, cudaStream_t st) {
  auto kern = decode_attn_kernel<T, PER, GH>;
  const size_t smem = AttnCfg<PER, GH>::smem(a.NH / a.KH);
  static DeviceOnce smem_set;  // per instantiation and device: the largest size opted in so far
  {
    cudaError_t e = smem_set.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }, smem);
    if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  }
  cudaError_t e = launch_chain(kern, dim3((unsigned)(a.B * a.KH), (unsigned)ks), dim3(DA_THREADS), smem, (unsigned)ks, st, a);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  return launched("decode_attn");
}

// heads per pass: the smallest of 1, 2, 4, ... that covers the group, while heads x dims-per-lane stays
// within 32 accumulators per lane (larger groups walk the keys again; they hit in L2)
template <typename T, int PER>
int launch_attn_g(const AttnArgs &a, int ks, cudaStream_t st) {
  constexpr int GMAX = 32 / PER < DA_MAX_G ? 32 / PER : DA_MAX_G;
  const int g = a.NH / a.KH;
  if constexpr (GMAX >= 2) {
    if (g <= GMAX / 2) {
      if constexpr (GMAX >= 4) {
        if (g <= GMAX / 4) return launch_attn<T, PER, GMAX / 4>(a, ks, st);
      }
      return launch_attn<T, PER, GMAX / 2>(a, ks, st);
    }
  }
  return launch_attn<T, PER, GMAX>(a, ks, st);
}

template <int D, bool G16>
int launch_mma(const AttnArgs &a, cudaStream_t st) {
  auto kern = decode_attn_mma_kernel<D, G16>;
  constexpr int HMAX = G16 ? 16 : 8;
  constexpr size_t smem = (size_t)((MA_WARPS + 1) * HMAX * (D + 2) + D + D) * sizeof(float);
  static DeviceOnce smem_set;
  cudaError_t e = smem_set.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }, smem);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  // as many CTAs along the keys as fit on the SMs at once, with 64 keys of the capacity (a block of each warp) or more for each
  const int slots = mma_ctas(D) * sm_count();
  int ks = 1;
  while (ks < 8 && a.B * a.KH * (ks + 1) <= slots && a.Cap >= 64 * (ks + 1)) ks++;
  e = launch_chain(kern, dim3((unsigned)(a.B * a.KH), (unsigned)ks), dim3(MA_THREADS), smem, (unsigned)ks, st, a);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  return launched("decode_attn");
}

template <int D, int GH>
int launch_f32(const AttnArgs &a, cudaStream_t st) {
  auto kern = decode_attn_f32_kernel<D, GH>;
  constexpr size_t smem = F32Cfg<D, GH>::SMEM;
  static DeviceOnce smem_set;
  cudaError_t e = smem_set.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }, smem);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  // as many CTAs along the keys as fit on the SMs at once, with a tile of the capacity or more for each
  const int slots = (D == 64 ? 2 : 1) * sm_count();
  int ks = 1;
  while (ks < 8 && a.B * a.KH * (ks + 1) <= slots && a.Cap >= FT_KEYS * (ks + 1)) ks++;
  e = launch_chain(kern, dim3((unsigned)(a.B * a.KH), (unsigned)ks), dim3(FT_THREADS), smem, (unsigned)ks, st, a);
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn: %s", cudaGetErrorString(e));
  return launched("decode_attn");
}

template <int D>
int launch_f32_g(const AttnArgs &a, int g, cudaStream_t st) {
  return g == 1 ? launch_f32<D, 1>(a, st) : g == 2 ? launch_f32<D, 2>(a, st) : g <= 4 ? launch_f32<D, 4>(a, st) : g <= 8 ? launch_f32<D, 8>(a, st) : launch_f32<D, 16>(a, st);
}

template <typename T>
int launch_attn_d(const AttnArgs &a, int D, int ks, cudaStream_t st) {
  switch (D / 32) {
    case 1: return launch_attn_g<T, 1>(a, ks, st);
    case 2:
      if constexpr (sizeof(T) == 2) return launch_attn_g<T, 2>(a, ks, st);  // a bf16 cache that is not on 32 bytes
      break;
    case 4:
      if constexpr (sizeof(T) == 2) return launch_attn_g<T, 4>(a, ks, st);
      break;
    case 8: return launch_attn_g<T, 8>(a, ks, st);
    case 16: return launch_attn_g<T, 16>(a, ks, st);
  }
  return fail(LB200_E_SHAPE, "light_b200: decode_attn: head dim %d (want 32, 64, 128, 256 or 512)", D);
}

}  // namespace

int decode_attn(const lb200_decode_attn_args *p, cudaStream_t st) {
  if (!p) return fail(LB200_E_NULL, "light_b200: decode_attn: null argument block");
  if (!p->q || !p->kbuf || !p->vbuf || !p->pos || !p->out || (!p->k_new) != (!p->v_new))
    return fail(LB200_E_NULL, "light_b200: decode_attn: null pointer (k_new and v_new come together)");
  if (p->dtype != LB200_F32 && p->dtype != LB200_BF16) return fail(LB200_E_DTYPE, "light_b200: decode_attn: element type %d", p->dtype);
  if (p->B <= 0 || p->NH <= 0 || p->KH <= 0 || p->Cap <= 0 || p->D <= 0 || p->NH % p->KH || p->window < 0)
    return fail(LB200_E_SHAPE, "light_b200: decode_attn: B %d NH %d KH %d Cap %d D %d window %d", p->B, p->NH, p->KH, p->Cap, p->D, p->window);
  const int g = p->NH / p->KH;
  // the reference's own limits (kernels/cuda/decode_attn.go:36-38): other shapes take its composed path
  if (p->D % 32 || p->D > 512 || g > DA_MAX_G) return fail(LB200_E_SHAPE, "light_b200: decode_attn: head dim %d / group %d unsupported", p->D, g);
  if ((long long)p->B * p->KH > 65535ll * 1024) return fail(LB200_E_TOO_LARGE, "light_b200: decode_attn: B x KH too large");
  const uintptr_t al = (uintptr_t)p->q | (uintptr_t)p->kbuf | (uintptr_t)p->vbuf | (uintptr_t)p->k_new | (uintptr_t)p->v_new;
  if (al & 15) return fail(LB200_E_ALIGN, "light_b200: decode_attn: q / k / v must be 16-byte aligned");
  if (p->rope_base < 0.f) return fail(LB200_E_SHAPE, "light_b200: decode_attn: rope_base %g", (double)p->rope_base);
  const double rope_k = p->rope_base > 0.f ? -2.0 * log2((double)p->rope_base) / (double)p->D : 0.0;
  AttnArgs a{p->q, p->k_new, p->v_new, p->kbuf, p->vbuf, p->out, (const long long *)p->pos, p->B, p->NH, p->KH, p->Cap, p->window, p->scale, rope_k};
  // bf16 caches with 64- or 128-wide heads: the tensor-core kernel (its 256-bit loads want rows on 32 bytes)
  if (p->dtype == LB200_BF16 && (p->D == 64 || p->D == 128) && !(((uintptr_t)p->kbuf | (uintptr_t)p->vbuf) & 31)) {
    if (p->D == 64) return g <= 8 ? launch_mma<64, false>(a, st) : launch_mma<64, true>(a, st);
    return g <= 8 ? launch_mma<128, false>(a, st) : launch_mma<128, true>(a, st);
  }
  if (p->dtype == LB200_F32 && p->D == 64) return launch_f32_g<64>(a, g, st);
  if (p->dtype == LB200_F32 && p->D == 128) return launch_f32_g<128>(a, g, st);
  // enough CTAs to fill the GPU, at least 32 keys of the capacity each, a portable cluster
  int ks = 1;
  while (ks < 8 && p->B * p->KH * ks < 148 && p->Cap >= 64 * ks) ks *= 2;
  return p->dtype == LB200_F32 ? launch_attn_d<float>(a, p->D, ks, st) : launch_attn_d<__nv_bfloat16>(a, p->D, ks, st);
}

int kv_append(const void *k, const void *v, void *kbuf, void *vbuf, const int64_t *pos, int dtype, int B, int KH, int D, int Cap,
              cudaStream_t st) {
  if (!k || !v || !kbuf || !vbuf || !pos) return fail(LB200_E_NULL, "light_b200: kv_append: null pointer");
  if (B <= 0 || KH <= 0 || D <= 0 || Cap <= 0) return fail(LB200_E_SHAPE, "light_b200: kv_append: B %d KH %d D %d Cap %d", B, KH, D, Cap);
  const long long n = (long long)B * KH * D;
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaError_t e;
  if (dtype == LB200_F32)
    e = launch_chain(kv_append_kernel<float>, dim3(grid), dim3(256), 0, 1, st, (const float *)k, (const float *)v, (float *)kbuf, (float *)vbuf,
                     (const long long *)pos, n, D, Cap);
  else if (dtype == LB200_BF16)
    e = launch_chain(kv_append_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, 1, st, (const __nv_bfloat16 *)k, (const __nv_bfloat16 *)v,
                     (__nv_bfloat16 *)kbuf, (__nv_bfloat16 *)vbuf, (const long long *)pos, n, D, Cap);
  else
    return fail(LB200_E_DTYPE, "light_b200: kv_append: element type %d", dtype);
  if (e != cudaSuccess) return fail((int)e, "light_b200: kv_append: %s", cudaGetErrorString(e));
  return launched("kv_append");
}

int inc_i64(int64_t *p, int n, cudaStream_t st) {
  if (!p) return fail(LB200_E_NULL, "light_b200: inc_i64: null pointer");
  if (n <= 0) return fail(LB200_E_SHAPE, "light_b200: inc_i64: n %d", n);
  cudaError_t e = launch_chain(inc_i64_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, 1, st, (long long *)p, n);
  if (e != cudaSuccess) return fail((int)e, "light_b200: inc_i64: %s", cudaGetErrorString(e));
  return launched("inc_i64");
}

int decode_attn_status() {
  unsigned int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_attn_status, sizeof(v));
  if (e != cudaSuccess) return fail((int)e, "light_b200: decode_attn_status: %s", cudaGetErrorString(e));
  return (int)v;
}

}  // namespace lb
