// Grouped expert matmul over routed (token, slot) pairs (contract: reference
// kernels/cuda/src/moe.cu:1-24, ops/moe.go:96-107):
//
//   out[p, :] = w(p) * input[row(p), :] . weights[e, :, :]^T      for every sorted pair
//
// Pairs arrive sorted by expert, so expert e owns the index range offsets[e] .. offsets[e+1].
// The ranges come from boundary detection on the sorted expert ids (no atomics, deterministic);
// every output row is written by exactly one warp lane set, so the result is deterministic too.
#include <cuda_fp8.h>

#include <mutex>

#include "gguf_decode.cuh"
#include "mma_sync.cuh"

namespace lb {

// Non-zero once an expert id outside [0, E) was seen by the offsets kernel (sticky; light_b200_moe_route_status
// reports it together with the routing kernels' own word).
__device__ unsigned int g_moe_bad_ids;

// First sorted index whose expert id is >= e.
__device__ __forceinline__ int first_of(const int64_t *ids, long long M, long long e) {
  int lo = 0, hi = (int)M;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ids[mid] < e) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// offsets[e] = first sorted index whose expert id is >= e, for e <= E (so offsets[E] = M when every id is an expert), and
// counts[e], each by its own binary search: every entry is written whatever the ids are, so nothing has to be cleared before.
// Nobody validates the ids before this kernel, so it does.  A search is monotone in e even over unsorted ids: the offsets never
// decrease and stay in [0, M].  A negative id owns no range, an id >= E lies at or beyond offsets[E], outside every
// expert's range (the matmul kernels skip both), and either sets the status word.
// `clear`: words that the launches after this one want zero.
__global__ void __launch_bounds__(256) moe_prep_kernel(const int64_t *__restrict__ ids, int32_t *__restrict__ offsets, int32_t *__restrict__ counts,
                                                       long long M, int E, uint32_t *__restrict__ clear, int clear_words) {
  pdl_launch_dependents();
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (int c = (int)i; c < clear_words; c += gridDim.x * 256) clear[c] = 0u;
  if (i < M) {
    const long long e = ids[i];
    if (e < 0 || e >= E) g_moe_bad_ids = 1u;
  }
  if (i > E) return;
  const int o = first_of(ids, M, i);
  offsets[i] = o;
  if (i < E) counts[i] = first_of(ids, M, i + 1) - o;
}

// The output rows that no pair of the routing writes (ids that are no experts, pair ids out of range or missing) are zero.  A bit
// per row is set by the pairs that are sure to write, and the rows without one are cleared: clearing all of `out` instead costs a
// pass over it (32768 x 7168 bf16: 110 us against 5).  Sure are those with an expert's id that lie in [offsets[0], offsets[E]) as
// well: some of the matmul kernels go by the one, some by the other, and over ids that are not sorted the two differ.
__global__ void __launch_bounds__(256) moe_mark_kernel(const int64_t *__restrict__ pairs, const int64_t *__restrict__ ids, uint32_t *__restrict__ bits,
                                                       long long M, long long rows, int E) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int range[2];
  if (threadIdx.x < 2) range[threadIdx.x] = first_of(ids, M, threadIdx.x ? E : 0);
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  const long long p = pairs[i], e = ids[i];
  if (p >= 0 && p < rows && e >= 0 && e < E && i >= range[0] && i < range[1]) atomicOr(bits + (p >> 5), 1u << (p & 31));
}
__global__ void __launch_bounds__(256) moe_clear_kernel(const uint32_t *__restrict__ bits, char *__restrict__ out, long long rows, long long row_bytes) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // a warp to 32 rows
  if (w * 32 >= rows) return;
  for (uint32_t left = ~bits[w]; left; left &= left - 1) {
    const long long r = w * 32 + __ffs(left) - 1;
    if (r >= rows) break;
    for (long long k = lane * 2; k < row_bytes; k += 64) *reinterpret_cast<uint16_t *>(out + r * row_bytes + k) = 0;
  }
}

__device__ __forceinline__ void load8(const float *p, float v[8]) {
  float4 a = __ldg(reinterpret_cast<const float4 *>(p)), b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16 *p, float v[8]) {
  uint4 u = __ldg(reinterpret_cast<const uint4 *>(p));
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x, v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const __half *p, float v[8]) {
  uint4 u = __ldg(reinterpret_cast<const uint4 *>(p));
  const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float2 f = __half22float2(h[i]);
    v[2 * i] = f.x, v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void st_out(float *p, long long i, float v) { p[i] = v; }
__device__ __forceinline__ void st_out(__nv_bfloat16 *p, long long i, float v) { p[i] = __float2bfloat16_rn(v); }
__device__ __forceinline__ void st_out(__half *p, long long i, float v) { p[i] = __float2half_rn(v); }

constexpr int MOE_MT = 8;     // sorted pairs per tile
constexpr int MOE_WARPS = 8;  // output columns per CTA

// What a row fetcher needs beyond the weight pointer: block-scaled FP8 (scale, bR, bC) and group-quantized 4-bit
// (scale, zeros, bC = group).
struct RowAux {
  const float *scale;
  int bR, bC;
  const float *zeros;
};

// Weight row fetchers: eight consecutive K elements of row n of expert e as f32.
template <typename T>
struct DenseRow {
  const T *row;
  __device__ DenseRow(const void *w, long long e, int n, int N, int K, const RowAux &) : row((const T *)w + ((size_t)e * N + n) * K) {}
  __device__ __forceinline__ void get(int k, float v[8]) const { load8(row + k, v); }
};
template <int QT>
struct QuantRow {
  const uint8_t *row;
  __device__ QuantRow(const void *w, long long e, int n, int N, int K, const RowAux &)
      : row((const uint8_t *)w + ((size_t)e * N + n) * (size_t)(K / block_elems(QT)) * block_bytes(QT)) {}
  __device__ __forceinline__ void get(int k, float v[8]) const {
    int b = k / block_elems(QT);
    decode8<QT>(row + (size_t)b * block_bytes(QT), k - b * block_elems(QT), v);
  }
};

// Block-scaled e4m3 codes (E, N, K) with f32 scales (E, N / bR, K / bC), bC % 8 == 0: the weight is code * scale
// rounded to the activation type TA, i.e. the value a dequantize-then-matmul at that type multiplies with
// (reference ops/fp8_block.go:13-60 followed by ops.MoEGemm).
template <typename TA>
struct F8BlockRow {
  const uint8_t *row;
  const float *srow;
  int bC;
  __device__ F8BlockRow(const void *w, long long e, int n, int N, int K, const RowAux &aux)
      : row((const uint8_t *)w + ((size_t)e * N + n) * K),
        srow(aux.scale + ((size_t)e * (N / aux.bR) + n / aux.bR) * (size_t)(K / aux.bC)),
        bC(aux.bC) {}
  __device__ __forceinline__ void get(int k, float v[8]) const {
    const uint2 q = __ldg(reinterpret_cast<const uint2 *>(row + k));
    const float sc = __ldg(srow + k / bC);
    const uint32_t u[2] = {q.x, q.y};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(u[h] & 0xFFFFu), __NV_E4M3);
      __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(u[h] >> 16), __NV_E4M3);
      const float2 a = __half22float2(__half2(lo)), b = __half22float2(__half2(hi));
      v[4 * h + 0] = round_to(a.x * sc), v[4 * h + 1] = round_to(a.y * sc), v[4 * h + 2] = round_to(b.x * sc), v[4 * h + 3] = round_to(b.y * sc);
    }
  }
  static __device__ __forceinline__ float round_to(float f) {
    if constexpr (sizeof(TA) == 2) return __bfloat162float(__float2bfloat16_rn(f));
    return f;
  }
};

// Group-quantized 4-bit rows in the canonical layout (codes u32 (N, K/8), nibble j of word c = W[n, 8c + j]; scales and
// zeros f32 (N, K/G), G % 8 == 0): eight weights are one code word, w = s * (q - z) with the two operations rounded
// separately, as the dequantize kernel forms them.
struct Int4Row {
  const uint32_t *row;
  const float *srow, *zrow;
  int G;
  __device__ Int4Row(const void *w, long long e, int n, int N, int K, const RowAux &aux)
      : row((const uint32_t *)w + ((size_t)e * N + n) * (size_t)(K / 8)),
        srow(aux.scale + ((size_t)e * N + n) * (size_t)(K / aux.bC)),
        zrow(aux.zeros + ((size_t)e * N + n) * (size_t)(K / aux.bC)),
        G(aux.bC) {}
  __device__ __forceinline__ void get(int k, float v[8]) const {
    const uint32_t q = __ldg(row + (k >> 3));
    const float sc = __ldg(srow + k / G), zp = __ldg(zrow + k / G);
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __fmul_rn(sc, __fsub_rn((float)((q >> (4 * j)) & 0xFu), zp));
  }
};

// One warp: one output column n, the pairs of one tile.  A tile may straddle experts; each run
// of equal expert id inside it is handled with that expert's weight row.
template <typename TI, typename TO, typename Row>
__global__ void __launch_bounds__(MOE_WARPS * 32) moe_gemm_kernel(
    const TI *__restrict__ in, const void *__restrict__ w, const int64_t *__restrict__ pairs,
    const int64_t *__restrict__ ids, const int32_t *__restrict__ offsets, const float *__restrict__ topkw,
    TO *__restrict__ out, long long M, long long sizeM, int E, int N, int K, int topk, int rowPerPair, RowAux aux) {
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * MOE_WARPS + (threadIdx.x >> 5);
  if (n >= N) return;
  const long long t0 = (long long)blockIdx.y * MOE_MT, t1 = t0 + MOE_MT < M ? t0 + MOE_MT : M;
  long long i = t0;
  while (i < t1) {
    const long long e = ids ? ids[i] : 0;  // no routing: one weight matrix, row m of the input gives row m of the output
    if (e < 0 || e >= E) {  // not an expert: the pair is skipped, as an out-of-range pair id is
      i++;
      continue;
    }
    long long r1 = ids ? offsets[e + 1] : t1;
    if (r1 > t1) r1 = t1;
    if (r1 <= i) r1 = i + 1;  // unsorted input: still make progress
    const int cnt = (int)(r1 - i);
    const TI *xrow[MOE_MT];
    long long pr[MOE_MT];
#pragma unroll
    for (int m = 0; m < MOE_MT; m++) {
      long long p = m < cnt ? (pairs ? pairs[i + m] : i + m) : -1;
      if (p < 0 || p >= sizeM) p = -1;
      pr[m] = p;
      xrow[m] = p < 0 ? nullptr : in + (size_t)(rowPerPair ? p : p / topk) * K;
    }
    float acc[MOE_MT];
#pragma unroll
    for (int m = 0; m < MOE_MT; m++) acc[m] = 0.f;
    Row wr(w, e, n, N, K, aux);
    for (int k = lane * 8; k < K; k += 256) {
      float wv[8];
      wr.get(k, wv);
#pragma unroll
      for (int m = 0; m < MOE_MT; m++) {
        if (xrow[m]) {
          float xv[8];
          load8(xrow[m] + k, xv);
#pragma unroll
          for (int j = 0; j < 8; j++) acc[m] = fmaf(wv[j], xv[j], acc[m]);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MOE_MT; m++) {
      float v = warp_sum(acc[m]);
      if (lane == 0 && pr[m] >= 0) st_out(out, pr[m] * N + n, topkw ? v * topkw[pr[m]] : v);
    }
    i = r1;
  }
}

static int prep(const lb200_moe_args *a, cudaStream_t st, void *scratch = nullptr, size_t scratch_bytes = 0) {
  if (a->M > 0x7fffffffLL) return fail(LB200_E_TOO_LARGE, "light_b200: moe: %lld pairs", (long long)a->M);
  const int words = scratch && scratch_bytes >= moe_scratch_bytes(a->M, a->K) ? (int)(gemm_tmem_sync_bytes() / 4) : 0;
  long long work = a->M > a->E + 1 ? a->M : a->E + 1;
  if (words && work < 4096) work = 4096;  // (a few words a thread)
  launch_early(moe_prep_kernel, dim3((unsigned)((work + 255) / 256)), dim3(256), st, a->expert_ids, a->offsets, a->counts, (long long)a->M, a->E,
               (uint32_t *)scratch, words);
  return launched("moe expert offsets");
}

int moe_clear_unrouted(const int64_t *pairs, const int64_t *ids, uint32_t *bits, void *out, long long M, long long rows, long long row_bytes, int E,
                       cudaStream_t st) {
  if (rows == 0) return 0;
  const long long words = (rows + 31) / 32;
  cudaError_t e = cudaMemsetAsync(bits, 0, (size_t)words * 4, st);
  if (e != cudaSuccess) return fail((int)e, "light_b200: moe: %s", cudaGetErrorString(e));
  if (M > 0) launch_early(moe_mark_kernel, dim3((unsigned)((M + 255) / 256)), dim3(256), st, pairs, ids, bits, M, rows, E);
  launch_early(moe_clear_kernel, dim3((unsigned)((words + 7) / 8)), dim3(256), st, (const uint32_t *)bits, (char *)out, rows, row_bytes);
  return launched("moe: clear unrouted rows");
}

// ------------------------------------------------------------------------------------ Q6_K rows that start on any even byte
//
// An odd number of 210-byte blocks per row: the tensor-core kernels would round both operands to 11 bits, and these rows have always had
// f32 products, as below 256 pairs.  What bounds moe_gemm_kernel is the load unit: a warp to one weight row reads eight activation rows
// for every eight weights, and the weights a byte at a time.  Here a warp owns NC rows of one expert and MT of its tokens: an
// activation is loaded once for NC weights, a weight once for MT tokens, in 16-bit pieces.  Lanes split K, and the NC x MT sums end
// in a reduce-scatter over the warp (31 shuffles for 32 sums, not 160).  616 pairs over 128 experts of 2048 x 768: 780 -> 245 us;
// 2048 rows of 4096 x 14080: 42 -> 16 ms.  (With operands rounded to 11 bits the tensor-memory kernel takes 94 us and 0.25 ms.)

// Elements 4 lane .. + 3 of both halves of a block: sixteen bytes of activations to a lane are then whole lines to a warp.
__device__ __forceinline__ void q6k_eight(const uint8_t *b, int lane, float out[8]) {
  const int grp = lane >> 3, l0 = 4 * (lane & 7);
  const uint8_t *ql = b + (grp & 1) * 32 + l0, *qh = b + 128 + l0;
  const float d = f16_bits_to_f32(__ldg(reinterpret_cast<const uint16_t *>(b + 208)));
  auto word = [](const uint8_t *p) { return (uint32_t)__ldg(reinterpret_cast<const uint16_t *>(p)) | (uint32_t)__ldg(reinterpret_cast<const uint16_t *>(p) + 1) << 16; };
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float ds = __fmul_rn(d, (float)__ldg(reinterpret_cast<const int8_t *>(b) + 192 + 8 * h + 2 * grp + (l0 >> 4)));
    const uint32_t q = ((word(ql + 64 * h) >> (grp >> 1 ? 4 : 0)) & 0x0F0F0F0Fu) | ((word(qh + 32 * h) >> (2 * grp)) & 0x03030303u) << 4;
#pragma unroll
    for (int i = 0; i < 4; i++)  // 2^23 + code, less 2^23 + 32: exact
      out[4 * h + i] = __fmul_rn(ds, __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7440 + i)) - 8388640.f);
  }
}

// CHAIN: a lane's products one after the other into its sum, as moe_gemm_kernel adds them; else eight at a time, as the shape-generic
// matmul does (K = 14080: 1.6e-7 of the result against 3.8e-7).
template <int NC, int MT, bool CHAIN>
__global__ void __launch_bounds__(MOE_WARPS * 32, 2) q6k_rows_kernel(const float *__restrict__ in, const uint8_t *__restrict__ w, const int64_t *__restrict__ pairs,
                                                                 const int32_t *__restrict__ offsets, const float *__restrict__ topkw, float *__restrict__ out,
                                                                 long long M, long long size_m, int N, int K, int topk, int row_per_pair) {
  static_assert(NC * MT % 32 == 0 && MT <= 32, "a lane per token, whole sums per lane");
  const int lane = threadIdx.x & 31, n0 = (blockIdx.x * MOE_WARPS + (threadIdx.x >> 5)) * NC, e = blockIdx.y;
  if (n0 >= N) return;
  const size_t row_bytes = (size_t)(K >> 8) * 210;
  const uint8_t *row[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) row[c] = w + ((size_t)e * N + min(n0 + c, N - 1)) * row_bytes;
  const long long i0 = offsets ? offsets[e] : 0, i1 = offsets ? offsets[e + 1] : M;
  for (long long t = i0 + (long long)blockIdx.z * MT; t < i1; t += (long long)gridDim.z * MT) {
    const int cnt = (int)min((long long)MT, i1 - t);
    long long mine = -1;  // the pair of token `lane`
    if (lane < cnt) {
      mine = pairs ? pairs[t + lane] : t + lane;
      if (mine < 0 || mine >= size_m) mine = -1;
    }
    const long long from = mine < 0 ? 0 : row_per_pair ? mine : mine / topk;
    const float *x[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) x[m] = in + (size_t)__shfl_sync(0xffffffffu, from, m) * K;
    float acc[NC * MT];
#pragma unroll
    for (int i = 0; i < NC * MT; i++) acc[i] = 0.f;
    for (int b = 0; b < K >> 8; b++) {
      float wv[NC][8];
#pragma unroll
      for (int c = 0; c < NC; c++) q6k_eight(row[c] + b * 210, lane, wv[c]);
#pragma unroll
      for (int m = 0; m < MT; m++) {  // (a missing token reads row 0: with branches here the loads would wait for one another)
        const float4 *xp = reinterpret_cast<const float4 *>(x[m] + b * 256) + lane;
        const float4 u = __ldg(xp), v = __ldg(xp + 32);
        const float xv[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
        for (int c = 0; c < NC; c++) {
          if constexpr (CHAIN) {
#pragma unroll
            for (int j = 0; j < 8; j++) acc[m * NC + c] = fmaf(wv[c][j], xv[j], acc[m * NC + c]);
          } else {
            float s = wv[c][0] * xv[0];
#pragma unroll
            for (int j = 1; j < 8; j++) s = fmaf(wv[c][j], xv[j], s);
            acc[m * NC + c] += s;
          }
        }
      }
    }
    // Sum i of NC MT: a lane hands half of its sums to its partner at every step and keeps the other half.
    int base = 0;  // of the sums this lane still holds
#pragma unroll
    for (int off = 16, n = NC * MT / 2; off >= 1; off >>= 1, n /= 2) {
      const bool up = lane & off;
#pragma unroll
      for (int i = 0; i < NC * MT / 2; i++) {
        if (i < n) {
          const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
      if (up) base += n;
    }
#pragma unroll
    for (int i = 0; i < NC * MT / 32; i++) {
      const int m = (base + i) / NC, n = n0 + (base + i) % NC;
      const long long p = __shfl_sync(0xffffffffu, mine, m);
      if (p >= 0 && n < N) out[p * N + n] = topkw ? acc[i] * topkw[p] : acc[i];
    }
  }
}

template <bool CHAIN>
static int q6k_rows(const float *in, const void *w, const int64_t *pairs, const int32_t *offsets, const float *topkw, float *out, long long M, long long size_m,
                    int E, int N, int K, int topk, int row_per_pair, cudaStream_t st) {
  constexpr int NC = 4, MT = 8;
  const long long nb = (N + NC * MOE_WARPS - 1) / (NC * MOE_WARPS), tiles = (M + MT - 1) / MT, want = (8ll * sm_count() + nb * E - 1) / (nb * E);
  const unsigned z = (unsigned)(want < tiles ? want : tiles);  // CTAs that share an expert's tokens, where experts and rows alone do not fill the GPU
  q6k_rows_kernel<NC, MT, CHAIN><<<dim3((unsigned)nb, (unsigned)E, z), MOE_WARPS * 32, 0, st>>>(in, (const uint8_t *)w, pairs, offsets, topkw, out, M, size_m, N, K, topk,
                                                                                     row_per_pair);
  return launched("q6_k rows (f32)");
}

int q6k_rows_dense(const float *x, const void *w, float *out, int M, int N, int K, cudaStream_t st) {
  return q6k_rows<false>(x, w, nullptr, nullptr, nullptr, out, M, M, 1, N, K, 1, 1, st);
}

template <typename TI, typename TO, typename Row>
static int run(const lb200_moe_args *a, cudaStream_t st, RowAux aux = RowAux{nullptr, 0, 0, nullptr}) {
  if (a->M == 0 || a->N == 0) return 0;
  dim3 grid((a->N + MOE_WARPS - 1) / MOE_WARPS, (unsigned)((a->M + MOE_MT - 1) / MOE_MT));
  if ((a->M + MOE_MT - 1) / MOE_MT > 65535)
    return fail(LB200_E_TOO_LARGE, "moe_gemm: %lld pairs exceed the kernel's grid", (long long)a->M);
  moe_gemm_kernel<TI, TO, Row><<<grid, MOE_WARPS * 32, 0, st>>>(
      (const TI *)a->input, a->weights, a->sorted_pairs, a->expert_ids, a->offsets, a->topk_weights, (TO *)a->out, a->M,
      a->size_m, a->E, a->N, a->K, a->topk, a->row_per_pair, aux);
  return launched("moe_gemm");
}

// x (M, K) . W^T for one matrix through the same tile kernel (no routing): the shapes the tensor-core and one-row kernels
// of these formats do not take (K % 256 != 0, groups or blocks that are not multiples of 64).
template <typename T, typename Row>
static int run_plain(const void *x, const void *w, void *y, int M, int N, int K, const RowAux &aux, cudaStream_t st) {
  if (M == 0 || N == 0) return 0;
  dim3 grid((N + MOE_WARPS - 1) / MOE_WARPS, (unsigned)((M + MOE_MT - 1) / MOE_MT));
  if ((M + MOE_MT - 1) / MOE_MT > 65535) return fail(LB200_E_TOO_LARGE, "light_b200: matmul: %d rows exceed the kernel's grid", M);
  moe_gemm_kernel<T, T, Row><<<grid, MOE_WARPS * 32, 0, st>>>((const T *)x, w, nullptr, nullptr, nullptr, nullptr, (T *)y, M, M, 1, N, K, 1, 1, aux);
  return launched("matmul (row fetcher)");
}

int int4_rows_dot(const void *x, const uint32_t *codes, const float *s, const float *z, void *y, int act_dtype, int M, int N, int K, int G,
                  cudaStream_t st) {
  const RowAux aux{s, 0, G, z};
  if (act_dtype == LB200_F32) return run_plain<float, Int4Row>(x, codes, y, M, N, K, aux, st);
  return run_plain<__nv_bfloat16, Int4Row>(x, codes, y, M, N, K, aux, st);
}

int fp8_block_rows_dot(const void *x, const uint8_t *w, const float *s, void *y, int act_dtype, int M, int N, int K, int bR, int bC,
                       cudaStream_t st) {
  const RowAux aux{s, bR, bC, nullptr};
  if (act_dtype == LB200_F32) return run_plain<float, F8BlockRow<float>>(x, w, y, M, N, K, aux, st);
  return run_plain<__nv_bfloat16, F8BlockRow<__nv_bfloat16>>(x, w, y, M, N, K, aux, st);
}

int moe_bad_ids_status() {
  unsigned int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_moe_bad_ids, sizeof(v));
  if (e != cudaSuccess) return fail((int)e, "light_b200: moe status: %s", cudaGetErrorString(e));
  return (int)v;
}

size_t moe_scratch_bytes(long long M, int K) {
  return gemm_tmem_sync_bytes() + (((size_t)M * K * 2 + 1023) & ~(size_t)1023) + gemm_tmem_parts_bytes();
}

int moe_gemm(const lb200_moe_args *a, int device, cudaStream_t st, void *scratch, size_t scratch_bytes) {
  int rc = prep(a, st, scratch, scratch_bytes);
  if (rc) return rc;
  if (int took = moe_umma(a, 0, nullptr, 0, 0, device, st, scratch, scratch_bytes)) return took == 1 ? 0 : took;
  switch (a->dtype) {
    case LB200_F32: return run<float, float, DenseRow<float>>(a, st);
    case LB200_BF16: return run<__nv_bfloat16, __nv_bfloat16, DenseRow<__nv_bfloat16>>(a, st);
    case LB200_F16: return run<__half, __half, DenseRow<__half>>(a, st);
  }
  return fail(LB200_E_DTYPE, "moe_gemm: element type %d has no kernel", a->dtype);
}

// ---- grouped matmul whose expert counts / offsets live in this library's own device memory.
//
// The scratch is one file-scope device array, so the entry point needs no allocation by anyone:
// not by the caller, not by this library, not by a tensor pool.  In host code the array's name
// is only a stand-in for the device symbol, so its device address is looked up once per device
// (with that device current) and that address is what the kernels are given.
static __device__ __align__(256) int32_t g_moe_static_scratch[2 * LB200_MOE_STATIC_MAX_EXPERTS + 2];
static int32_t *g_moe_static_ptr[64];
static std::mutex g_moe_static_mu;

int moe_gemm_static_scratch(const lb200_moe_args *a, int device, cudaStream_t st) {
  if (a->E > LB200_MOE_STATIC_MAX_EXPERTS)
    return fail(LB200_E_TOO_LARGE, "light_b200: moe_gemm_static_scratch: %d experts exceed the built-in scratch (max %d)",
                a->E, LB200_MOE_STATIC_MAX_EXPERTS);
  int32_t *base;
  {
    std::lock_guard<std::mutex> lk(g_moe_static_mu);
    base = g_moe_static_ptr[device];
    if (!base) {  // first call on this device: resolve the symbol's device address
      cudaError_t e = cudaGetSymbolAddress((void **)&base, g_moe_static_scratch);
      if (e != cudaSuccess)
        return fail((int)e, "light_b200: moe_gemm_static_scratch: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      g_moe_static_ptr[device] = base;
    }
  }
  lb200_moe_args b = *a;
  b.counts = base;                                      // E entries
  b.offsets = base + LB200_MOE_STATIC_MAX_EXPERTS + 1;  // E + 1 entries
  // Both ranges are fully overwritten by the offsets / counts kernels before the matmul reads
  // them, so what an earlier call left behind never matters and nothing needs clearing.
  return moe_gemm(&b, device, st);
}

int moe_gemm_f8block(const lb200_moe_args *a, const float *w_scale, int bR, int bC, int device, cudaStream_t st, void *scratch, size_t scratch_bytes) {
  int rc = prep(a, st, scratch, scratch_bytes);
  if (rc) return rc;
  int took = moe_umma(a, 2, w_scale, bR, bC, device, st, scratch, scratch_bytes);
  if (took == 1) return 0;
  if (took) return took;
  // Few pairs (a decode step) without scratch of the call's own, or a shape the tensor-core path does not take: one warp per output column and
  // tile of sorted pairs, the weight row read once per tile.
  if (bR <= 0 || bC <= 0 || bC % 8 || a->K % bC || a->N % bR || a->K % 8)
    return fail(LB200_E_SHAPE, "light_b200: moe_gemm_f8block: N=%d K=%d with blocks (%d, %d): block_c must be a multiple of 8 and the blocks must tile the weight",
                a->N, a->K, bR, bC);
  const RowAux aux{w_scale, bR, bC, nullptr};
  if (a->dtype == LB200_F32) return run<float, float, F8BlockRow<float>>(a, st, aux);
  return run<__nv_bfloat16, __nv_bfloat16, F8BlockRow<__nv_bfloat16>>(a, st, aux);
}

int moe_gemm_q(const lb200_moe_args *a, int device, cudaStream_t st) {
  int rc = prep(a, st);
  if (rc) return rc;
  if (int took = moe_umma(a, 1, nullptr, 0, 0, device, st)) return took == 1 ? 0 : took;
  // From as many pairs on as the tensor-core path takes of the other formats.
  if (a->dtype == LB200_Q6_K && a->M >= 256 && a->K % 256 == 0 && a->E <= 65535 && a->N > 0)
    return q6k_rows<true>((const float *)a->input, a->weights, a->sorted_pairs, a->offsets, a->topk_weights, (float *)a->out, a->M, a->size_m, a->E, a->N, a->K,
                       a->topk, a->row_per_pair, st);
  switch (a->dtype) {
    case LB200_Q4_0: return run<float, float, QuantRow<LB200_Q4_0>>(a, st);
    case LB200_Q5_0: return run<float, float, QuantRow<LB200_Q5_0>>(a, st);
    case LB200_Q8_0: return run<float, float, QuantRow<LB200_Q8_0>>(a, st);
    case LB200_Q4_K: return run<float, float, QuantRow<LB200_Q4_K>>(a, st);
    case LB200_Q5_K: return run<float, float, QuantRow<LB200_Q5_K>>(a, st);
    case LB200_Q6_K: return run<float, float, QuantRow<LB200_Q6_K>>(a, st);
  }
  return fail(LB200_E_DTYPE, "moe_gemm_q: ggml type %d has no kernel", a->dtype);
}

}  // namespace lb
