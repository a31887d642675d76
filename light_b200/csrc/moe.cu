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
#include "umma.cuh"

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
// An odd number of 210-byte blocks per row: the tensor-memory kernel would round both operands to 11 bits, where this call multiplies f32 by
// f32 (as below 256 pairs it does at any K).  These are the products one by one, for calls without scratch; the limbs further down
// are what calls with scratch have.  What bounds moe_gemm_kernel is the load unit: a warp to one weight row reads eight activation rows
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

// ------------------------------------------------------------------------------------ the same products on the tensor cores
//
// What bounds q6k_rows_kernel is f32 issue: eight multiply-adds per lane, token and weight row for every block.  Here an activation is the sum
// of three f16 values (LIMBS), and a code is exact in f16.  The first limb is a whole number of 2^-8 of the power of two above the largest
// of the block's 256, so that its sums are exact; the second and third are the rest, rounded to eleven bits and again.  An activation above
// 2^-9 of that power so keeps all its bits, one below 23 of its own, down to 2^-37: f32 products hold 24.  (In fixed point to the
// end, the third limb 2^-30 of that power, small activations lost bits: 512 outputs of 768 whose weights are zero at one
// element of 1000 beside N(0, 0.05) were 5.5e-6 off; 9.5e-8 now, 8.9e-8 with f32 products.)  Below 2^-37 of it an element is off by up to 2^-52 of the
// first limb's unit, all 256 of a block together by up to 2^-32 of that unit times |d| (a weight is at most 2^12 |d|).  Such blocks carry a mark (ups is negative), and
// an output that is not 2^25 times as large as what its marked blocks may have lost is multiplied again, element by element: its weights are zero, or cancel, at the
// large activations (beside 1e12 such outputs were 6.3e-6 off, beside 3e30 nothing was left of them).  One MMA (m16n8k16: 16 rows, 8 tokens, one limb) is a sub-block's sum: three of
// them and 12 f32 operations a lane (limbs together, times the sub-block's scale) replace 64 multiply-adds.  Building
// the operand takes some 900 of the 1665 instructions per 16 rows, block and 16 tokens, and issue is what bounds this kernel
// (63 % of the slots, the tensor pipe 24 %).
//   616 pairs over 128 experts of 2048 x 768:  247 -> 117 us;   2048 rows of 4096 x 14080:  16.2 -> 5.4 ms;   65 rows of 4096 x 2816:
//   110 -> 68 us.  Blocks are added with their rounding errors kept (5 % of the time): 2.5e-8 off against 64 bits with normal inputs where the
//   f32 products are 8.1e-8 to 1.59e-7 off (K = 256 to 14080; without, 1.1e-7 at 11008).
// Tried: limbs of eight bits and the integer MMAs (m16n8k32), 194 us and 19.5 ms: they run at a fraction of the f16 rate here; limbs
// straight from L2, 152 us and 8.8 ms; 32 rows to a warp and half the warps, 115 us and 5.5 ms.
// Tokens with infinities or NaN (whose limbs mean nothing; their power of two is NaN) are too.
constexpr int LIMB_RECORD = 1536;  // a token's block: [sub-block][t][limbs 0, 1 of four k], then [sub-block][t][limb 2 of four k]
constexpr int LIMB_CHUNK = 4096;   // rows whose limbs are kept at a time: six bytes per activation
constexpr int LIMB_PASS = 16, LIMB_WARPS = 8, LIMB_RT = 1, LIMB_ROWS = 16 * LIMB_RT;
constexpr int LIMB_RING = 2, LIMB_PITCH = 240, LIMB_SLOT = LIMB_ROWS * LIMB_PITCH;  // blocks of a warp's rows on their way
constexpr int LIMB_TOKEN = LIMB_RECORD + 64, LIMB_STAGE = LIMB_PASS * LIMB_TOKEN;   // the pass's tokens, in shared memory for all warps; the pad
                                                                                   // puts neighbours' 64 bytes on different banks
constexpr int LIMB_SMEM = LIMB_WARPS * LIMB_RING * LIMB_SLOT + 2 * LIMB_STAGE;      // (two CTAs to an SM)
__device__ int g_limb_status;  // non-zero: a bounded wait gave up (sticky)

// Records of rows (of pairs, in expert order) first .. first + M - 1.
__global__ void __launch_bounds__(256) x_limbs_kernel(const float *__restrict__ in, const int64_t *__restrict__ pairs, uint8_t *__restrict__ limbs, float *__restrict__ ups,
                                                      long long first, long long M, int K, int topk, int row_per_pair, long long size_m) {
  pdl_launch_dependents();
  pdl_wait();
  const int nb = K >> 8, lane = threadIdx.x & 31;
  const long long rec = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (rec >= M * nb) return;
  const long long i = rec / nb;
  const int b = (int)(rec - i * nb);
  long long p = pairs ? pairs[first + i] : first + i;
  if (p < 0 || p >= size_m) p = 0;  // (not stored)
  const float4 *x = reinterpret_cast<const float4 *>(in + (size_t)(row_per_pair ? p : p / topk) * K + b * 256);
  const float4 v[2] = {__ldg(x + lane), __ldg(x + lane + 32)};
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 2; j++)
    m = max(max(m, max(__float_as_uint(v[j].x) & 0x7fffffffu, __float_as_uint(v[j].y) & 0x7fffffffu)),
            max(__float_as_uint(v[j].z) & 0x7fffffffu, __float_as_uint(v[j].w) & 0x7fffffffu));
  m = __reduce_max_sync(0xffffffffu, m);
  const int s = min(156 - (int)(m >> 23), 126);  // |x| 2^s < 2^30
  const float scale = __uint_as_float((uint32_t)(127 + s) << 23);
  bool small = false;  // an element other than zero below 2^-37 of the power of two above the largest
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
    for (int k = 0; k < 4; k++) small |= e[k] != 0.f && fabsf(e[k] * scale) < 0x1p-7f;
  }
  small = __any_sync(0xffffffffu, small);
  const uint32_t unit = (uint32_t)(149 - s) << 23 | (small ? 0x80000000u : 0u);  // of the first limb: 2^22
  if (lane == 0) ups[rec] = __uint_as_float(m >= 0x7f800000u ? 0x7fc00000u : unit);
  uint8_t *dst = limbs + (size_t)rec * LIMB_RECORD;
#pragma unroll
  for (int j = 0; j < 2; j++) {  // elements 128 j + 4 lane ..: sub-block 8 j + lane / 4, t = lane % 4
    const float xs[4] = {v[j].x * scale, v[j].y * scale, v[j].z * scale, v[j].w * scale};
    uint32_t l[3][2];
#pragma unroll
    for (int k = 0; k < 2; k++) {  // x 2^s = 2^22 l2 + 2^6 l1 + 2^-5 l0; every difference is exact
      const float a = xs[2 * k], b = xs[2 * k + 1], ta = rintf(a * 0x1p-22f), tb = rintf(b * 0x1p-22f);
      const float ra = fmaf(ta, -0x1p22f, a), rb = fmaf(tb, -0x1p22f, b);
      const __half2 h2 = __floats2half2_rn(ta, tb), h1 = __floats2half2_rn(ra * 0x1p-6f, rb * 0x1p-6f);
      const float2 back = __half22float2(h1);
      const __half2 h0 = __floats2half2_rn(fmaf(back.x, -0x1p6f, ra) * 0x1p5f, fmaf(back.y, -0x1p6f, rb) * 0x1p5f);
      l[0][k] = *reinterpret_cast<const uint32_t *>(&h0), l[1][k] = *reinterpret_cast<const uint32_t *>(&h1), l[2][k] = *reinterpret_cast<const uint32_t *>(&h2);
    }
    const int at = (8 * j + (lane >> 2)) * 4 + (lane & 3);
    *reinterpret_cast<uint4 *>(dst + at * 16) = make_uint4(l[0][0], l[0][1], l[1][0], l[1][1]);
    *reinterpret_cast<uint2 *>(dst + 1024 + at * 8) = make_uint2(l[2][0], l[2][1]);
  }
}

__device__ __forceinline__ void mma_from_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

__global__ void __launch_bounds__(LIMB_WARPS * 32, 2) q6k_limbs_kernel(const float *__restrict__ in, const uint8_t *__restrict__ w, const uint8_t *__restrict__ limbs,
                                                                   const float *__restrict__ ups, const int64_t *__restrict__ pairs, const int32_t *__restrict__ offsets,
                                                                   const float *__restrict__ topkw, float *__restrict__ out, long long first, long long M, long long size_m, int E,
                                                                   int N, int K, int topk, int row_per_pair) {
  extern __shared__ __align__(16) unsigned char ring_mem[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, e = blockIdx.y;
  const uint32_t bar0 = umma::smem_u32(bars), stages = umma::smem_u32(ring_mem) + LIMB_WARPS * LIMB_RING * LIMB_SLOT;
  if (threadIdx.x == 0) {
    umma::mbar_init(bar0, 1), umma::mbar_init(bar0 + 8, 1);
    umma::fence_barrier_init();
    abort_flag = 0;
  }
  pdl_launch_dependents();
  pdl_wait();
  __syncthreads();
  const long long i0 = max(offsets ? (long long)offsets[e] : 0ll, first), i1 = min(offsets ? (long long)offsets[e + 1] : first + M, first + M);
  if (i0 + (long long)blockIdx.z * LIMB_PASS >= i1) return;
  const int r0 = min((int)(blockIdx.x * LIMB_WARPS + warp) * LIMB_ROWS, N - LIMB_ROWS), nb = K >> 8;  // the last rows are pulled back: duplicates store equal values
  const size_t row_bytes = (size_t)nb * 210;
  const uint8_t *const rows = w + ((size_t)e * N + r0) * row_bytes, *const w_end = w + (size_t)E * N * row_bytes;
  const uint32_t ring = umma::smem_u32(ring_mem) + warp * (LIMB_RING * LIMB_SLOT);
  const uint32_t skew0 = (uint32_t)(uintptr_t)(rows + g * row_bytes);  // (rows g, g + 8, .. lie multiples of 16 bytes apart)
  // Lanes 0 .. 13 / 16 .. 29 copy the 14 granules that cover a block of rows 2 i / 2 i + 1.
  auto issue = [&](int b, int slot) {
    if ((lane & 15) < 14 && b < nb) {
      const uint8_t *at = rows + (size_t)(lane >> 4) * row_bytes + (size_t)b * 210;
      uint32_t dst = ring + slot * LIMB_SLOT + (lane >> 4) * LIMB_PITCH + (lane & 15) * 16;
#pragma unroll 4
      for (int i = 0; i < LIMB_ROWS / 2; i++, at += 2 * row_bytes, dst += 2 * LIMB_PITCH) {
        const uint8_t *src = reinterpret_cast<const uint8_t *>((uintptr_t)at & ~(uintptr_t)15) + (lane & 15) * 16;
        if (src + 16 <= w_end) cp_async16(dst, src);
        else if (src < w_end) cp_async16_part(dst, src, (uint32_t)(w_end - src));
      }
    }
    cp_async_commit();
  };
  uint32_t used = 0;  // stages consumed so far
  for (long long t0 = i0 + (long long)blockIdx.z * LIMB_PASS; t0 < i1; t0 += (long long)gridDim.z * LIMB_PASS) {
    const int cnt = (int)min((long long)LIMB_PASS, i1 - t0);
    const bool two = cnt > 8;  // groups of eight tokens
    for (int b = 0; b < LIMB_RING - 1; b++) issue(b, b);
    auto fetch = [&](int b) {  // the tokens' records of block b, by the first warp
      if (warp == 0 && b < nb) {
        const uint32_t at = (used + b) & 1u, bar = bar0 + 8 * at;
        if (lane == 0) umma::mbar_arrive_expect_tx(bar, (uint32_t)(cnt * LIMB_RECORD));
        __syncwarp();
        if (lane < cnt)
          asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(stages + at * LIMB_STAGE + lane * LIMB_TOKEN),
                       "l"(limbs + ((size_t)(t0 - first + lane) * nb + b) * LIMB_RECORD), "r"(LIMB_RECORD), "r"(bar)
                       : "memory");
      }
    };
    fetch(0), fetch(1);
    float acc[LIMB_RT][2][4], rest[LIMB_RT][2][4];  // [16 rows][group][rows g, g + 8 x tokens 2 t, 2 t + 1]: sum, and what its roundings left out
#pragma unroll
    for (int i = 0; i < 8 * LIMB_RT; i++) acc[i >> 3][(i >> 2) & 1][i & 3] = rest[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
    float lost[2 * LIMB_RT][2][2] = {};  // [row][group][token] marked blocks: unit of the first limb times |d|
    int slot = 0;
    for (int b = 0; b < nb; b++) {
      issue(b + LIMB_RING - 1, slot == 0 ? LIMB_RING - 1 : slot - 1);
      float two_to[2][2];  // what the tokens' first limbs count in
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int c = 0; c < 2; c++) two_to[j][c] = __ldg(ups + (size_t)(t0 - first + min(8 * j + 2 * t + c, cnt - 1)) * nb + b);
      cp_async_wait<LIMB_RING - 1>();
      const uint32_t at = (used + b) & 1u, xs = stages + at * LIMB_STAGE + g * LIMB_TOKEN;  // operand column g: token g of each group
      if (!umma::mbar_wait(bar0 + 8 * at, ((used + b) >> 1) & 1u, &abort_flag)) g_limb_status = 1;
      if (__syncthreads_or(abort_flag)) {  // (all warps, together) copies still in flight get some time to land before the CTA retires
        cp_async_wait<0>();
        __nanosleep(50000);
        return;
      }
      const uint32_t blk = ring + slot * LIMB_SLOT + g * LIMB_PITCH + ((skew0 + (uint32_t)b * 210u) & 15u);  // row g's block
      const uint32_t al = blk & ~3u, sh = (blk & 2u) * 8u;
      auto word = [&](int r, int at) {  // of row g + 8 r
        const uint32_t a = al + r * (8 * LIMB_PITCH) + at;
        return __funnelshift_r(lds32(a), lds32(a + 4), sh);
      };
      float top[LIMB_RT][2][4], low[LIMB_RT][2][4];  // scale x sub-block's sum: limb 2 (whole, and exact below 2^24), limbs 1 and 0 (in units of the latter)
#pragma unroll
      for (int i = 0; i < 8 * LIMB_RT; i++) top[i >> 3][(i >> 2) & 1][i & 3] = low[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
#pragma unroll 1
      for (int hu = 0; hu < 4; hu++) {  // half h of the block, elements 16 u .. of each of its four groups
        const int h = hu >> 1, u = hu & 1;
        uint32_t wa[2 * LIMB_RT], wc[2 * LIMB_RT], wh[2 * LIMB_RT], sc[2 * LIMB_RT];
#pragma unroll
        for (int r = 0; r < 2 * LIMB_RT; r++) {
          wa[r] = word(r, 64 * h + 16 * u + 4 * t), wc[r] = word(r, 64 * h + 32 + 16 * u + 4 * t), wh[r] = word(r, 128 + 32 * h + 16 * u + 4 * t);
          sc[r] = __byte_perm(word(r, 192 + 8 * h), word(r, 196 + 8 * h), u ? 0x7531 : 0x6420) ^ 0x80808080u;  // of the four groups, plus 128
        }
        const int first = (8 * h + u) * 4 + t;  // the record's place of sub-block 8 h + u; group q's is 8 q further
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint4 x01[2];
          uint2 x2[2];
#pragma unroll
          for (int j = 0; j < 2; j++) {
            if (j == 0 || two) {
              x01[j] = lds128(xs + j * (8 * LIMB_TOKEN) + 16 * (first + 8 * q)), x2[j] = lds64(xs + j * (8 * LIMB_TOKEN) + 1024 + 8 * (first + 8 * q));
            }
          }
#pragma unroll
          for (int rt = 0; rt < LIMB_RT; rt++) {
            uint32_t a[4];
            float f[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
              const int i = 2 * rt + r;
              const uint32_t nib = (q & 1 ? wc[i] : wa[i]) >> (q & 2 ? 4 : 0), bits = q == 0 ? wh[i] << 4 : q == 1 ? wh[i] << 2 : q == 2 ? wh[i] : wh[i] >> 2;
              const uint32_t code = and_or(nib, 0x0F0F0F0Fu, bits & 0x30303030u);  // code + 32
              const __half2 off = __float2half2_rn(-1056.f);
              auto f16 = [&](uint32_t bits) {
                const __half2 v = __hadd2(*reinterpret_cast<const __half2 *>(&bits), off);
                return *reinterpret_cast<const uint32_t *>(&v);
              };
              a[r] = f16(__byte_perm(code, 0x64646464u, 0x4140)), a[2 + r] = f16(__byte_perm(code, 0x64646464u, 0x4342));
              f[r] = __uint_as_float(__byte_perm(sc[i], 0x4B000000u, 0x7440 + q)) - 8388736.f;
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
              if (j == 0 || two) {
                float d0[4], d1[4], d2[4];
                mma_from_zero(d0, a, x01[j].x, x01[j].y);
                mma_from_zero(d1, a, x01[j].z, x01[j].w);
                mma_from_zero(d2, a, x2[j].x, x2[j].y);
#pragma unroll
                for (int c = 0; c < 4; c++)
                  top[rt][j][c] = fmaf(f[c >> 1], d2[c], top[rt][j][c]), low[rt][j][c] = fmaf(f[c >> 1], fmaf(2048.f, d1[c], d0[c]), low[rt][j][c]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 2 * LIMB_RT; r++) {
        uint16_t dh;
        asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(dh) : "r"(blk + r * (8 * LIMB_PITCH) + 208));
        const float d = f16_bits_to_f32(dh);
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int c = 0; c < 2; c++) {
            lost[r][j][c] = fmaf(fmaxf(-two_to[j][c], 0.f), fabsf(d), lost[r][j][c]);
            // acc + d 2^.. (top + 2^-27 low), the roundings of both products and of both sums kept (d 2^.. has eleven bits: exact)
            const int i = 2 * (r & 1) + c;
            float &y = acc[r >> 1][j][i];
            const float s = d * fabsf(two_to[j][c]), l = low[r >> 1][j][i] * 0x1p-27f, v = s * top[r >> 1][j][i], w = fmaf(s, l, v), t = y + w, z = t - y;
            rest[r >> 1][j][i] += ((y - (t - z)) + (w - z)) + (fmaf(s, l, v - w) + fmaf(s, top[r >> 1][j][i], -v));
            y = t;
          }
      }
      slot = slot + 1 == LIMB_RING ? 0 : slot + 1;
      __syncthreads();  // every warp is done with the stage, and with its own slot
      fetch(b + 2);
    }
    used += nb;
    cp_async_wait<0>();
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int mine = 8 * j + 2 * t + c;
        long long p = -1;
        if (mine < cnt) {
          p = pairs ? pairs[t0 + mine] : t0 + mine;
          if (p >= size_m) p = -1;
        }
        bool again[2 * LIMB_RT] = {};  // not a number, or too small beside what may be lost (of a row by itself: a row that two warps have comes out alike)
        if (p >= 0) {
          const float f = topkw ? topkw[p] : 1.f;
#pragma unroll
          for (int r = 0; r < 2 * LIMB_RT; r++) {
            const float y = acc[r >> 1][j][2 * (r & 1) + c] + rest[r >> 1][j][2 * (r & 1) + c];
            again[r] = !(fabsf(y) >= 0x1p-7f * lost[r][j][c]);
            out[p * N + r0 + g + 8 * r] = topkw ? y * f : y;
          }
        }
        unsigned odd[2 * LIMB_RT], left = 0;
#pragma unroll
        for (int r = 0; r < 2 * LIMB_RT; r++) odd[r] = __ballot_sync(0xffffffffu, again[r]), left |= odd[r];
        while (left) {  // those rows of a token once more, one after the other
          const int tt = (__ffs(left) - 1) & 3;
          left &= ~(0x11111111u << tt);  // (the lanes of that token: row g + 8 r is lane 4 g + tt's)
          const long long i = t0 + 8 * j + 2 * tt + c, q = pairs ? pairs[i] : i;
          const float4 *x = reinterpret_cast<const float4 *>(in + (size_t)(row_per_pair ? q : q / topk) * K) + lane;
          __syncwarp();  // (after the stores above)
          for (int r = 0; r < LIMB_ROWS; r++) {
            unsigned which = odd[0];
#pragma unroll
            for (int h = 1; h < 2 * LIMB_RT; h++) which = r >> 3 == h ? odd[h] : which;
            if (!(which >> (4 * (r & 7) + tt) & 1u)) continue;
            double sum = 0.;  // (in f32 one after the other they would be further off than limbs are where little is lost: 3.4e-7 at K = 11008)
            for (int b = 0; b < nb; b++) {
              float wv[8];
              q6k_eight(rows + r * row_bytes + (size_t)b * 210, lane, wv);
              const float4 u = __ldg(x + b * 64), v = __ldg(x + b * 64 + 32);
              const float xv[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
              for (int k = 0; k < 8; k++) sum = fma((double)wv[k], (double)xv[k], sum);
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float y = (float)sum;
            if (lane == 0) out[q * N + r0 + r] = topkw ? y * topkw[q] : y;
          }
        }
      }
  }
}

size_t q6k_limbs_bytes(long long M, int K) {
  const size_t records = (size_t)(M < LIMB_CHUNK ? M : LIMB_CHUNK) * (K >> 8);
  return records * LIMB_RECORD + ((records * 4 + 1023) & ~(size_t)1023);
}

// In memory of the call's own: these calls never shared the workspace, so that streams may have one each.  1: took the call; 0: no
// (or too little) scratch, or fewer rows than a warp's.
static int q6k_limbs(const float *in, const void *w, const int64_t *pairs, const int32_t *offsets, const float *topkw, float *out, long long M, long long size_m,
                     int E, int N, int K, int topk, int row_per_pair, void *scratch, size_t bytes, cudaStream_t st) {
  uint8_t *const ws = (uint8_t *)scratch;
  if (!ws || bytes < q6k_limbs_bytes(M, K) || N < LIMB_ROWS || ((uintptr_t)in & 15)) return 0;
  static DeviceOnce attr;
  const cudaError_t err = attr.ensure([] { return cudaFuncSetAttribute(q6k_limbs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LIMB_SMEM); });
  if (err != cudaSuccess) return fail((int)err, "light_b200: q6_k rows: %s", cudaGetErrorString(err));
  for (long long first = 0; first < M; first += LIMB_CHUNK) {
    const long long m = M - first < LIMB_CHUNK ? M - first : LIMB_CHUNK, records = m * (K >> 8);
    float *ups = (float *)(ws + (size_t)records * LIMB_RECORD);
    launch_early(x_limbs_kernel, dim3((unsigned)((records + 7) / 8)), dim3(256), st, in, pairs, ws, ups, first, m, K, topk, row_per_pair, size_m);
    if (int rc = launched("q6_k: activations to limbs")) return rc;
    const long long nb = (N + LIMB_ROWS * LIMB_WARPS - 1) / (LIMB_ROWS * LIMB_WARPS), passes = (m + LIMB_PASS - 1) / LIMB_PASS, want = (4ll * sm_count() + nb * E - 1) / (nb * E);
    const long long z = want < passes ? want : passes;  // CTAs that share an expert's tokens, where experts and rows alone do not fill the GPU
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nb, (unsigned)E, (unsigned)z), cfg.blockDim = dim3(LIMB_WARPS * 32), cfg.dynamicSmemBytes = LIMB_SMEM, cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at, cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, q6k_limbs_kernel, in, (const uint8_t *)w, (const uint8_t *)ws, (const float *)ups, pairs, offsets, topkw, out, first, m,
                                             size_m, E, N, K, topk, row_per_pair);
    if (e != cudaSuccess) return fail((int)e, "light_b200: q6_k rows: %s", cudaGetErrorString(e));
    if (int rc = launched("q6_k rows (limbs)")) return rc;
  }
  return 1;
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

int q6k_rows_dense(const float *x, const void *w, float *out, int M, int N, int K, void *scratch, size_t scratch_bytes, cudaStream_t st) {
  if (int took = q6k_limbs(x, w, nullptr, nullptr, nullptr, out, M, M, 1, N, K, 1, 1, scratch, scratch_bytes, st)) return took == 1 ? 0 : took;
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

int q6k_limbs_status() {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, g_limb_status, sizeof(int));
  return e == cudaSuccess ? v : -(int)e;
}

int moe_bad_ids_status() {
  unsigned int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_moe_bad_ids, sizeof(v));
  if (e != cudaSuccess) return fail((int)e, "light_b200: moe status: %s", cudaGetErrorString(e));
  return (int)v;
}

size_t moe_scratch_bytes(long long M, int K) {
  return gemm_tmem_sync_bytes() + (((size_t)M * K * 2 + 1023) & ~(size_t)1023) + (((size_t)M * 4 + 1023) & ~(size_t)1023) + gemm_tmem_parts_bytes();
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

int moe_gemm_q(const lb200_moe_args *a, int device, cudaStream_t st, void *scratch, size_t scratch_bytes) {
  int rc = prep(a, st);
  if (rc) return rc;
  if (int took = moe_umma(a, 1, nullptr, 0, 0, device, st)) return took == 1 ? 0 : took;
  // From as many pairs on as the tensor-core path takes of the other formats.
  if (a->dtype == LB200_Q6_K && a->M >= 256 && a->K % 256 == 0 && a->E <= 65535 && a->N > 0) {
    if (int took = q6k_limbs((const float *)a->input, a->weights, a->sorted_pairs, a->offsets, a->topk_weights, (float *)a->out, a->M, a->size_m, a->E, a->N, a->K, a->topk,
                             a->row_per_pair, scratch, scratch_bytes, st))
      return took == 1 ? 0 : took;
    return q6k_rows<true>((const float *)a->input, a->weights, a->sorted_pairs, a->offsets, a->topk_weights, (float *)a->out, a->M, a->size_m, a->E, a->N, a->K,
                       a->topk, a->row_per_pair, st);
  }
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
