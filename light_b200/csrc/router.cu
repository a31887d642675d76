// Router logits of a sparse block: x (T, K) bf16 or f32 times W (E, K) f32, f32 arithmetic in effect, on the tensor cores.
//
// What bounds it.  As f32 multiply-adds 4096 tokens by 256 experts of 7168 are 7.5 G of them, 200 us at the f32 rate and 305 as the library's matmul runs
// them (65 more for the tokens in f32).  Here every f32 operand is the sum of three bf16 values (8 + 8 + 8 bits, each the rounding of what the ones before
// left; a bf16 activation is one as it is) whose products are exact, and their sums go through mma.sync: three MMAs a step for bf16 activations, the six
// largest products for f32 ones (what is left out is below 2^-26 of a product).  The tensor core's own sum is kept to 32 k, smallest terms first, and added to the
// running sum in f32.  The error against 64 bits is a fifth to two thirds of the library's f32 matmul (K = 1024 to 7168).  Splitting the weights takes about
// as many issue slots as the MMAs take clocks, and both are re-read for every 64 tokens.
//   us, the library (with the pass to f32 for bf16) / here:  bf16 4096 x 256 x 7168 369 / 212, 1024 x 128 x 4096 79 / 26, 32 x 256 x 7168 53 / 12.9, 8 x 256 x 7168
//   22.3 / 11.4;  f32 77 x 128 x 2048 20.3 / 7.3, 300 x 200 x 3072 59 / 24, 2048 x 64 x 2048 38 / 20, 1024 x 256 x 4096 76 / 59, 4096 x 128 x 4096 119 / 114, but 3000 x
//   200 x 1536 69 / 80, 4096 x 256 x 4096 170 / 214: which calls of a sparse block come here is nn.py's choice.
//
// A CTA holds a tile of BM tokens x BN experts and a share of K; the CTAs of a cluster hold the others and add up through each other's shared memory, in their
// order.  A sum that is not finite (an infinity times the zero rest of another operand is no number) is made again by multiply-adds.
#include <cuda_bf16.h>

#include "common.cuh"
#include "mma_sync.cuh"
#include "umma.cuh"

namespace lb {
namespace {

constexpr int RT_KC = 32, RT_THREADS = 128;
constexpr int RT_PITCH32 = 160, RT_PITCH16 = 80;  // bytes of a staged row of 32 f32 / bf16: an operand's reads meet every bank once

// Operands are split 2^24 times as large as they are, so that the last bit of the smallest f32 (2^-149) still has its place in a normal bf16; as they are, operands
// below 2^-109 lost theirs (w of 2^-120: 2e-5 of an output).  What leaves f32's range that way is not finite, and made again.
constexpr float SPLIT_UP = 0x1p24f;

struct RouterArgs {
  const void *x;
  const float *w;
  float *out;
  int T, E, K;
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two f32 times SPLIT_UP as three pairs of bf16 each, largest first (sm_100 multiplies and adds two f32 with one instruction)
__device__ __forceinline__ void split3(uint2 v, uint32_t (&p)[3]) {
  uint64_t ab;
  asm("{\n\t.reg .b64 x, up;\n\tmov.b64 x, {%1, %2};\n\tmov.b64 up, {%3, %3};\n\tmul.rn.f32x2 %0, x, up;\n\t}\n" : "=l"(ab) : "r"(v.x), "r"(v.y), "f"(SPLIT_UP));
#pragma unroll
  for (int i = 0; i < 3; i++) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(ab));
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    p[i] = *reinterpret_cast<const uint32_t *>(&h);
    if (i < 2)  // what is left: exact
      asm("{\n\t.reg .b64 h, m;\n\tmov.b64 h, {%1, %2};\n\tmov.b64 m, {%3, %3};\n\tfma.rn.f32x2 %0, h, m, %0;\n\t}\n" : "+l"(ab) : "r"(p[i] << 16), "r"(p[i] & 0xFFFF0000u), "f"(-1.f));
  }
}

template <typename XT, int WM, int MI, int NI, int STAGES>  // warps along the tokens, MMA tiles of 16 tokens and of 8 experts to a warp; chunks on their way
__global__ void __launch_bounds__(RT_THREADS, STAGES == 3 ? 4 : 3) router_kernel(const __grid_constant__ RouterArgs a) {
  constexpr bool F32 = sizeof(XT) == 4;
  constexpr int WN = 4 / WM, BM = 16 * MI * WM, BN = 8 * NI * WN, XP = F32 ? RT_PITCH32 : RT_PITCH16, STAGE = BM * XP + BN * RT_PITCH32;
  constexpr int XA = F32 ? 3 : 1;
  extern __shared__ __align__(16) unsigned char mem[];
  const uint32_t base = umma::smem_u32(mem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, wm = warp % WM, wn = warp / WM;
  const int ranks = gridDim.z, rank = blockIdx.z;  // (the cluster is the whole z of the grid)
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, chunks = (a.K + RT_KC - 1) / RT_KC;
  const int c0 = chunks * rank / ranks, c1 = chunks * (rank + 1) / ranks;
  pdl_launch_dependents();
  auto fetch = [&](int c, bool weights) {  // chunk c of the operand; rows past the end are the last one's again
    const uint32_t to = base + (c - c0) % STAGES * STAGE + (weights ? BM * XP : 0);
    const int rows = weights ? BN : BM, per = weights || F32 ? 8 : 4, each = weights || F32 ? 4 : 8, k0 = c * RT_KC;
    for (int i = threadIdx.x; i < rows * per; i += RT_THREADS) {
      const int r = i / per, q = i - r * per, k = k0 + q * each;
      const void *src = weights ? (const void *)(a.w + (size_t)min(n0 + r, a.E - 1) * a.K + k) : (const void *)((const XT *)a.x + (size_t)min(m0 + r, a.T - 1) * a.K + k);
      const uint32_t dst = to + r * (weights ? RT_PITCH32 : XP) + 16 * q;
      if (k < a.K) cp_async16(dst, src);  // (K is whole granules)
      else asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};\n" ::"r"(dst), "r"(0u) : "memory");
    }
  };
  pdl_wait();  // (the weights too may be the kernel before's)
  for (int s = 0; s < STAGES - 1; s++) {
    if (c0 + s < c1) fetch(c0 + s, true), fetch(c0 + s, false);
    cp_async_commit();
  }
  float acc[MI][NI][4];
#pragma unroll
  for (int i = 0; i < MI * NI * 4; i++) acc[i / (4 * NI)][i / 4 % NI][i % 4] = 0.f;
  for (int c = c0; c < c1; c++) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();  // the chunk is there, and everybody has left the stage that the next one overwrites
    if (c + STAGES - 1 < c1) fetch(c + STAGES - 1, true), fetch(c + STAGES - 1, false);
    cp_async_commit();
    const uint32_t xs = base + (c - c0) % STAGES * STAGE + (wm * 16 * MI + g) * XP, ws = base + (c - c0) % STAGES * STAGE + BM * XP + (wn * 8 * NI + g) * RT_PITCH32 + 8 * t;
    float d[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI * NI * 4; i++) d[i / (4 * NI)][i / 4 % NI][i % 4] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
      uint32_t xa[MI][XA][4];
#pragma unroll
      for (int i = 0; i < MI; i++)
#pragma unroll
        for (int r = 0; r < 4; r++) {  // rows g, g + 8; k 2 t .. and 8 + 2 t ..
          const uint32_t at = xs + (16 * i + 8 * (r & 1)) * XP;
          if constexpr (F32) {
            uint32_t p[3];
            split3(lds64(at + 64 * kk + 32 * (r >> 1) + 8 * t), p);
            xa[i][0][r] = p[0], xa[i][1][r] = p[1], xa[i][2][r] = p[2];
          } else {
            xa[i][0][r] = lds32(at + 32 * kk + 16 * (r >> 1) + 4 * t);
          }
        }
      uint32_t wb[NI][2][3];
#pragma unroll
      for (int j = 0; j < NI; j++) split3(lds64(ws + 8 * j * RT_PITCH32 + 64 * kk), wb[j][0]), split3(lds64(ws + 8 * j * RT_PITCH32 + 64 * kk + 32), wb[j][1]);
      auto products = [&](int px, int pw) {  // of two parts, for all tiles: one after the other they would wait for each other's sums
#pragma unroll
        for (int j = 0; j < NI; j++)
#pragma unroll
          for (int i = 0; i < MI; i++) mma_bf16(d[i][j], xa[i][px], wb[j][0][pw], wb[j][1][pw]);
      };
      if constexpr (F32) products(2, 0), products(1, 1), products(0, 2), products(1, 0);
      else products(0, 2);
      products(0, 1), products(0, 0);
    }
#pragma unroll
    for (int i = 0; i < MI * NI * 4; i++) acc[i / (4 * NI)][i / 4 % NI][i % 4] += d[i / (4 * NI)][i / 4 % NI][i % 4];
  }
  cp_async_wait<0>();
  __syncthreads();
  // [BM][BN] sums of this share, then row r of the tile is added up by rank r % ranks
  float *const tile = reinterpret_cast<float *>(mem);
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < NI; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) tile[((wm * MI + i) * 16 + g + 8 * (q >> 1)) * (BN + 4) + (wn * NI + j) * 8 + 2 * t + (q & 1)] = acc[i][j][q];
  if (ranks > 1) umma::cluster_sync();
  else __syncthreads();
  for (int i = threadIdx.x; i < BM / ranks * BN; i += RT_THREADS) {
    const int r = i / BN * ranks + rank, n = i % BN;
    const uint32_t at = base + (uint32_t)(r * (BN + 4) + n) * 4;
    float v = 0.f;
    if (ranks == 1) v = tile[r * (BN + 4) + n];
    else
      for (int z = 0; z < ranks; z++) v += umma::ld_cluster_f32(umma::map_to_rank(at, z));
    const int m = m0 + r, e = n0 + n;
    if (m >= a.T || e >= a.E) continue;
    if (!(fabsf(v) < INFINITY)) {
      const XT *x = (const XT *)a.x + (size_t)m * a.K;
      const float *w = a.w + (size_t)e * a.K;
      v = 0.f;
      for (int k = 0; k < a.K; k++) v = fmaf(ld_act(x, k), w[k], v);
    } else {
      v *= F32 ? 1.f / (SPLIT_UP * SPLIT_UP) : 1.f / SPLIT_UP;
    }
    a.out[(size_t)m * a.E + e] = v;
  }
  if (ranks > 1) umma::cluster_sync();  // nobody leaves while its sums may still be read
}

template <typename XT, int WM, int MI, int NI, int STAGES = 4>
int go(const RouterArgs &a, cudaStream_t st) {
  constexpr int BM = 16 * MI * WM, BN = 8 * NI * (4 / WM), SMEM = STAGES * (BM * (sizeof(XT) == 4 ? RT_PITCH32 : RT_PITCH16) + BN * RT_PITCH32);
  static_assert(SMEM >= BM * (BN + 4) * 4 && BM % 8 == 0, "the sums take the stages' place");
  auto kern = router_kernel<XT, WM, MI, NI, STAGES>;
  static DeviceOnce attr;
  cudaError_t e = attr.ensure([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); });
  if (e != cudaSuccess) return fail((int)e, "light_b200: router_logits: %s", cudaGetErrorString(e));
  const long long tiles = (long long)((a.T + BM - 1) / BM) * ((a.E + BN - 1) / BN);
  int ranks = 1;  // shares of K: until there are two CTAs to an SM, of eight chunks or more
  while (ranks < 8 && tiles * ranks < 2 * sm_count() && a.K >= 2 * ranks * 8 * RT_KC) ranks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((a.E + BN - 1) / BN), (unsigned)((a.T + BM - 1) / BM), (unsigned)ranks);
  cfg.blockDim = dim3(RT_THREADS), cfg.dynamicSmemBytes = SMEM, cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = (unsigned)ranks;
  cfg.attrs = at, cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e != cudaSuccess) return fail((int)e, "light_b200: router_logits: %s", cudaGetErrorString(e));
  return launched("router_logits");
}

}  // namespace

// Tiles of 16 tokens by 32 experts while they take no more than 512 CTAs with their shares of K (about as many as the GPU holds of them at once), of 64 by 64
// beyond.  us, 64 x 64 / 16 x 32 (tokens x experts x K):  f32 17 x 64 x 256 12.6 / 5.2, 77 x 128 x 2048 12.7 / 7.3, 256 x 256 x 512 15.8 / 7.6, 512 x 8 x 4096 21.4 /
// 15.0, 1024 x 64 x 1024 13.8 / 13.6;  bf16 32 x 256 x 7168 23.7 / 12.9, 64 x 256 x 7168 23.9 / 15.4, 512 x 64 x 2048 9.9 / 8.5;  but f32 512 x 64 x 4096 21.8 / 23.3, 256 x 256 x
// 2048 17.7 / 23.6, bf16 700 x 64 x 2048 11.0 / 11.9, 1024 x 256 x 2048 27.0 / 48.0.  (64 x 64 from 17 tokens on took longer than the library's matmul where K is
// short: f32 17 x 64 x 256 12.6, the library 7.1.)
int router_logits(const void *x, int dtype, const float *w, float *out, int T, int E, int K, cudaStream_t st) {
  if (T == 0 || E == 0) return 0;
  const RouterArgs a{x, w, out, T, E, K};
  const long long narrow = ((long long)T + 15) / 16 * ((E + 31) / 32);
  if (narrow * (K < 2048 ? K : 2048) <= 64 * 2048) return dtype == LB200_F32 ? go<float, 1, 1, 1>(a, st) : go<__nv_bfloat16, 1, 1, 1>(a, st);
  if (dtype == LB200_F32) return go<float, 2, 2, 4>(a, st);
  // Where the tiles fill the GPU, four CTAs of three chunks each to an SM (4096 x 256 x 7168: 226 -> 203 us), else three of four (1024 x 128 x 4096: 31.7 ->
  // 26.6): with a CTA or two to an SM the chunks on their way are what hides the latency.
  if ((long long)((T + 63) / 64) * ((E + 63) / 64) >= sm_count()) return go<__nv_bfloat16, 2, 2, 4, 3>(a, st);
  return go<__nv_bfloat16, 2, 2, 4>(a, st);
}

}  // namespace lb
