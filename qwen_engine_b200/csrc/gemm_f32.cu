// The float32 product (see gemm_f32.cuh): every multiply-add is a float32 fma, two at a time (`fma.rn.f32x2`).
//
// Order of a sum, whatever M is: K is cut into S equal chunks (a function of N and K alone), a chunk is summed as two
// chains, one over its even and one over its odd k, the chunk's sum is even + odd, and the chunks are added in order.  So a
// row's bits do not depend on what else is in the batch, and the chains are 2 S times shorter than one over all of K.
//
// What bounds it: a few rows stream the weights, 4 bytes for each, and some hundreds of rows are bound by the float32
// multiply-adds.  Hence
//  - both operands go into shared memory as they lie (k fastest, rows padded to 36 floats: eight rows' 16-byte words are
//    conflict-free) by 16-byte cp.async, several k-blocks of 32 ahead; with at most 16 rows the weights' first blocks are
//    asked for before the wait for the kernel before;
//  - a thread keeps TM x TN pairs of sums and reads 4 k of a row in one load: the pair (k, k + 1) is the register pair that
//    the two-wide fma takes, so nothing is packed or duplicated;
//  - tiles are 64 weight rows, and a cluster of S CTAs shares K where the tiles alone would leave SMs idle; the partial
//    tiles meet through distributed shared memory, each CTA finishing a share of the outputs;
//  - the tile's height is the smallest of 4, 8, 16 that takes all rows, beyond that the one of 32, 48, 64 that wastes least.
// Measured on a B200, chains of launches over weights larger than L2: 4096 x 1024 at 3 rows 7.3 us (2.3 TB/s), 151936 x 1024 at
// 3 rows 186 us (3.3 TB/s), 6144 x 1024 at 141 rows 52 us (34 TFLOP/s).  Qwen3-0.6B in float32, 141 prompt tokens and four
// steps of three tokens: 164 ms with the kernel of gemm_generic.cu (scalar loads, a CTA's one chain over all of K), of which
// the products were 93 %; 17.8 ms with this one.
#include "gemm_f32.cuh"

#define GF_BN 64
#define GF_BK 32
#define GF_LD (GF_BK + 4)

__device__ __forceinline__ void gf_copy16(float* smem, const float* gmem, bool valid) {
  const int bytes = valid ? 16 : 0;                     // nothing is read for a place outside; the 16 bytes become zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
               :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gf_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}

template <int BM, int TM, int TN, int STAGES>
struct GfShape {
  static constexpr int MT = BM / TM, NT = GF_BN / TN, THREADS = MT * NT;
  static constexpr int LANES_M = MT >= 4 ? 4 : MT, LANES_N = 32 / LANES_M;      // a warp's threads over the tile
  static constexpr int STAGE = (GF_BN + BM) * GF_LD;                            // floats
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float);
  static_assert(THREADS % 32 == 0 && NT % LANES_N == 0 && MT % LANES_M == 0, "whole warps");
  static_assert((size_t)BM * GF_BN * sizeof(float) <= SMEM, "the partial tile takes the stages' place");
};

template <int BM, int TM, int TN, int STAGES>
__global__ void __launch_bounds__(GfShape<BM, TM, TN, STAGES>::THREADS)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                int M, int N, int K, int chunk, int splits, int act, int vec) {
  using S = GfShape<BM, TM, TN, STAGES>;
  constexpr bool EARLY = BM <= 16;
  extern __shared__ __align__(16) float gf_smem[];
  const int rank = blockIdx.x % splits;
  const int n0 = blockIdx.x / splits * GF_BN, m0 = blockIdx.y * BM;
  const int k_begin = min(K, rank * chunk), k_end = min(K, k_begin + chunk);
  const int blocks = (k_end - k_begin + GF_BK - 1) / GF_BK;
  constexpr int WORDS = GF_BK / 4;                      // 16-byte words of a row's k-block

  auto load_w = [&](int b) {
    float* ws = gf_smem + (b % STAGES) * S::STAGE;
#pragma unroll
    for (int e = threadIdx.x; e < GF_BN * WORDS; e += S::THREADS) {
      const int r = e / WORDS, k = k_begin + b * GF_BK + (e % WORDS) * 4;
      const bool ok = n0 + r < N && k < k_end;
      gf_copy16(ws + r * GF_LD + (e % WORDS) * 4, ok ? w + (size_t)(n0 + r) * K + k : w, ok);
    }
  };
  auto load_x = [&](int b) {
    float* xs = gf_smem + (b % STAGES) * S::STAGE + GF_BN * GF_LD;
#pragma unroll
    for (int e = threadIdx.x; e < BM * WORDS; e += S::THREADS) {
      const int r = e / WORDS, k = k_begin + b * GF_BK + (e % WORDS) * 4;
      const bool ok = m0 + r < M && k < k_end;
      gf_copy16(xs + r * GF_LD + (e % WORDS) * 4, ok ? x + (size_t)(m0 + r) * K + k : x, ok);
    }
  };

  pdl_launch_dependents();
  if (EARLY) {
#pragma unroll 1
    for (int b = 0; b < STAGES - 1; ++b) if (b < blocks) load_w(b);
  }
  pdl_wait();
#pragma unroll 1
  for (int b = 0; b < STAGES - 1; ++b) {
    if (b < blocks) {
      if (!EARLY) load_w(b);
      load_x(b);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tm = lane % S::LANES_M + S::LANES_M * (warp % (S::MT / S::LANES_M));
  const int tn = lane / S::LANES_M + S::LANES_N * (warp / (S::MT / S::LANES_M));
  unsigned long long acc[TM][TN];                       // (sum over even k, sum over odd k)
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;\n" :: "n"(STAGES - 2) : "memory");
    __syncthreads();                                    // block b has landed; block b - 1 is read no more
    if (b + STAGES - 1 < blocks) { load_w(b + STAGES - 1); load_x(b + STAGES - 1); }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* ws = gf_smem + (b % STAGES) * S::STAGE + tn * GF_LD;
    const float* xs = gf_smem + (b % STAGES) * S::STAGE + (GF_BN + tm) * GF_LD;
#pragma unroll
    for (int k = 0; k < GF_BK; k += 4) {
      ulonglong2 a[TM], c[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * S::MT * GF_LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) c[j] = *reinterpret_cast<const ulonglong2*>(ws + j * S::NT * GF_LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a[i].x, c[j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a[i].y, c[j].y);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // the CTA's partial tile [BM][64] in the stages' place
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const float even = __uint_as_float((unsigned)(acc[i][j] & 0xffffffffull)), odd = __uint_as_float((unsigned)(acc[i][j] >> 32));
      gf_smem[(tm + i * S::MT) * GF_BN + tn + j * S::NT] = even + odd;
    }
  if (splits > 1) cluster_sync_all(); else __syncthreads();
  for (int e = (rank * S::THREADS + threadIdx.x) * 4; e < BM * GF_BN; e += splits * S::THREADS * 4) {
    const int gm = m0 + e / GF_BN, gn = n0 + e % GF_BN;
    if (gm >= M || gn >= N) continue;
    float4 v;
    if (splits > 1) {
      v = cluster_ld_f32x4(cluster_map_shared(gf_smem + e, 0));
      for (int r = 1; r < splits; ++r) {
        const float4 p = cluster_ld_f32x4(cluster_map_shared(gf_smem + e, r));
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
      }
    } else {
      v = *reinterpret_cast<const float4*>(gf_smem + e);
    }
    if (act) { v.x = act_exact(v.x, act); v.y = act_exact(v.y, act); v.z = act_exact(v.z, act); v.w = act_exact(v.w, act); }
    float* o = out + (size_t)gm * N + gn;
    if (vec) {
      *reinterpret_cast<float4*>(o) = v;
    } else {
      o[0] = v.x;
      if (gn + 1 < N) o[1] = v.y;
      if (gn + 2 < N) o[2] = v.z;
      if (gn + 3 < N) o[3] = v.w;
    }
  }
  if (splits > 1) cluster_sync_all();                   // the other CTAs read this one's shared memory
}

template <int BM, int TM, int TN, int STAGES>
static int gf_launch(const float* x, const float* w, float* out, int M, int N, int K, int chunk, int splits, int act, cudaStream_t stream) {
  using S = GfShape<BM, TM, TN, STAGES>;
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_f32_kernel<BM, TM, TN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (configured != cudaSuccess) QE_REFUSE("linear: shared memory %d: %s", (int)S::SMEM, cudaGetErrorString(configured));
  const dim3 grid((N + GF_BN - 1) / GF_BN * splits, (M + BM - 1) / BM);
  const int vec = N % 4 == 0 && (uintptr_t)out % 16 == 0;
  if (splits > 1)
    qe_launch_cluster(gemm_f32_kernel<BM, TM, TN, STAGES>, grid, dim3(S::THREADS), S::SMEM, stream, (unsigned)splits, x, w, out, M, N, K, chunk, splits, act, vec);
  else
    qe_launch(gemm_f32_kernel<BM, TM, TN, STAGES>, grid, dim3(S::THREADS), S::SMEM, stream, x, w, out, M, N, K, chunk, splits, act, vec);
  QE_CHECK_LAUNCH("linear_f32");
  return 0;
}

int qe_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int act, cudaStream_t stream) {
  // K is shared by up to 8 CTAs as long as two rounds of CTAs for a tile of rows hold them and a share is at least 128
  const int tiles = (N + GF_BN - 1) / GF_BN;
  int splits = 1;
  while (splits < 8 && (long)tiles * splits * 2 <= 2 * 148 && K / (2 * splits) >= 128) splits *= 2;
  const int chunk = ((K + splits - 1) / splits + GF_BK - 1) / GF_BK * GF_BK;
  if (M <= 4) return gf_launch<4, 4, 1, 8>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (M <= 8) return gf_launch<8, 4, 1, 8>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (M <= 16) return gf_launch<16, 4, 2, 6>(x, w, out, M, N, K, chunk, splits, act, stream);
  // rows that the tiles cover, a tile's own cost counted as 8 more
  auto cost = [&](long bm) { return (M + bm - 1) / bm * (bm + 8); };
  if (M > 4096 || (cost(64) <= cost(48) && cost(64) <= cost(32))) return gf_launch<64, 8, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (cost(48) <= cost(32)) return gf_launch<48, 6, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  return gf_launch<32, 4, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
}
