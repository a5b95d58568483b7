// The float32 product (see gemm_f32.cuh): every multiply-add is a float32 fma, two at a time (`fma.rn.f32x2`).
//
// Order of a sum, whatever M is: K is cut into S equal chunks of whole runs (a function of N and K alone), a chunk into runs of 16 that
// are dealt to four groups in turn; a group's k are summed as two chains, the even and the odd ones, and even + odd, the
// groups and the chunks are added in order.  So a row's bits do not depend on
// what else is in the batch, and the chains are 8 S times shorter than one over all of K.
//
// What bounds it: a few rows stream the weights, 4 bytes for each, and some hundreds of rows are bound by the float32
// multiply-adds.  Hence
//  - both operands go into shared memory as they lie (k fastest, rows padded by four floats: eight rows' 16-byte words
//    are conflict-free) by 16-byte cp.async, several k-blocks ahead; with at most 16 rows the weights' first blocks are
//    asked for before the wait for the kernel before;
//  - a thread keeps TM x TN pairs of sums and reads 4 k of a row in one load: the pair (k, k + 1) is the register pair that
//    the two-wide fma takes, so nothing is packed or duplicated; up to 8 x 4 sums, since a 16-byte load from shared memory
//    costs four of its cycles even where lanes read the same word;
//  - in tiles of up to 16 rows the four groups are warps of their own, so that a tile has enough of them to hide its loads (a block is 64
//    k, a run of each); beyond, a thread takes one group after the other (a block is two runs of a group);
//  - tiles are 64 weight rows, and a cluster of S CTAs shares K where the tiles alone would leave SMs idle; the partial
//    tiles meet through distributed shared memory, each CTA finishing a share of the outputs;
//  - the tile's height is the smallest of 4, 8, 16 that takes all rows, beyond that the one of 32, 48, 64 that wastes least (K up
//    to 64: 16 or 48).
// Measured on a B200, chains of launches over weights larger than L2: 4096 x 1024 at 3 rows 5.5 us (3.1 TB/s), 151936 x 1024
// at 3 rows 99 us (6.3 TB/s), 6144 x 1024 at 141 rows 57 us (31 TFLOP/s).  With two threads' worth of k in one group and
// four rows of one column a thread, 3 rows took 7.3 and 186 us; 8 x 8 sums a thread from 32 rows on (8 warps an SM instead
// of 12) took 74 us at 141 rows.  Qwen3-0.6B in float32, 141 prompt tokens and four steps of three tokens: 164 ms with
// the kernel of gemm_generic.cu (scalar loads, a CTA's one chain over all of K), of which the products were 93 %; 11.9 ms
// with this one and the attention kernel of attention_generic.cu as it is now (5.1 of those 164 ms were saved there).
#include "gemm_f32.cuh"

#define GF_BN 64
#define GF_GROUPS 4
#define GF_RUN 16                     // consecutive k of a group

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
  static constexpr bool SLICED = BM <= 16;                                      // the groups are warps of their own
  static constexpr int MT = BM / TM, NT = GF_BN / TN, GROUP = MT * NT, THREADS = SLICED ? GF_GROUPS * GROUP : GROUP;
  static constexpr int LANES_M = MT >= 4 ? 4 : MT, LANES_N = 32 / LANES_M;      // a warp's threads over the tile
  static constexpr int CTAS = BM == 64 ? 2 : 3;                                 // an SM's registers hold at least
  static constexpr int BK = SLICED ? GF_GROUPS * GF_RUN : 2 * GF_RUN;           // k of a loaded block
  static constexpr int LD = BK + 4;
  static constexpr int STAGE = (GF_BN + BM) * LD;                            // floats
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float);
  static_assert(GROUP % 32 == 0 && NT % LANES_N == 0 && MT % LANES_M == 0, "whole warps");
  static_assert((size_t)(SLICED ? GF_GROUPS : 1) * BM * GF_BN * sizeof(float) <= SMEM, "the groups' partial tiles take the stages' place");
};

// TAIL: runs behind the share's end are neither loaded nor summed (a group's blocks hold two runs each).
template <int BM, int TM, int TN, int STAGES, bool TAIL>
__global__ void __launch_bounds__(GfShape<BM, TM, TN, STAGES>::THREADS, GfShape<BM, TM, TN, STAGES>::CTAS)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                int M, int N, int K, int chunk, int splits, int act, int vec) {
  using S = GfShape<BM, TM, TN, STAGES>;
  constexpr bool EARLY = S::SLICED;
  extern __shared__ __align__(16) float gf_smem[];
  const int rank = blockIdx.x % splits;
  const int n0 = blockIdx.x / splits * GF_BN, m0 = blockIdx.y * BM;
  const int k_begin = min(K, rank * chunk), k_end = min(K, k_begin + chunk);
  // blocks to load: of a run of each group; or, where a thread takes the groups in turn, `turn` of two runs for each
  const int rounds = (k_end - k_begin + GF_GROUPS * GF_RUN - 1) / (GF_GROUPS * GF_RUN);
  const int turn = (rounds + 1) / 2;
  const int groups = TAIL && rounds == 1 ? (k_end - k_begin + GF_RUN - 1) / GF_RUN : GF_GROUPS;     // that have any k
  const int blocks = S::SLICED ? rounds : turn * groups;
  constexpr int LD = S::LD, WORDS = S::BK / 4;                      // 16-byte words of a row's k-block
  static_assert(S::THREADS % WORDS == 0, "a thread's words are the same one of every row");
  const int word = threadIdx.x % WORDS, row = threadIdx.x / WORDS;
  const int word_k = S::SLICED ? word * 4 : word / (GF_RUN / 4) * (GF_GROUPS * GF_RUN) + word % (GF_RUN / 4) * 4;
  const int k_in_run = word_k % GF_RUN;
  auto k_of = [&](int b) {                              // the k of this thread's word of block b
    if (S::SLICED) return k_begin + b * S::BK + word_k;
    const int group = b / turn;
    return k_begin + (b - group * turn) * (2 * GF_GROUPS * GF_RUN) + group * GF_RUN + word_k;
  };
  auto load_w = [&](int b) {
    float* ws = gf_smem + (b % STAGES) * S::STAGE + word * 4;
    const int k = k_of(b);
    if (TAIL && k - k_in_run >= k_end) return;
#pragma unroll
    for (int r = row; r < GF_BN; r += S::THREADS / WORDS) {
      const bool ok = n0 + r < N && k < k_end;
      gf_copy16(ws + r * LD, ok ? w + (size_t)(n0 + r) * K + k : w, ok);
    }
  };
  auto load_x = [&](int b) {
    float* xs = gf_smem + (b % STAGES) * S::STAGE + GF_BN * LD + word * 4;
    const int k = k_of(b);
    if (TAIL && k - k_in_run >= k_end) return;
#pragma unroll
    for (int r = row; r < BM; r += S::THREADS / WORDS) {
      const bool ok = m0 + r < M && k < k_end;
      gf_copy16(xs + r * LD, ok ? x + (size_t)(m0 + r) * K + k : x, ok);
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

  const int lane = threadIdx.x & 31, group = threadIdx.x / S::GROUP, warp = threadIdx.x % S::GROUP >> 5;
  const int tm = lane % S::LANES_M + S::LANES_M * (warp % (S::MT / S::LANES_M));
  const int tn = lane / S::LANES_M + S::LANES_N * (warp / (S::MT / S::LANES_M));
  unsigned long long acc[TM][TN];                       // (sum over even k, sum over odd k)
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  float total[TM][TN];                                  // the groups before
  auto even_and_odd = [&](int i, int j) {
    return __uint_as_float((unsigned)(acc[i][j] & 0xffffffffull)) + __uint_as_float((unsigned)(acc[i][j] >> 32));
  };

  const int offset = S::SLICED ? group * GF_RUN : 0;
  int left = turn;                                      // blocks of the group in turn
  int k_run = k_begin + offset;                         // where this block's (first) run starts
  int k_next = k_begin + GF_RUN;                        // ... and the first of the group after the one in turn
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;\n" :: "n"(STAGES - 2) : "memory");
    __syncthreads();                                    // block b has landed; block b - 1 is read no more
    if (b + STAGES - 1 < blocks) { load_w(b + STAGES - 1); load_x(b + STAGES - 1); }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* ws = gf_smem + (b % STAGES) * S::STAGE + tn * LD + offset;
    const float* xs = gf_smem + (b % STAGES) * S::STAGE + (GF_BN + tm) * LD + offset;
#pragma unroll
    for (int run = 0; run < S::BK / (S::SLICED ? GF_GROUPS * GF_RUN : GF_RUN); ++run) {
      if (TAIL && k_run + run * (GF_GROUPS * GF_RUN) >= k_end) break;     // uniform within the group
#pragma unroll
      for (int k = run * GF_RUN; k < (run + 1) * GF_RUN; k += 4) {
        ulonglong2 a[TM], c[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * S::MT * LD + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) c[j] = *reinterpret_cast<const ulonglong2*>(ws + j * S::NT * LD + k);
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
    k_run += S::BK / GF_RUN * (S::SLICED ? GF_RUN : GF_GROUPS * GF_RUN);
    if (!S::SLICED && --left == 0) {
      left = turn;
      k_run = k_next;
      k_next += GF_RUN;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          total[i][j] = b < turn ? even_and_odd(i, j) : total[i][j] + even_and_odd(i, j);
          acc[i][j] = 0ull;
        }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // the CTA's partial tile [BM][64] in the stages' place (the groups' four, added into the first)
  constexpr int TILE = BM * GF_BN;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      gf_smem[(S::SLICED ? group * TILE : 0) + (tm + i * S::MT) * GF_BN + tn + j * S::NT] = S::SLICED || blocks == 0 ? even_and_odd(i, j) : total[i][j];
  if (S::SLICED) {
    __syncthreads();
    for (int e = threadIdx.x * 4; e < TILE; e += S::THREADS * 4) {
      float4 v = *reinterpret_cast<const float4*>(gf_smem + e);
#pragma unroll
      for (int g = 1; g < GF_GROUPS; ++g) {
        const float4 p = *reinterpret_cast<const float4*>(gf_smem + g * TILE + e);
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
      }
      *reinterpret_cast<float4*>(gf_smem + e) = v;
    }
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

template <int BM, int TM, int TN, int STAGES, bool TAIL = false>
static int gf_launch(const float* x, const float* w, float* out, int M, int N, int K, int chunk, int splits, int act, cudaStream_t stream) {
  using S = GfShape<BM, TM, TN, STAGES>;
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_f32_kernel<BM, TM, TN, STAGES, TAIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (configured != cudaSuccess) QE_REFUSE("linear: shared memory %d: %s", (int)S::SMEM, cudaGetErrorString(configured));
  const dim3 grid((N + GF_BN - 1) / GF_BN * splits, (M + BM - 1) / BM);
  const int vec = N % 4 == 0 && (uintptr_t)out % 16 == 0;
  if (splits > 1)
    qe_launch_cluster(gemm_f32_kernel<BM, TM, TN, STAGES, TAIL>, grid, dim3(S::THREADS), S::SMEM, stream, (unsigned)splits, x, w, out, M, N, K, chunk, splits, act, vec);
  else
    qe_launch(gemm_f32_kernel<BM, TM, TN, STAGES, TAIL>, grid, dim3(S::THREADS), S::SMEM, stream, x, w, out, M, N, K, chunk, splits, act, vec);
  QE_CHECK_LAUNCH("linear_f32");
  return 0;
}

int qe_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int act, cudaStream_t stream) {
  // K is shared by up to 8 CTAs as long as two rounds of CTAs for a tile of rows hold them and a share is at least 128
  const int tiles = (N + GF_BN - 1) / GF_BN;
  int splits = 1;
  while (splits < 8 && (long)tiles * splits * 2 <= 2 * 148 && K / (2 * splits) >= 128) splits *= 2;
  const int chunk = ((K + splits - 1) / splits + GF_RUN - 1) / GF_RUN * GF_RUN;
  if (M <= 4) return gf_launch<4, 4, 2, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (M <= 8) return gf_launch<8, 8, 2, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (M <= 16) return gf_launch<16, 8, 4, 3>(x, w, out, M, N, K, chunk, splits, act, stream);
  // One run of each group at most: the tiles with two runs a block are mostly padding.  The groups' own warps do better up to some
  // rounds of CTAs, then 48 rows a tile (1 024 x 64 at 256 rows 8.5 -> 3.4 us, at 2 048 20.4 -> 14.5; the kernel of gemm_generic.cu
  // 6.3 and 16.3).
  if (K <= GF_GROUPS * GF_RUN) {
    if ((long)M * N <= 1 << 20 && M <= 1 << 16) return gf_launch<16, 8, 4, 3>(x, w, out, M, N, K, chunk, splits, act, stream);
    if (M <= 48 * 65535) return gf_launch<48, 6, 4, 4, true>(x, w, out, M, N, K, chunk, splits, act, stream);
    return gf_launch<64, 8, 4, 4, true>(x, w, out, M, N, K, chunk, splits, act, stream);
  }
  // rows that the tiles cover, a tile's own cost counted as 8 more
  auto cost = [&](long bm) { return (M + bm - 1) / bm * (bm + 8); };
  const int bm = M > 4096 || (cost(64) <= cost(48) && cost(64) <= cost(32)) ? 64 : cost(48) <= cost(32) ? 48 : 32;
  // runs behind the share's end are left out where they are a fifth of the work and more (1 024 x 1 056 at 2 048 rows, shares of 144:
  // 276 -> 209 us, 227 with the kernel of gemm_generic.cu; where they are less, asking costs as much)
  const int rounds = (chunk + 2 * GF_GROUPS * GF_RUN - 1) / (2 * GF_GROUPS * GF_RUN);
  if (rounds * 2 * GF_GROUPS * GF_RUN * 4 >= chunk * 5) {
    if (bm == 64) return gf_launch<64, 8, 4, 4, true>(x, w, out, M, N, K, chunk, splits, act, stream);
    if (bm == 48) return gf_launch<48, 6, 4, 4, true>(x, w, out, M, N, K, chunk, splits, act, stream);
    return gf_launch<32, 4, 4, 4, true>(x, w, out, M, N, K, chunk, splits, act, stream);
  }
  if (bm == 64) return gf_launch<64, 8, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  if (bm == 48) return gf_launch<48, 6, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
  return gf_launch<32, 4, 4, 4>(x, w, out, M, N, K, chunk, splits, act, stream);
}
