// out[M, N] (+)= x[M, K] · w[N, K]^T in bfloat16 for up to 64 rows when the weight rows alone are too
// few to give every SM a CTA (the output and down projections of a decode step of many requests:
// N = hidden size): a cluster of S CTAs shares a tile of 64 or 128 weight rows, and each CTA of the
// cluster takes one share of K.  (Same contract as the reference's linear, src/layers/ops/linear.py:101-122.)
//
// As in gemm_tcgen05_swap.cu the weights take the 128-row side of tcgen05.mma and the tokens its narrow
// side, a CTA streams its weights once through a TMA ring, and the accumulator lies in tensor memory.
// The partial sums then meet on chip: every CTA puts its partial tile into its own shared
// memory, the cluster meets at a barrier, and CTA r adds up, for the tokens r, r + S, ..., the S
// partial tiles through distributed shared memory, always in the order of the shares (so the result
// does not depend on timing), and writes those tokens' outputs.  A second barrier keeps every CTA's
// shared memory alive until its neighbours have read it.
//
// RESID: out is the float32 residual stream and the product is added to it (every element is read
// and written by exactly one thread).
//
// What bounds it: the walk of a CTA over its share of K, 0.27 us for a stage of 128 k (the issuing warp's waits and
// instructions, not the bytes; 64 k a stage took 0.23), then about 2 us until the sums have met.  So a stage is 128 k,
// and up to 32 tokens clusters of 2 and 4 take tiles of 64 rows (twice the CTAs, with a ring small enough for two per SM).
// Measured on a B200, a chain of launches, 28 rows, against tiles of 128 rows and stages of 64 k: 2 560 x 9 728 in clusters
// of 4 14.7 -> 12.1 us, 2 048 x 6 144 10.0 -> 7.7, 6 144 x 2 560 in clusters of 2 10.0 -> 8.6.  Clusters of 8 gained in a
// chain with tiles of 64 rows too (1 024 x 3 072 5.2 -> 4.2) but not in the step (a prompt of 23 tokens 0.4 % slower).
//
// Six warps: warp 0 feeds TMA, warp 1 owns tensor memory and issues the MMAs, warps 2-5 read the
// accumulator (lane = weight row; the 64-row form keeps row r in lane r mod 16 of the quarter r / 16; column = token) and do
// the sum.  Every wait on an mbarrier is bounded,
// as in gemm_tcgen05.cu; a CTA whose wait ran out still takes part in both cluster barriers, so that
// its neighbours return; qe_gemm_tc_splitk_status() reads this kernel's flag.
//
// Needs K % 8 == 0, N % 4 == 0 and 16-byte aligned bases; the launcher refuses the rest.
#include "tcgen05.cuh"

#define SK_HALF 64              // k of a box (128 bytes: the swizzle's width)
#define SK_BK (2 * SK_HALF)     // k of a stage: two boxes of each operand
#define SK_MAX_M 64             // tokens at most
#define SK_THREADS 192

static __device__ int g_tc_status = 0;      // 0 = fine; else code of the first wait that ran out

template <int BM, int BT, int STAGES>    // BM: weight rows per cluster; BT: tokens at most (rows of the token operand's box)
struct __align__(1024) SkSmem {
  __nv_bfloat16 w[STAGES][2][BM * SK_HALF];
  __nv_bfloat16 x[STAGES][2][BT * SK_HALF];
  float part[BT][BM];                           // this CTA's partial sums, [token][weight row]
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

template <typename TOut, int S, int BM, int BT, int STAGES, bool RESID>
__global__ void __launch_bounds__(SK_THREADS)
gemm_tcgen05_splitk_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                           TOut* __restrict__ out, int M, int N, int K, int act) {
  extern __shared__ unsigned char smem_raw[];
  using Smem = SkSmem<BM, BT, STAGES>;
  constexpr uint32_t TMEM_COLS = BT < 32 ? 32 : BT;
  pdl_launch_dependents();
  // the same offset in every CTA of the cluster: the dynamic shared memory starts at the same address
  Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_cta_rank();           // this CTA's share of K
  const int n0 = (blockIdx.x / S) * BM;
  const int num_kb = (K + SK_BK - 1) / SK_BK;
  const int per = (num_kb + S - 1) / S;
  const int kb0 = min(num_kb, rank * per), kb1 = min(num_kb, kb0 + per);
  const int n_kb = kb1 - kb0;
  const int mt = (M + 15) / 16 * 16;                  // tokens as the instruction sees them
  volatile int* abort_flag = &sm.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    mbar_init(&sm.acc_full, 1);
    sm.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tc_alloc(&sm.tmem_base, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ---- producer: the weights are nobody's output, so the ring is filled before the wait for the
    // kernel that produces x; the token operand of those k-blocks follows after the wait ----------
    if (lane == 0) {
      auto load_w = [&](int i) {
        const int s = i % STAGES;
        mbar_expect_tx(&sm.full[s], (BM + BT) * SK_BK * sizeof(__nv_bfloat16));
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_2d(sm.w[s][h], &map_w, &sm.full[s], (kb0 + i) * SK_BK + h * SK_HALF, n0);   // (behind K: zeros)
      };
      auto load_x = [&](int i) {
        const int s = i % STAGES;
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_2d(sm.x[s][h], &map_x, &sm.full[s], (kb0 + i) * SK_BK + h * SK_HALF, 0);
      };
      const int ahead = min(n_kb, STAGES);
      for (int i = 0; i < ahead; ++i) load_w(i);
      pdl_wait();
      for (int i = 0; i < ahead; ++i) load_x(i);
      int issued = ahead;
      for (int i = ahead; i < n_kb; ++i) {
        const int s = i % STAGES;
        if (!mbar_wait(&sm.empty[s], ((i / STAGES) - 1) & 1, abort_flag, 21, &g_tc_status)) break;
        load_w(i);
        load_x(i);
        ++issued;
      }
      if (*abort_flag) {
        for (int i = max(0, issued - STAGES); i < issued; ++i)
          for (uint32_t spin = 0; spin < TC_WAIT_LIMIT; ++spin)
            if (mbar_try_wait(&sm.full[i % STAGES], (i / STAGES) & 1)) break;
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer -------------------------------------------------------------------------------
    if (n_kb > 0) {                                   // (the whole warp: one lane is elected per instruction)
      const uint32_t idesc = make_idesc(BM, mt);
      bool ok = true;
      for (int i = 0; i < n_kb && ok; ++i) {
        const int s = i % STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.full[s], (i / STAGES) & 1, abort_flag, 22, &g_tc_status));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t da = make_smem_desc(smem_u32(sm.w[s][h]));
          const uint64_t db = make_smem_desc(smem_u32(sm.x[s][h]));
#pragma unroll
          for (int k = 0; k < SK_HALF / 16; ++k) tc_mma_bf16_elect(tmem, da + 2 * k, db + 2 * k, idesc, (i | h | k) != 0);
        }
        tc_commit_elect(&sm.empty[s]);
      }
      if (ok) tc_commit_elect(&sm.acc_full);
    }
  } else {
    // ---- this CTA's partial sums into its shared memory: lane = weight row, columns = tokens -----------
    const int quarter = warp & 3;
    const int row = BM == 64 ? quarter * 16 + lane : quarter * 32 + lane;
    bool ok = true;
    if (n_kb > 0) ok = __all_sync(0xffffffffu, mbar_wait(&sm.acc_full, 0, abort_flag, 23, &g_tc_status));
    tc_fence_after();
#pragma unroll 1
    for (int c0 = 0; c0 < mt; c0 += 16) {
      uint32_t r[16];
      if (n_kb > 0 && ok) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + ((uint32_t)(quarter * 32) << 16) + c0) : "memory");
        tc_wait_ld();
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = 0u;      // a share without k-blocks adds nothing
      }
      if (BM == 128 || lane < 16) {
#pragma unroll
        for (int j = 0; j < 16; ++j) sm.part[c0 + j][row] = __uint_as_float(r[j]);
      }
    }
    if (RESID) pdl_wait();                            // the stream is an earlier kernel's output
  }

  cluster_sync_all();                                 // every CTA's partial sums are in place

  if (warp >= 2) {
    // ---- CTA r: tokens r, r + S, ...; half a warp (or a whole one) per token, a lane per 4 weight rows ----
    constexpr int LANES = BM / 4, AT_ONCE = 128 / LANES;
    const int wt = (threadIdx.x - 64) / LANES, lr = lane % LANES;
    uint32_t base[S];
#pragma unroll
    for (int s = 0; s < S; ++s) base[s] = cluster_map_shared(&sm.part[0][0], (uint32_t)s);
    const int n = n0 + 4 * lr;
#pragma unroll 2
    for (int c = rank + S * wt; c < M; c += AT_ONCE * S) {
      float4 v[S];
#pragma unroll
      for (int s = 0; s < S; ++s) v[s] = cluster_ld_f32x4(base[s] + (uint32_t)(c * BM + 4 * lr) * 4u);
      float4 acc = v[0];
#pragma unroll
      for (int s = 1; s < S; ++s) { acc.x += v[s].x; acc.y += v[s].y; acc.z += v[s].z; acc.w += v[s].w; }
      if (!RESID && act) {
        acc.x = act_for<TOut>(acc.x, act); acc.y = act_for<TOut>(acc.y, act);
        acc.z = act_for<TOut>(acc.z, act); acc.w = act_for<TOut>(acc.w, act);
      }
      if (n < N) {                                    // N % 4 == 0: the four lie inside together
        TOut* dst = out + (size_t)c * N + n;
        if constexpr (sizeof(TOut) == 4) {
          float4* d4 = reinterpret_cast<float4*>(dst);
          if (RESID) { const float4 o = *d4; acc.x += o.x; acc.y += o.y; acc.z += o.z; acc.w += o.w; }
          *d4 = acc;
        } else {
          __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
          uint2 u;
          u.x = *reinterpret_cast<uint32_t*>(&lo);
          u.y = *reinterpret_cast<uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(dst) = u;
        }
      }
    }
  }

  cluster_sync_all();                                 // nobody reads this CTA's shared memory any more
  // every thread waits for the previous kernel before the CTA ends (a kernel of this library never
  // completes before its predecessor)
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tc_dealloc(tmem, TMEM_COLS);
  }
}

template <typename TOut, int S, int BM, int BT, int STAGES, bool RESID>
static int launch_splitk_as(const void* x, const void* w, void* out, int M, int N, int K, cudaStream_t stream, int act) {
  CUtensorMap map_w, map_x;
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)N};
    const uint64_t strides[1] = {(uint64_t)K * 2};
    const uint32_t box[2] = {SK_HALF, BM};
    if (!qe_tensor_map_bf16(w, 2, dims, strides, box, &map_w)) return 1;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t strides[1] = {(uint64_t)K * 2};
    const uint32_t box[2] = {SK_HALF, (uint32_t)BT};
    if (!qe_tensor_map_bf16(x, 2, dims, strides, box, &map_x)) return 1;
  }
  const size_t smem = sizeof(SkSmem<BM, BT, STAGES>) + 1024;
  static_assert(tc_room_for_all(sizeof(SkSmem<BM, BT, STAGES>) + 1024, BT < 32 ? 32 : BT), "tensor memory for every CTA that finds room on an SM");
  static const cudaError_t configured = cudaFuncSetAttribute(gemm_tcgen05_splitk_kernel<TOut, S, BM, BT, STAGES, RESID>,
                                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (configured != cudaSuccess) QE_REFUSE("linear_tcgen05_splitk: shared memory %zu: %s", smem, cudaGetErrorString(configured));
  const dim3 grid((unsigned)((N + BM - 1) / BM) * S);
  qe_launch_cluster(gemm_tcgen05_splitk_kernel<TOut, S, BM, BT, STAGES, RESID>, grid, dim3(SK_THREADS), smem, stream, (unsigned)S,
                    map_w, map_x, (TOut*)out, M, N, K, act);
  QE_CHECK_LAUNCH("linear_tcgen05_splitk");
  return 0;
}

template <int S, int BM, int BT, int STAGES>
static int launch_splitk_rows(const void* x, const void* w, void* out, int M, int N, int K, int mode, cudaStream_t stream, int act) {
  if (mode == 2) return launch_splitk_as<float, S, BM, BT, STAGES, true>(x, w, out, M, N, K, stream, act);
  if (mode == 1) return launch_splitk_as<float, S, BM, BT, STAGES, false>(x, w, out, M, N, K, stream, act);
  return launch_splitk_as<__nv_bfloat16, S, BM, BT, STAGES, false>(x, w, out, M, N, K, stream, act);
}
// Clusters of 2 and 4 up to 32 tokens: 64 rows (the ring and the sums: 85 and 105 KB, two CTAs per SM).  Clusters of 8, whose
// shares of K are short and which find room less easily the more they are, and more tokens: 128 rows, a CTA per SM.
template <int S>
static int launch_splitk(const void* x, const void* w, void* out, int M, int N, int K, int mode, cudaStream_t stream, int act) {
  if constexpr (S < 8) {
    if (M <= 16) return launch_splitk_rows<S, 64, 16, 4>(x, w, out, M, N, K, mode, stream, act);
    if (M <= 32) return launch_splitk_rows<S, 64, 32, 4>(x, w, out, M, N, K, mode, stream, act);
  }
  return launch_splitk_rows<S, 128, 64, 3>(x, w, out, M, N, K, mode, stream, act);
}

extern "C" int qe_gemm_tc_splitk_status() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int));
  return v;
}
extern "C" void qe_gemm_tc_splitk_clear_status() {
  int v = 0;
  cudaMemcpyToSymbol(g_tc_status, &v, sizeof(int));
}

// 1 <= M <= 64; splits: 2, 4 or 8 CTAs per tile of weight rows (each gets ceil(K / 128 / splits) blocks of
// K; shares beyond K's end add nothing).  mode 0: out bfloat16; 1: out float32; 2: out float32 += the
// product.  Returns 0 when run, 1 when refused (qe_last_error says why), 2 on a launch error.
extern "C" int qe_linear_tcgen05_splitk(const void* x, const void* w, void* out, int M, int N, int K, int splits, int mode,
                                        cudaStream_t stream) {
  const int act = mode >> 2;                          // (modes 0 and 1: the activation of the sums, common.cuh)
  mode &= 3;
  if (act < 0 || act > QE_ACT_MAX || (act && mode == 2)) QE_REFUSE("linear_tcgen05_splitk: activation %d", act);
  if (M <= 0 || N <= 0) return 0;
  if (M > SK_MAX_M) QE_REFUSE("linear_tcgen05_splitk: M = %d is above %d", M, SK_MAX_M);
  if (K <= 0 || K % 8) QE_REFUSE("linear_tcgen05_splitk: K = %d is not a positive multiple of 8", K);
  if (N % 4) QE_REFUSE("linear_tcgen05_splitk: N = %d is not a multiple of 4", N);
  if (mode < 0 || mode > 2) QE_REFUSE("linear_tcgen05_splitk: mode %d", mode);
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) QE_REFUSE("linear_tcgen05_splitk: operands must be 16-byte aligned");
  if (splits == 2) return launch_splitk<2>(x, w, out, M, N, K, mode, stream, act);
  if (splits == 4) return launch_splitk<4>(x, w, out, M, N, K, mode, stream, act);
  if (splits == 8) return launch_splitk<8>(x, w, out, M, N, K, mode, stream, act);
  QE_REFUSE("linear_tcgen05_splitk: %d splits (2, 4 or 8)", splits);
}
