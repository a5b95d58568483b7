// out[M, N] = x[M, K] · w[N, K]^T in bfloat16 for up to 32 rows, and act(x · gate^T) * (x · up^T) over stacked weights for up to
// 64, where the weight rows are many but no multiple of what the other kernels spread evenly: 64 weight rows a CTA.
//
// What bounds it: the weights' way from memory.  gemm_tcgen05_swap.cu gives 128 weight rows to a CTA that fills an SM's
// shared memory, so 19 456 rows (Qwen3-4B's gate and up) are 152 CTAs, four more than the SMs, and take two rounds, and
// 12 288 leave 52 SMs idle.  Here a CTA has 64 rows (the 64-row form of tcgen05.mma) and a ring small enough for two or
// three CTAs per SM (three up to 32 rows, two beyond): all of them are on the GPU at once, whatever their number within 444 or
// 296, and an SM's loads are as many.  What goes beyond that takes another round: 19 456 rows with the activation, 304 CTAs, 18.7 us
// at 32 rows and 27.4 at 33 (a product and the activation's launch: 32.8 and 33.1).
// The ring starts with the weights, before the wait for the kernel that writes x.
//
// GLU: a CTA's rows are 32 of the gate's and the same 32 of the up projection's (two boxes side by side), and the
// activation is formed on the float32 sums in the epilogue, rounded once: gate and up never exist in memory, and the
// activation needs no launch of its own.
//
// Precision: tensor memory adds a product in without rounding to nearest, and the error grows with the length of the chain (1e-6 of
// the result for K = 1 024 in one chain, 4e-6 for 4 096).  Up to 16 rows, where the weight-streaming product gives the k to eight
// warps at most, every 64 k go to the next of eight accumulators of 16 columns, which are added up in order at the end: chains no
// longer than there (151 936 x 1 024 1.3e-7, that product 2.2e-7; 16 384 x 4 096 both 4.8e-7).  It costs 0.3-0.5 us a launch and 1.3 over the vocabulary.
//
// Six warps as in gemm_tcgen05_swap.cu: TMA, MMA, and four that read the accumulator (the 64-row form keeps row r in lane
// r mod 16 of the quarter r / 16), put it into the ring's memory as [token][row] and store whole runs of a token's outputs.
// Every wait on an mbarrier is bounded; qe_gemm_tc_stream_status() reads this kernel's flag.
// A stage holds 128 k: the thread that waits for one, issues its products and releases it needs 0.19 us a stage and 0.01 for a
// product, whatever a stage holds (64 k a stage: 6 144 x 2 560 at 16 rows 14 us, 128: 10.4), and more stages change nothing.
// Measured on a B200, chains over weights larger than L2, with the activation: 19 456 x 2 560 at 16 rows 17.4 us (5.7 TB/s) where
// the weight-streaming product takes 30.0, 12 288 x 2 048 at 28 rows 11.2 where a product and the activation take 13.6; without:
// 151 936 x 2 560 at 16 rows 120 us (6.5 TB/s), 167 before.
//
// Needs K % 8 == 0 and x and w on 16-byte boundaries; the launcher refuses the rest.
#include "tcgen05.cuh"

#define SR_BM 64                // weight rows per CTA
#define SR_HALF 64              // k of a box (128 bytes: the swizzle's width)
#define SR_BK (2 * SR_HALF)     // k of a stage: two boxes of each operand
#define SR_THREADS 192

static __device__ int g_tc_status = 0;      // 0 = fine; else code of the first wait that ran out

template <int BT, int STAGES>    // BT: tokens at most (rows of the token operand's box)
struct __align__(1024) SrSmem {
  __nv_bfloat16 w[STAGES][2][SR_BM * SR_HALF];  // 16 KB each
  __nv_bfloat16 x[STAGES][2][BT * SR_HALF];
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

// 16 columns of this warp's quarter of the lanes (a lane's row), to be waited for
__device__ __forceinline__ void sr_load16(uint32_t at, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(at) : "memory");
}

template <typename TOut, int BT, int STAGES, bool GLU, int ACCS>    // ACCS: accumulators, BT columns each
__global__ void __launch_bounds__(SR_THREADS)
gemm_tcgen05_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                           TOut* __restrict__ out, int M, int N, int K, int act) {
  extern __shared__ unsigned char smem_raw[];
  using Smem = SrSmem<BT, STAGES>;
  static_assert(sizeof(float) * BT * SR_BM <= sizeof(__nv_bfloat16) * STAGES * SR_BM * SR_BK, "the sums take the ring's place");
  constexpr uint32_t TMEM_COLS = BT * ACCS < 32 ? 32 : BT * ACCS;
  constexpr int COLS = GLU ? SR_BM / 2 : SR_BM;       // outputs of a token per CTA
  pdl_launch_dependents();
  Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * COLS;
  const int num_kb = (K + SR_BK - 1) / SR_BK;
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
    if (lane == 0) {
      auto load_w = [&](int kb) {
        const int s = kb % STAGES;
        mbar_expect_tx(&sm.full[s], (SR_BM + BT) * SR_BK * sizeof(__nv_bfloat16));
#pragma unroll
        for (int h = 0; h < 2; ++h) {                 // (a half that lies behind K is zeros)
          tma_load_2d(sm.w[s][h], &map_w, &sm.full[s], kb * SR_BK + h * SR_HALF, n0);
          if (GLU) tma_load_2d(sm.w[s][h] + SR_BM / 2 * SR_HALF, &map_w, &sm.full[s], kb * SR_BK + h * SR_HALF, N + n0);   // (N: the gate's rows)
        }
      };
      auto load_x = [&](int kb) {
        const int s = kb % STAGES;
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_2d(sm.x[s][h], &map_x, &sm.full[s], kb * SR_BK + h * SR_HALF, 0);
      };
      const int ahead = min(num_kb, STAGES);
      for (int kb = 0; kb < ahead; ++kb) load_w(kb);
      pdl_wait();
      for (int kb = 0; kb < ahead; ++kb) load_x(kb);
      int issued = ahead;
      for (int kb = ahead; kb < num_kb; ++kb) {
        const int s = kb % STAGES;
        if (!mbar_wait(&sm.empty[s], ((kb / STAGES) - 1) & 1, abort_flag, 31, &g_tc_status)) break;
        load_w(kb);
        load_x(kb);
        ++issued;
      }
      if (*abort_flag) {
        for (int i = max(0, issued - STAGES); i < issued; ++i)
          for (uint32_t spin = 0; spin < TC_WAIT_LIMIT; ++spin)
            if (mbar_try_wait(&sm.full[i % STAGES], (i / STAGES) & 1)) break;
      }
    }
  } else if (warp == 1) {
    // (the whole warp walks the k-blocks and one lane is elected per instruction: what an instruction is given stays in
    // uniform registers)
    const uint32_t idesc = make_idesc(SR_BM, mt);
    bool ok = true;
    for (int kb = 0; kb < num_kb; ++kb) {
      const int s = kb % STAGES;
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.full[s], (kb / STAGES) & 1, abort_flag, 32, &g_tc_status));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint64_t da = make_smem_desc(smem_u32(sm.w[s][h]));
        const uint64_t db = make_smem_desc(smem_u32(sm.x[s][h]));
#pragma unroll
        for (int k = 0; k < SR_HALF / 16; ++k)
          tc_mma_bf16_elect(tmem + (2 * kb + h) % ACCS * BT, da + 2 * k, db + 2 * k, idesc, 2 * kb + h >= ACCS || k != 0);
      }
      tc_commit_elect(&sm.empty[s]);
    }
    if (ok) tc_commit_elect(&sm.acc_full);
  } else {
    const int quarter = warp & 3;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&sm.acc_full, 0, abort_flag, 33, &g_tc_status));
    tc_fence_after();
    float* sums = reinterpret_cast<float*>(sm.w[0][0]);  // [token][64]: every load has landed and been read
    if (ok) {
#pragma unroll 1
      for (int c0 = 0; c0 < mt; c0 += 16) {
        uint32_t r[16];
        if constexpr (ACCS == 1) {
          sr_load16(tmem + ((uint32_t)(quarter * 32) << 16) + c0, r);
          tc_wait_ld();
        } else {                                        // added in order, four at a time on their way
          static_assert(ACCS == 8, "two rounds");
#pragma unroll
          for (int a0 = 0; a0 < ACCS; a0 += 4) {
            if (a0 >= 2 * num_kb) break;                // accumulators that no k reached hold nothing
            uint32_t u[4][16];
#pragma unroll
            for (int a = 0; a < 4; ++a) sr_load16(tmem + ((uint32_t)(quarter * 32) << 16) + (a0 + a) * BT + c0, u[a]);
            tc_wait_ld();
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const bool any = a0 + a < 2 * num_kb;
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                asm volatile("" : "+r"(u[a][j]));       // (not read before the wait)
                if (a0 + a == 0) r[j] = u[a][j];
                else r[j] = __float_as_uint(__uint_as_float(r[j]) + (any ? __uint_as_float(u[a][j]) : 0.f));
              }
            }
          }
        }
        if (lane < 16) {
#pragma unroll
          for (int j = 0; j < 16; ++j) sums[(c0 + j) * SR_BM + quarter * 16 + lane] = __uint_as_float(r[j]);
        }
      }
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (ok) {
      for (int t = warp - 2; t < M; t += 4) {
        const float* row = sums + t * SR_BM;
        TOut* dst = out + (size_t)t * N + n0;
        if (GLU) {
          if (n0 + lane < N) dst[lane] = from_f32<TOut>(glu_fast(row[lane], row[SR_BM / 2 + lane], act));
        } else {
#pragma unroll
          for (int h = 0; h < SR_BM; h += 32)
            if (n0 + h + lane < N) dst[h + lane] = from_f32<TOut>(act_for<TOut>(row[h + lane], act));
        }
      }
    }
  }
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

template <typename TOut, int BT, int STAGES, bool GLU, int ACCS = 1>
static int launch_stream(const void* x, const void* w, void* out, int M, int N, int K, int act, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)N * (GLU ? 2 : 1)};
    const uint64_t strides[1] = {(uint64_t)K * 2};
    const uint32_t box[2] = {SR_HALF, GLU ? SR_BM / 2 : SR_BM};
    if (!qe_tensor_map_bf16(w, 2, dims, strides, box, &map_w)) return 1;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t strides[1] = {(uint64_t)K * 2};
    const uint32_t box[2] = {SR_HALF, (uint32_t)BT};
    if (!qe_tensor_map_bf16(x, 2, dims, strides, box, &map_x)) return 1;
  }
  const size_t smem = sizeof(SrSmem<BT, STAGES>) + 1024;
  static_assert(tc_room_for_all(sizeof(SrSmem<BT, STAGES>) + 1024, BT * ACCS < 32 ? 32 : BT * ACCS), "tensor memory for every CTA that finds room on an SM");
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_tcgen05_stream_kernel<TOut, BT, STAGES, GLU, ACCS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (configured != cudaSuccess) QE_REFUSE("linear_tcgen05_stream: shared memory %zu: %s", smem, cudaGetErrorString(configured));
  const int cols = GLU ? SR_BM / 2 : SR_BM;
  qe_launch(gemm_tcgen05_stream_kernel<TOut, BT, STAGES, GLU, ACCS>, dim3((unsigned)((N + cols - 1) / cols)), dim3(SR_THREADS), smem, stream,
            map_w, map_x, (TOut*)out, M, N, K, act);
  QE_CHECK_LAUNCH("linear_tcgen05_stream");
  return 0;
}

extern "C" int qe_gemm_tc_stream_status() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int));
  return v;
}
extern "C" void qe_gemm_tc_stream_clear_status() {
  int v = 0;
  cudaMemcpyToSymbol(g_tc_status, &v, sizeof(int));
}

// (the ring's stages: three CTAs per SM up to 32 tokens, two beyond)
template <typename TOut, bool GLU>
static int launch_stream_rows(const void* x, const void* w, void* out, int M, int N, int K, int act, cudaStream_t stream) {
  if (M <= 16) return launch_stream<TOut, 16, 3, GLU, GLU ? 1 : 8>(x, w, out, M, N, K, act, stream);
  if (M <= 32) return launch_stream<TOut, 32, 3, GLU>(x, w, out, M, N, K, act, stream);
  if constexpr (GLU) return launch_stream<TOut, 64, 3, GLU>(x, w, out, M, N, K, act, stream);
  else QE_REFUSE("linear_tcgen05_stream: M = %d is above 32", M);
}

// The forms of qe_linear_tcgen05_swap (which has checked the operands) with 64 weight rows a CTA, 1 <= M <= 32.  glu: N outputs
// over w [2 N, K], M <= 64, act as glu_fast takes it, out bfloat16; else act as act_for does.
int qe_gemm_tc_stream(const void* x, const void* w, void* out, int M, int N, int K, int out_f32, int act, bool glu, cudaStream_t stream) {
  if (glu) return launch_stream_rows<__nv_bfloat16, true>(x, w, out, M, N, K, act, stream);
  if (out_f32) return launch_stream_rows<float, false>(x, w, out, M, N, K, act, stream);
  return launch_stream_rows<__nv_bfloat16, false>(x, w, out, M, N, K, act, stream);
}
