// Attention of a step's new queries over the paged cache, for any mixture of prompt portions
// and single decoded tokens, any head size up to 640, any page size, any number of heads and
// groups, float32 or bfloat16 storage; all arithmetic in float32 with expf.
//
// For the query at position i of a request, key j is allowed iff j <= i and (window == 0 or
// j > i - window) (reference src/layers/fused_ops/attn.py:195, 239); scores are scale * q·k, less
// slopes[head] * (i - j) where a mixer biases by distance,
// softmax runs online over key tiles of 32 that start at multiples of 32 of the absolute key
// position, so the order of a query's reduction does not depend on how the request was cut into
// steps (attn.py:236-267 has the same algebra per BLOCK_N).  Query head h reads kv head
// h / (Hq / Hkv) (attn.py:181-182).
//
// Options of other designs: `softcap` > 0 bends the scaled score s to softcap tanh(s / softcap) ahead of the mask; `sinks`
// [Hq] adds exp(sinks[h]) to head h's denominator (no key, no value); `v_shift` lets a head whose kv head is c read the
// values of kv head (c + v_shift) mod Hkv (the keys stay its own).  A page of 1 + n planes (n > 1) holds the keys and n blocks of
// D value channels; the grid's z runs over the blocks and a head's output has n D channels.
//
// One CTA per (tile of 16 queries of one request, query head); 4 warps, 4 queries each.  Within a
// warp lane j owns key j of the tile for the scores and dims d = lane + 32 i of the output.
//
// What bounds it: a CTA's chain of tiles, each a copy of 32 keys and values into shared memory, four chains of D
// multiply-adds a lane and 32 steps of the weighted sum.  A warp therefore takes its four queries together (a key's words are
// read once for the four chains, which hide each other's latency; a query's own order of sums is what it is alone), words of
// four channels are read at a time (rows of keys padded to an odd number of them: no bank conflicts), float32
// tiles are copied asynchronously one ahead, and the accumulators are as many as the head size needs.  Measured on a B200,
// Qwen3-0.6B's sizes in float32 (three prompts of 141 tokens together, then steps of three tokens): 49.9 us a launch on
// average with a query at a time and element-wise copies, 22.8 with four queries at a time, 13.3 with copies a tile ahead.
#include "common.cuh"
#include <math.h>

#define AG_BM 16
#define AG_BN 32
#define AG_WARPS 4
#define AG_MAX_D 640       // (heads beyond 512 channels run an instantiation with more accumulators a lane)
#define AG_QPW (AG_BM / AG_WARPS)      // queries per warp

// floats of a key's row in shared memory: whole 16-byte words, an odd number of them
__host__ __device__ constexpr int ag_key_stride(int D) { return 4 * (((D + 3) / 4) | 1); }
__host__ __device__ constexpr int ag_value_stride(int D) { return (D + 3) / 4 * 4; }
static size_t ag_smem(int D, int bufs) {
  return ((size_t)AG_BM * ag_value_stride(D) + (size_t)bufs * AG_BN * (ag_key_stride(D) + ag_value_stride(D)) + AG_BM * AG_BN) * sizeof(float);
}

__device__ __forceinline__ float4 ag_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ag_load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

// VEC: D is a multiple of 4 and queries and pages can be read four elements at a time.  Float32 pages are then copied
// straight into shared memory (cp.async), and up to AG_TWO_BUFFERS_D channels the next tile's copy runs under this one's sums.
// (Beyond 128 channels two buffers leave one CTA per SM, 150 KB at 256, and are faster all the same than the kernel with a query at a
// time: three prompts of 47 tokens 68 -> 18 us at 160 channels, 90 -> 18 at 256; one of 2 048 7.3 -> 2.3 and 13.3 -> 3.8 ms.)
#define AG_TWO_BUFFERS_D 256
template <typename T, int DREG, bool VEC>
__global__ void __launch_bounds__(AG_WARPS * 32)
attention_generic_kernel(const T* __restrict__ q, long q_stride, const T* __restrict__ pages,
                         const int* __restrict__ block_tables, int max_blocks,
                         const int* __restrict__ cu_q, const int* __restrict__ ctx_lens,
                         const int* __restrict__ tiles, T* __restrict__ out, float scale, int window,
                         int Hq, int Hkv, int D, int page_size, const float* __restrict__ slopes, int kv_planes,
                         float softcap, const float* __restrict__ sinks, int v_shift) {
  extern __shared__ __align__(16) float smem[];
  pdl_launch_dependents();
  pdl_wait();
  constexpr bool ASYNC = VEC && sizeof(T) == 4;
  constexpr bool TWO = ASYNC && 32 * DREG <= AG_TWO_BUFFERS_D;
  const int Dk = ag_key_stride(D), Dv = ag_value_stride(D);
  int buf_w = AG_BN * (Dk + Dv);              // from this tile's buffer to the next one's
  float* qs = smem;                           // [AG_BM][Dv], zeros behind channel D
  float* ps = qs + AG_BM * Dv;                // [AG_BM][AG_BN]: the queries' weights of the tile
  float* ks = ps + AG_BM * AG_BN;             // [AG_BN][Dk], zeros behind channel D; then the values [AG_BN][Dv]; then the other buffer
  const int tile = blockIdx.x, hq = blockIdx.y;
  const int hkv = hq / (Hq / Hkv);
  const int hv = (hkv + v_shift) % Hkv;                 // the kv head whose values the head's weights meet (its own unless shifted)
  const float slope = slopes ? slopes[hq] : 0.f;        // distance bias: slope * (i - j) is taken off the score
  const int req = tiles[2 * tile], q0 = tiles[2 * tile + 1];
  const int row0 = cu_q[req];
  const int q_len = cu_q[req + 1] - row0;
  const int ctx = ctx_lens[req];
  const int nq = min(AG_BM, q_len - q0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* table = block_tables + (size_t)req * max_blocks;
  const int words = Dv / 4;

  for (int e = threadIdx.x; e < AG_BM * words; e += AG_WARPS * 32) {
    const int r = e / words, d = (e - r * words) * 4;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nq) {
      const T* src = q + (size_t)(row0 + q0 + r) * q_stride + (size_t)hq * D + d;
      if (VEC) {
        t = ag_load4(src);
      } else {
        t.x = to_f32(src[0]);
        if (d + 1 < D) t.y = to_f32(src[1]);
        if (d + 2 < D) t.z = to_f32(src[2]);
        if (d + 3 < D) t.w = to_f32(src[3]);
      }
    }
    *reinterpret_cast<float4*>(qs + r * Dv + d) = t;
  }

  float m[AG_QPW], l[AG_QPW];
  float acc[AG_QPW][DREG];
#pragma unroll
  for (int i = 0; i < AG_QPW; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < DREG; ++c) acc[i][c] = 0.f;
  }

  const int first_pos = ctx + q0;                       // position of the tile's first query
  const int kv_end = ctx + q0 + nq;                     // one past the last allowed key
  const int kv_begin = window > 0 ? max(0, first_pos - window + 1) : 0;
  // (kv_planes 1: a page holds one plane per kv head, and the values are its channels)
  const size_t to_values = kv_planes == 1 ? 0 : ((size_t)Hkv * (1 + blockIdx.z) + hv - hkv) * page_size * D;
  // keys and values kt..kt + 31 into a buffer: a warp takes every fourth of them, zeros where there is none
  auto stage = [&](int kt, float* kb) {
    float* vb = kb + AG_BN * Dk;
#pragma unroll
    for (int i = 0; i < AG_BN / AG_WARPS; ++i) {
      const int j = warp + i * AG_WARPS, kj = kt + j;
      const bool there = kj >= kv_begin && kj < kv_end;
      const T* src = pages;
      if (there) src += ((((size_t)table[kj / page_size] * kv_planes) * Hkv + hkv) * page_size + (kj % page_size)) * D;
      for (int d = lane * 4; d < Dv; d += 128) {
        if (ASYNC) {
          const int bytes = there ? 16 : 0;             // nothing is read for a key outside; the 16 bytes become zeros
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                       :: "r"((uint32_t)__cvta_generic_to_shared(kb + j * Dk + d)), "l"(there ? src + d : src), "r"(bytes) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                       :: "r"((uint32_t)__cvta_generic_to_shared(vb + j * Dv + d)), "l"(there ? src + to_values + d : src), "r"(bytes) : "memory");
          continue;
        }
        float4 kvl = make_float4(0.f, 0.f, 0.f, 0.f), vvl = kvl;
        if (there) {
          const T* vsrc = src + to_values + d;
          const T* ksrc = src + d;
          if (VEC) {
            kvl = ag_load4(ksrc);
            vvl = kv_planes == 1 ? kvl : ag_load4(vsrc);
          } else {
            kvl.x = to_f32(ksrc[0]); vvl.x = to_f32(vsrc[0]);
            if (d + 1 < D) { kvl.y = to_f32(ksrc[1]); vvl.y = to_f32(vsrc[1]); }
            if (d + 2 < D) { kvl.z = to_f32(ksrc[2]); vvl.z = to_f32(vsrc[2]); }
            if (d + 3 < D) { kvl.w = to_f32(ksrc[3]); vvl.w = to_f32(vsrc[3]); }
          }
        }
        *reinterpret_cast<float4*>(kb + j * Dk + d) = kvl;
        *reinterpret_cast<float4*>(vb + j * Dv + d) = vvl;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  const int kt0 = (kv_begin / AG_BN) * AG_BN;
  if (TWO) stage(kt0, ks);
  for (int kt = kt0; kt < kv_end; kt += AG_BN) {
    __syncthreads();                                    // the tile before is read no more
    if (TWO) {
      if (kt + AG_BN < kv_end) stage(kt + AG_BN, ks + buf_w); else asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      stage(kt, ks);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float* kb = ks;
    const float* vb = ks + AG_BN * Dk;
    if (TWO) { ks += buf_w; buf_w = -buf_w; }
    const int r0 = warp * AG_QPW;
    if (r0 >= nq) continue;                             // uniform within the warp
    float s[AG_QPW];
#pragma unroll
    for (int i = 0; i < AG_QPW; ++i) s[i] = 0.f;
    const float* kr = kb + lane * Dk;
#pragma unroll 8
    for (int d = 0; d < Dv; d += 4) {
      const float4 kd = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
      for (int i = 0; i < AG_QPW; ++i) {
        const float4 qd = *reinterpret_cast<const float4*>(qs + (r0 + i) * Dv + d);
        s[i] = fmaf(qd.x, kd.x, s[i]);
        s[i] = fmaf(qd.y, kd.y, s[i]);
        s[i] = fmaf(qd.z, kd.z, s[i]);
        s[i] = fmaf(qd.w, kd.w, s[i]);
      }
    }
    bool live[AG_QPW];                                  // the query is one of the tile's and may see a key of these
#pragma unroll
    for (int i = 0; i < AG_QPW; ++i) {
      const int pos = first_pos + r0 + i;
      const int kj = kt + lane;
      const bool ok = r0 + i < nq && kj <= pos && (window <= 0 || kj > pos - window);
      float t = s[i] * scale;
      if (softcap > 0.f) t = softcap * tanhf(t / softcap);          // the score bent towards +-softcap
      t = ok ? fmaf(-slope, (float)(pos - kj), t) : -INFINITY;
      const float tile_max = warp_max(t);
      live[i] = tile_max != -INFINITY;
      if (!live[i]) continue;
      const float m_new = fmaxf(m[i], tile_max);
      const float alpha = expf(m[i] - m_new);           // exp(-inf) = 0 on the first tile
      const float p = ok ? expf(t - m_new) : 0.f;
      l[i] = l[i] * alpha + warp_sum(p);
      m[i] = m_new;
#pragma unroll
      for (int c = 0; c < DREG; ++c) acc[i][c] *= alpha;
      ps[(r0 + i) * AG_BN + lane] = p;
    }
    __syncwarp();
#pragma unroll 2
    for (int j = 0; j < AG_BN; j += 4) {
      float v[4][DREG];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < DREG; ++c) {
          const int d = lane + 32 * c;
          v[u][c] = d < D ? vb[(j + u) * Dv + d] : 0.f;
        }
#pragma unroll
      for (int i = 0; i < AG_QPW; ++i) {
        if (!live[i]) continue;
        const float4 p = *reinterpret_cast<const float4*>(ps + (r0 + i) * AG_BN + j);
#pragma unroll
        for (int c = 0; c < DREG; ++c) {
          acc[i][c] = fmaf(p.x, v[0][c], acc[i][c]);
          acc[i][c] = fmaf(p.y, v[1][c], acc[i][c]);
          acc[i][c] = fmaf(p.z, v[2][c], acc[i][c]);
          acc[i][c] = fmaf(p.w, v[3][c], acc[i][c]);
        }
      }
    }
    __syncwarp();                                       // the next tile's weights take the place of these
  }
#pragma unroll
  for (int i = 0; i < AG_QPW; ++i) {
    const int r = warp * AG_QPW + i;
    if (r >= nq) continue;
    // a sink: exp(sinks[head]) joins the denominator; it has no key and no value
    const float inv = 1.f / (sinks ? l[i] + expf(sinks[hq] - m[i]) : l[i]);
    T* o = out + (((size_t)(row0 + q0 + r) * Hq + hq) * gridDim.z + blockIdx.z) * D;
#pragma unroll
    for (int c = 0; c < DREG; ++c) {
      const int d = lane + 32 * c;
      if (d < D) o[d] = from_f32<T>(acc[i][c] * inv);
    }
  }
}

template <typename T, int DREG, bool VEC>
static int ag_launch(const void* q, long q_stride, const void* pages, const int* block_tables, int max_blocks, const int* cu_q,
                     const int* ctx_lens, const int* tiles, int n_tiles, void* out, float scale, int window, int Hq, int Hkv, int D,
                     int page_size, const float* slopes, int kv_planes, float softcap, const float* sinks, int v_shift, cudaStream_t stream) {
  // the instantiation's largest head size sets the limit once (not per launch: launches may be under stream capture)
  constexpr int bufs = VEC && sizeof(T) == 4 && 32 * DREG <= AG_TWO_BUFFERS_D ? 2 : 1;
  static const cudaError_t configured = cudaFuncSetAttribute(attention_generic_kernel<T, DREG, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                             (int)ag_smem(32 * DREG, bufs));
  if (configured != cudaSuccess) QE_REFUSE("paged_attention: shared memory %d: %s", (int)ag_smem(32 * DREG, bufs), cudaGetErrorString(configured));
  qe_launch(attention_generic_kernel<T, DREG, VEC>, dim3(n_tiles, Hq, kv_planes > 2 ? kv_planes - 1 : 1), dim3(AG_WARPS * 32), ag_smem(D, bufs), stream,
            (const T*)q, q_stride, (const T*)pages, block_tables, max_blocks, cu_q, ctx_lens, tiles, (T*)out, scale, window, Hq, Hkv, D,
            page_size, slopes, kv_planes, softcap, sinks, v_shift);
  QE_CHECK_LAUNCH("paged_attention_generic");
  return 0;
}

extern "C" int qe_paged_attention_generic(const void* q, long q_stride, const void* pages,
                                          const int* block_tables, int max_blocks, const int* cu_q,
                                          const int* ctx_lens, const int* tiles, int n_tiles, void* out,
                                          float scale, int window, int Hq, int Hkv, int D, int page_size,
                                          int dtype, const float* slopes, int kv_planes, float softcap, const float* sinks,
                                          int v_shift, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (D > AG_MAX_D || D < 1) QE_REFUSE("paged_attention: head_dim %d is outside 1..%d", D, AG_MAX_D);
  if (Hkv < 1 || Hq % Hkv) QE_REFUSE("paged_attention: %d query heads do not group over %d kv heads", Hq, Hkv);
  if (Hq > 65535) QE_REFUSE("paged_attention: too many heads (%d)", Hq);
  const int planes = kv_planes;
  if (planes < 1 || v_shift < 0 || v_shift >= Hkv || (v_shift && planes != 2)) QE_REFUSE("paged_attention: a shift of %d over %d kv heads", v_shift, Hkv);
  if (dtype != QE_DTYPE_F32 && dtype != QE_DTYPE_BF16) QE_REFUSE("paged_attention: unknown dtype %d", dtype);
  const int size = dtype == QE_DTYPE_F32 ? 4 : 2;
  const bool vec = D % 4 == 0 && q_stride % 4 == 0 && (uintptr_t)q % (4 * size) == 0 && (uintptr_t)pages % (4 * size) == 0;
#define AGL(TT, DR, VV) return ag_launch<TT, DR, VV>(q, q_stride, pages, block_tables, max_blocks, cu_q, ctx_lens, tiles, n_tiles, out, scale, \
                                                     window, Hq, Hkv, D, page_size, slopes, planes, softcap, sinks, v_shift, stream)
#define AGD(TT, VV) do { if (D <= 128) AGL(TT, 4, VV); if (D <= 256) AGL(TT, 8, VV); if (D <= 512) AGL(TT, 16, VV); AGL(TT, AG_MAX_D / 32, VV); } while (0)
  if (dtype == QE_DTYPE_F32) { if (vec) AGD(float, true); else AGD(float, false); }
  if (vec) AGD(__nv_bfloat16, true); else AGD(__nv_bfloat16, false);
#undef AGD
#undef AGL
}
