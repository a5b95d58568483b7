// The fused per-head norm + rotary encoding + cache write for head size 128 as device functions (see elementwise.cu).
#pragma once
#include "common.cuh"

// The common case, head size 128 with all of it rotated (or none): a lane holds 4
// consecutive elements, its rotation partner (d +- 64) is held by lane +- 16, no shared memory.
template <typename T>
struct RopeD128Args {
  T* q; T* k; const T* v;
  long q_stride, k_stride, v_stride;
  const int* positions; const float* qw; const float* kw; float eps; const float* inv_freq;
  const float2* cos_sin;            // optional [T, 64] (cos, sin) of position * inv_freq, made once per step
  T* pages; const int* slot_mapping;
  int T_tokens, Hq, Hkv, page_size, write_kv;
};

// four elements as they lie in memory
template <typename T> struct RopeRaw;
template <> struct RopeRaw<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void unpack(float (&f)[4]) const {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
  }
  __device__ __forceinline__ void pack(const float (&f)[4]) {
    __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    v.x = *reinterpret_cast<uint32_t*>(&a);
    v.y = *reinterpret_cast<uint32_t*>(&b);
  }
};
template <> struct RopeRaw<float> {
  uint4 v;
  __device__ __forceinline__ void unpack(float (&f)[4]) const {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
  }
  __device__ __forceinline__ void pack(const float (&f)[4]) {
    v = make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};

// One (token, head) by the calling warp.  In two halves, so that
// a warp can have the loads of several items in flight before it works on the first: the load of the
// lane's 4 elements, and the rest.  Loads of q, k, v bypass L1 (they are another kernel's or an
// earlier phase's output).
template <typename T>
__device__ __forceinline__ RopeRaw<T> rope_d128_load(const RopeD128Args<T>& A, int t, int head) {
  constexpr int D = 128;
  const int lane = threadIdx.x & 31;
  RopeRaw<T> raw = {};
  if (t >= A.T_tokens) return raw;
  const T* src;
  if (head < A.Hq) src = A.q + (size_t)t * A.q_stride + (size_t)head * D;
  else if (head < A.Hq + A.Hkv) src = A.k + (size_t)t * A.k_stride + (size_t)(head - A.Hq) * D;
  else {
    if (!A.write_kv) return raw;
    src = A.v + (size_t)t * A.v_stride + (size_t)(head - A.Hq - A.Hkv) * D;
  }
  raw.v = __ldcg(reinterpret_cast<const decltype(raw.v)*>(src + 4 * lane));
  return raw;
}

// What a lane needs besides the head's elements, none of it written by a kernel of the step (positions and
// slots come with the step's host copy, the rest are weights): a kernel may fetch it before it waits for
// its predecessor.  Angles only where the step has no table of them.
struct RopeD128Pre {
  float cs[4], sn[4];
  float4 wv;                        // the norm's weights: those of the first head's kind
  float4 wk;                        // MIXED: k's, for a warp that has heads of q and of k
  int slot;
};
// (for heads `head` to `last` of token t; MIXED: they may be of several kinds, q, k and v)
template <bool MIXED, typename T>
__device__ __forceinline__ void rope_d128_prepare(const RopeD128Args<T>& A, int t, int head, int last, RopeD128Pre& P) {
  const int lane = threadIdx.x & 31;
  P.slot = 0;
  P.wv = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) { P.cs[i] = 1.f; P.sn[i] = 0.f; }
  if (t >= A.T_tokens) return;
  if (A.write_kv && last >= A.Hq) P.slot = __ldg(A.slot_mapping + t);
  if (head >= A.Hq + A.Hkv) return;
  const float* w = head < A.Hq ? A.qw : A.kw;
  if (w) P.wv = __ldg(reinterpret_cast<const float4*>(w + 4 * lane));
  if (MIXED) P.wk = A.kw && last >= A.Hq ? __ldg(reinterpret_cast<const float4*>(A.kw + 4 * lane)) : P.wv;
  if (A.inv_freq && !A.cos_sin) {
    const float pos = (float)__ldg(A.positions + t);
#pragma unroll
    for (int i = 0; i < 4; ++i) sincosf(pos * __ldg(A.inv_freq + ((4 * lane + i) & 63)), &P.sn[i], &P.cs[i]);
  }
}

// The angles from the step's table, where it has one: a kernel of the step made it, so they are asked for after the wait, but
// together with the elements (behind the norm's sum they were a second round trip).  The models make a table for
// bfloat16 alone; the entry point takes one for either type.
template <typename T>
__device__ __forceinline__ void rope_d128_angles(const RopeD128Args<T>& A, int t, int head, RopeD128Pre& P) {
  if (!A.inv_freq || !A.cos_sin || t >= A.T_tokens || head >= A.Hq + A.Hkv) return;
  // the lane's four (cos, sin) pairs lie side by side in the table: two 16-byte loads
  const float4* tp = reinterpret_cast<const float4*>(A.cos_sin + (size_t)t * 64 + ((4 * (threadIdx.x & 31)) & 63));
  const float4 t01 = __ldg(tp), t23 = __ldg(tp + 1);
  P.cs[0] = t01.x; P.sn[0] = t01.y; P.cs[1] = t01.z; P.sn[1] = t01.w;
  P.cs[2] = t23.x; P.sn[2] = t23.y; P.cs[3] = t23.z; P.sn[3] = t23.w;
}

template <bool MIXED, typename T>
__device__ __forceinline__ void rope_d128_finish(const RopeD128Args<T>& A, int t, int head, const RopeRaw<T>& raw,
                                                 const RopeD128Pre& pre) {
  constexpr int D = 128;
  T* q = A.q; T* k = A.k;
  const long q_stride = A.q_stride, k_stride = A.k_stride;
  const float* qw = A.qw; const float* kw = A.kw; const float eps = A.eps;
  T* pages = A.pages;
  const int Hq = A.Hq, Hkv = A.Hkv, page_size = A.page_size, write_kv = A.write_kv;
  const int lane = threadIdx.x & 31;
  if (t >= A.T_tokens) return;
  if (head >= Hq + Hkv) {           // a value head: copy into the cache
    if (!write_kv) return;
    const int h = head - Hq - Hkv;
    const int slot = pre.slot;
    // slot = page * page_size + off: the row of (page, V, h, off) is slot + (page * (2 Hkv - 1) + Hkv + h) * page_size
    const int page = (page_size & (page_size - 1)) == 0 ? slot >> (__ffs(page_size) - 1) : slot / page_size;
    *reinterpret_cast<decltype(raw.v)*>(pages + ((size_t)slot + ((size_t)page * (2 * Hkv - 1) + Hkv + h) * page_size) * D + 4 * lane) = raw.v;
    return;
  }
  const bool is_q = head < Hq;
  const int h = is_q ? head : head - Hq;
  T* x = (is_q ? q + (size_t)t * q_stride : k + (size_t)t * k_stride) + (size_t)h * D + 4 * lane;
  const float* w = is_q ? qw : kw;
  float f[4];
  raw.unpack(f);
  if (w) {
    const float ss = warp_sum(f[0] * f[0] + f[1] * f[1] + f[2] * f[2] + f[3] * f[3]);
    const float rstd = rsqrtf(ss / (float)D + eps);
    const float4 wv = MIXED && !is_q ? pre.wk : pre.wv;
    f[0] = f[0] * rstd * wv.x; f[1] = f[1] * rstd * wv.y; f[2] = f[2] * rstd * wv.z; f[3] = f[3] * rstd * wv.w;
  }
  if (A.inv_freq) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float partner = __shfl_xor_sync(0xffffffffu, f[i], 16);
      f[i] = lane < 16 ? pre.cs[i] * f[i] - pre.sn[i] * partner : pre.sn[i] * partner + pre.cs[i] * f[i];
    }
  }
  RopeRaw<T> res;
  res.pack(f);
  *reinterpret_cast<decltype(res.v)*>(x) = res.v;
  if (!is_q && write_kv) {
    const int slot = pre.slot;
    const int page = (page_size & (page_size - 1)) == 0 ? slot >> (__ffs(page_size) - 1) : slot / page_size;
    *reinterpret_cast<decltype(res.v)*>(pages + ((size_t)slot + ((size_t)page * (2 * Hkv - 1) + h) * page_size) * D + 4 * lane) = res.v;
  }
}
