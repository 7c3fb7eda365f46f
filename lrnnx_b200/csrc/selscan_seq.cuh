// Shared pieces of the state-parallel selective-scan kernels (selscan_seq.cu, selscan_seq_bwd.cu).
#pragma once
#include "common.cuh"
#include "dispatch.h"

namespace b200 {
namespace seq {

constexpr int kSeqBlock = 4;      // steps per block of the backward kernel
constexpr int QN = 16;            // states
constexpr int QS = 4;             // states per lane (two packed pairs)
constexpr int QCH = 8;            // channels per warp: 8 channels x 4 lanes
constexpr int QT = 32;            // timesteps per stage of the serial kernels
constexpr int DROW = 18;          // floats per timestep row of a tile of pairs per channel (16 + 2 of padding)
constexpr int QROW = 36;          // floats per timestep row of a shared tile (32 + 4 of padding)

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2f(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcpf(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 ex2f2(float2 x) { return make_float2(ex2f(x.x), ex2f(x.y)); }

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

// A in units of the binary logarithm.  The steps past the end have a step size of 0 and have to be neutral whatever A is:
// an infinite decay is the largest finite one here (0 times infinity is NaN).
__device__ __forceinline__ float decay2(float A) {
  const float v = A * kLog2e;
  return v < -3.402823466e38f ? -3.402823466e38f : v;
}

// softplus with the reference's pass-through above 20 (selective_scan.cuh:172-174) on two SFU
// operations, and e = exp(x) for its derivative.  log1p(e) is a degree-5 series for e < 1/32
// (relative error < 1e-8) and log(1 + e) above, where the absolute error of the SFU's logarithm
// (2^-22) and of 1 + e no longer matters.
__device__ __forceinline__ float softplus_e(float x, float &e) {
  e = ex2f(x * kLog2e);
  const float series = e * fmaf(e, fmaf(e, fmaf(e, fmaf(e, 0.2f, -0.25f), 0.33333334f), -0.5f), 1.f);
  const float big = lg2f(1.f + e) * 0.6931471805599453f;
  const float y = e < 0.03125f ? series : big;
  return x > 20.f ? x : y;
}
__device__ __forceinline__ float sigm(float x) { return rcpf(1.f + ex2f(-x * kLog2e)); }

// blocks of 4 steps in a sequence, rounded up to whole stages of the serial kernels
__host__ __device__ inline int seq_blocks(int seqlen) { return (seqlen + QT - 1) / QT * (QT / kSeqBlock); }

// ---- 16 bytes of a row at a time
template <typename T> constexpr int EPC = 16 / (int)sizeof(T);          // elements per 16-byte chunk
template <typename T> constexpr int PPR = QT / EPC<T>;                  // chunks per row of a stage
template <typename T> constexpr int CPL = QCH * PPR<T> / 32;            // chunks per lane of a warp's 8 rows

// every row of a (batch, rows, steps) tensor starts on a 16-byte boundary
template <typename T> inline bool row16(const void *ptr, int64_t bs, int64_t ds) {
  return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && bs % EPC<T> == 0 && ds % EPC<T> == 0;
}

// the first `valid` elements at p (the rest 0); `al`: p is 16-byte aligned
template <typename T> __device__ __forceinline__ uint4 ld_chunk(const T *p, int valid, bool al) {
  if (al && valid >= EPC<T>) return *reinterpret_cast<const uint4 *>(p);
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (valid > j) w[j] = __float_as_uint(p[j]);
  } else {
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (valid > j) w[j >> 1] |= (uint32_t)h[j] << (16 * (j & 1));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// the first `valid` of the 16 bytes' elements to p, which is 16-byte aligned
template <typename T> __device__ __forceinline__ void st_chunk(T *p, uint4 v, int valid) {
  if (valid >= EPC<T>) { *reinterpret_cast<uint4 *>(p) = v; return; }
  const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
  for (int j = 0; j < EPC<T>; ++j)
    if (valid > j) p[j] = e[j];
}
__device__ __forceinline__ void unpack(const uint4 &v, float (&o)[4], float) {
  o[0] = __uint_as_float(v.x); o[1] = __uint_as_float(v.y); o[2] = __uint_as_float(v.z); o[3] = __uint_as_float(v.w);
}
template <typename T> __device__ __forceinline__ void unpack(const uint4 &v, float (&o)[8], T) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const T *h = reinterpret_cast<const T *>(&w[i]);
    o[2 * i] = to_f(h[0]);
    o[2 * i + 1] = to_f(h[1]);
  }
}
__device__ __forceinline__ void cp16(void *smem_dst, const void *gsrc, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(src_bytes)
               : "memory");
}
// four states of two neighbouring blocks: one whole 32-byte sector in one store
__device__ __forceinline__ void st_states(float4 *p, float2 a0, float2 a1, float2 b0, float2 b1) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a0.x), "f"(a0.y), "f"(a1.x), "f"(a1.y), "f"(b0.x),
               "f"(b0.y), "f"(b1.x), "f"(b1.y)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A lane's share of 8 rows x 32 steps of an operand: CPL chunks of 16 bytes, in rows lane / PPR (and + 4).
template <typename T> struct RowCopy {
  const T *p;            // the lane's first chunk in the current stage
  const T *safe;         // a mapped address for copies of 0 bytes
  int64_t ds4;           // 4 rows further (second chunk of a lane, 32-bit types)
  __device__ __forceinline__ void init(const void *base, int64_t bs, int64_t ds, int b, int d, int lane, int nch, int t) {
    const int row = lane / PPR<T>, r = row < nch ? row : 0;
    p = reinterpret_cast<const T *>(base) + (int64_t)b * bs + (int64_t)(d + r) * ds + t + (lane % PPR<T>) * EPC<T>;
    safe = reinterpret_cast<const T *>(base);
    ds4 = 4 * ds;
  }
  // left: steps from the lane's chunk to the end of the sequence; what lies past it is filled with zeros
  __device__ __forceinline__ void fetch(unsigned char *dst, int lane, int nch, int left) const {
    const int row = lane / PPR<T>;
    const int n = left <= 0 ? 0 : (left >= EPC<T> ? 16 : left * (int)sizeof(T));
#pragma unroll
    for (int k = 0; k < CPL<T>; ++k) {
      const bool ok = row + 4 * k < nch && n > 0;
      cp16(dst + (lane + 32 * k) * 16, ok ? p + k * ds4 : safe, ok ? n : 0);
    }
  }
};

}  // namespace seq

}  // namespace b200
