// S4 structured kernels for sm_100a: symmetric Cauchy multiply and log-Vandermonde
// multiply, forward and backward.
//
// Math (csrc/s4/cauchy_cuda.cu:68-79,144-170,211-331 of lrnnx), n = half spectrum:
//   cauchy  out[b,l] = sum_n v/(z_l - w) + conj(v)/(z_l - conj(w))
//           dv[b,n]  = sum_l dout/(conj(z) - conj(w)) + conj(dout)/(z - conj(w))
//           dw[b,n]  = conj(v) sum_l dout/(conj(z) - conj(w))^2 + conj(dout)/(z - conj(w))^2
//   vand    out[b,l] = 2 Re sum_n v exp(x l)
//           dv[b,n]  = 2 sum_l dout conj(exp(x l));  dx[b,n] = 2 conj(v) sum_l dout l conj(exp(x l))
//
// These kernels are bound by the fp32 pipe (two complex reciprocals, or one complex
// exponential, per (b, l, n)), not by memory.  Forward: one thread owns FL output
// positions and loops over n with (v, w) broadcast from shared memory, so there is no
// cross-thread reduction.  Backward: a CTA owns (batch row, tile of TN poles, chunk of
// the sequence); threads stride over the chunk with TN complex accumulators each; CTA
// partials go to a scratch buffer and a second kernel folds the chunks in order.
#include "common.cuh"
#include <atomic>
#include "dispatch.h"

namespace b200 {
namespace {

constexpr int FT = 256;       // forward threads
constexpr int CT = 128;       // forward threads (Cauchy)
constexpr int FL = 4;         // output positions per thread (Cauchy), CT apart: two packed pairs
constexpr int VFL = 8;        // output positions per thread (Vandermonde), FT apart
constexpr int NMAX_SMEM = 1024;
constexpr int BTT = 256;      // backward threads
constexpr int TN = 4;         // poles per backward CTA
constexpr int BWARPS_ = BTT / 32;

// Reciprocals of squared moduli by the SFU (max. error 1 ulp) instead of an IEEE division.
__device__ __forceinline__ float2 rcp2(float2 m) {
  float2 r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(m.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(m.y));
  return r;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }

// Both terms of a conjugate pair share the real part dr of z - w and z - conj(w); with e1 = zi - wi, e2 = zi + wi
//     v / (z - w) + conj(v) / (z - conj(w)) = v (dr, -e1) / (dr^2 + e1^2) + conj(v) (dr, -e2) / (dr^2 + e2^2)
// are 18 fp32 operations beside two reciprocals (16 cycles of the SFU); as two complex reciprocals and products they
// were 24.  The reciprocals' parts are added before they meet v: an output's running sum is then rounded twice per pole and
// part, an error of 1.7e-7 (four chained multiply-adds: 2.4e-7, at the same number of operations).  The two reciprocals stay two (a common denominator would cancel near the poles), and v multiplies the
// finished reciprocal (v dr could overflow where the quotient does not).  Two positions per packed instruction halve
// the issue slots.  1024 rows, 32 poles, L = 4096: 117 -> 79 us (67 us are the fp32 pipe's floor, 58 the SFU's).
__global__ void __launch_bounds__(CT) cauchy_fwd_kernel(const cf *__restrict__ v, const cf *__restrict__ z,
                                                        const cf *__restrict__ w, cf *__restrict__ out, int n, int L) {
  __shared__ float4 vw[NMAX_SMEM];
  const int b = blockIdx.y;
  const int l0 = blockIdx.x * CT * FL + threadIdx.x;
  float2 zr[FL / 2], zi[FL / 2], ar[FL / 2], ai[FL / 2];
#pragma unroll
  for (int j = 0; j < FL / 2; ++j) {
    const int la = l0 + 2 * j * CT, lb = la + CT;
    const cf za = la < L ? z[la] : cf(2.f, 0.f), zb = lb < L ? z[lb] : cf(2.f, 0.f);
    zr[j] = make_float2(za.re, zb.re);
    zi[j] = make_float2(za.im, zb.im);
    ar[j] = ai[j] = make_float2(0.f, 0.f);
  }
  for (int nb = 0; nb < n; nb += NMAX_SMEM) {
    const int cnt = min(NMAX_SMEM, n - nb);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += CT) {
      const cf vv = v[(int64_t)b * n + nb + i], ww = w[(int64_t)b * n + nb + i];
      vw[i] = make_float4(vv.re, vv.im, ww.re, ww.im);
    }
    __syncthreads();
#pragma unroll 4
    for (int i = 0; i < cnt; ++i) {
      const float4 t = vw[i];
#pragma unroll
      for (int j = 0; j < FL / 2; ++j) {
        const float2 dr = add2(zr[j], both(-t.z)), e1 = add2(zi[j], both(-t.w)), e2 = add2(zi[j], both(t.w));
        const float2 dd = mul2(dr, dr);
        const float2 r1 = rcp2(fma2(e1, e1, dd)), r2 = rcp2(fma2(e2, e2, dd));
        const float2 r1r = mul2(dr, r1), r1n = mul2(e1, r1), r2r = mul2(dr, r2), r2n = mul2(e2, r2);
        ar[j] = fma2(both(t.x), add2(r1r, r2r), fma2(both(t.y), sub2(r1n, r2n), ar[j]));
        ai[j] = fma2(both(t.y), sub2(r1r, r2r), fma2(both(-t.x), add2(r1n, r2n), ai[j]));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < FL / 2; ++j) {
    const int la = l0 + 2 * j * CT, lb = la + CT;
    if (la < L) out[(int64_t)b * L + la] = cf(ar[j].x, ai[j].x);
    if (lb < L) out[(int64_t)b * L + lb] = cf(ar[j].y, ai[j].y);
  }
}

__global__ void __launch_bounds__(FT) vand_fwd_kernel(const cf *__restrict__ v, const cf *__restrict__ x,
                                                      float *__restrict__ out, int n, int L) {
  // A thread owns VFL positions l0, l0 + FT, ...: exp(x l) is evaluated exactly at l0 and advanced
  // by the per-pole constant exp(x FT) (a complex multiply instead of an exp and a sin/cos per term).
  __shared__ float4 vx[NMAX_SMEM];
  __shared__ float2 wstep[NMAX_SMEM];
  const int b = blockIdx.y;
  const int l0 = blockIdx.x * FT * VFL + threadIdx.x;
  const float lf = (float)l0;
  float acc[VFL];
#pragma unroll
  for (int j = 0; j < VFL; ++j) acc[j] = 0.f;
  for (int nb = 0; nb < n; nb += NMAX_SMEM) {
    const int cnt = min(NMAX_SMEM, n - nb);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += FT) {
      const cf vv = v[(int64_t)b * n + nb + i], xx = x[(int64_t)b * n + nb + i];
      vx[i] = make_float4(vv.re, vv.im, xx.re, xx.im);
      const cf w = cexp(xx * (float)FT);
      wstep[i] = make_float2(w.re, w.im);
    }
    __syncthreads();
#pragma unroll 2
    for (int i = 0; i < cnt; ++i) {
      const float4 t = vx[i];
      const float2 ws = wstep[i];
      const cf xx(t.z, t.w), W(ws.x, ws.y);
      cf E = cexp(xx * lf) * cf(t.x, t.y);      // v exp(x l0)
#pragma unroll
      for (int j = 0; j < VFL; ++j) {
        acc[j] += E.re;
        E = E * W;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < VFL; ++j) {
    const int l = l0 + j * FT;
    if (l < L) out[(int64_t)b * L + l] = 2.f * acc[j];
  }
}

// Partial sums of one (batch row, pole tile, sequence chunk).  scratch layout:
// [batch][n][n_chunks][2] complex (first: dv partial, second: dw / dx partial).
template <bool VAND>
__global__ void __launch_bounds__(BTT) s4_bwd_partial_kernel(const cf *__restrict__ z, const cf *__restrict__ w,
                                                             const void *__restrict__ dout_, cf *__restrict__ scratch,
                                                             int n, int L, int l_chunk, int n_chunks) {
  __shared__ cf red[2 * TN][BWARPS_];
  const int b = blockIdx.z, chunk = blockIdx.y, n0 = blockIdx.x * TN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cf wn[TN];
#pragma unroll
  for (int k = 0; k < TN; ++k) wn[k] = (n0 + k < n) ? w[(int64_t)b * n + n0 + k] : cf(3.f, 3.f);
  cf a1[TN], a2[TN];
#pragma unroll
  for (int k = 0; k < TN; ++k) { a1[k] = cf(0.f, 0.f); a2[k] = cf(0.f, 0.f); }
  const int lbeg = chunk * l_chunk, lend = min(L, lbeg + l_chunk);
  // Vandermonde: exp(w l) advanced by the per-pole constant exp(w BTT) between the positions of
  // a thread (BTT apart), re-evaluated exactly every 16 positions
  cf Ek[TN], Wk[TN];
  if constexpr (VAND) {
#pragma unroll
    for (int k = 0; k < TN; ++k) Wk[k] = cexp(wn[k] * (float)BTT);
  }
  if constexpr (!VAND) {
    // Positions l and l + BTT packed.  With dr, e1, e2 as in the forward and g = dout
    //     s1 = g (dr, e1) / m1,  s2 = conj(g) (dr, -e2) / m2,   dv += s1 + s2
    //     dw += s1 (dr, e1) / m1 + s2 (dr, -e2) / m2
    // 34 fp32 operations and two reciprocals; the terms are formed before they are added.  1024 rows, 32 poles, L = 4096:
    // 227 -> 182 us (127 us are the fp32 pipe's floor).
    float2 b1r[TN], b1i[TN], b2r[TN], b2i[TN];
#pragma unroll
    for (int k = 0; k < TN; ++k) b1r[k] = b1i[k] = b2r[k] = b2i[k] = make_float2(0.f, 0.f);
    const cf *dp = reinterpret_cast<const cf *>(dout_) + (int64_t)b * L;
    for (int l = lbeg + threadIdx.x; l < lend; l += 2 * BTT) {
      const bool two = l + BTT < lend;
      const cf ga = dp[l], za = z[l];
      const cf gb = two ? dp[l + BTT] : cf(0.f, 0.f), zb = two ? z[l + BTT] : za;
      const float2 gr = make_float2(ga.re, gb.re), gi = make_float2(ga.im, gb.im);
      const float2 zr = make_float2(za.re, zb.re), zi = make_float2(za.im, zb.im);
#pragma unroll
      for (int k = 0; k < TN; ++k) {
        const float2 dr = add2(zr, both(-wn[k].re)), e1 = add2(zi, both(-wn[k].im)), e2 = add2(zi, both(wn[k].im));
        const float2 dd = mul2(dr, dr);
        const float2 i1 = rcp2(fma2(e1, e1, dd)), i2 = rcp2(fma2(e2, e2, dd));
        const float2 r1r = mul2(dr, i1), r1i = mul2(e1, i1), r2r = mul2(dr, i2), r2n = mul2(e2, i2);     // r2 = (r2r, -r2n)
        const float2 m = make_float2(-1.f, -1.f);
        const float2 gin = mul2(gi, m);
        const float2 s1r = fma2(gin, r1i, mul2(gr, r1r)), s1i = fma2(gr, r1i, mul2(gi, r1r));
        const float2 s2r = fma2(gin, r2n, mul2(gr, r2r)), s2n = fma2(gr, r2n, mul2(gi, r2r));            // s2 = (s2r, -s2n)
        b1r[k] = add2(b1r[k], add2(s1r, s2r));
        b1i[k] = add2(b1i[k], fma2(s2n, m, s1i));
        const float2 tr = fma2(s2r, r2r, mul2(s1r, r1r)), ur = fma2(s2n, r2n, mul2(s1i, r1i));
        const float2 ti = fma2(s1i, r1r, mul2(s1r, r1i)), ui = fma2(s2r, r2n, mul2(s2n, r2r));
        b2r[k] = add2(b2r[k], fma2(ur, m, tr));
        b2i[k] = add2(b2i[k], fma2(ui, m, ti));
      }
    }
#pragma unroll
    for (int k = 0; k < TN; ++k) {
      a1[k] = cf(b1r[k].x + b1r[k].y, b1i[k].x + b1i[k].y);
      a2[k] = cf(b2r[k].x + b2r[k].y, b2i[k].x + b2i[k].y);
    }
  } else {
    int iter = 0;
    for (int l = lbeg + threadIdx.x; l < lend; l += BTT, ++iter) {
      const float d = reinterpret_cast<const float *>(dout_)[(int64_t)b * L + l];
      const float lf = (float)l;
      const bool exact = (iter & 15) == 0;
#pragma unroll
      for (int k = 0; k < TN; ++k) {
        Ek[k] = exact ? cexp(wn[k] * lf) : Ek[k] * Wk[k];
        const cf e = conj(Ek[k]) * d;
        a1[k] = a1[k] + e;
        a2[k] = a2[k] + e * lf;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < TN; ++k) {
    a1[k] = warp_sum(a1[k]);
    a2[k] = warp_sum(a2[k]);
    if (lane == 0) { red[2 * k][warp] = a1[k]; red[2 * k + 1][warp] = a2[k]; }
  }
  __syncthreads();
  if (threadIdx.x < 2 * TN) {
    cf s = cf(0.f, 0.f);
#pragma unroll
    for (int wv = 0; wv < BWARPS_; ++wv) s = s + red[threadIdx.x][wv];
    const int k = threadIdx.x >> 1, which = threadIdx.x & 1;
    if (n0 + k < n) scratch[(((int64_t)b * n + n0 + k) * n_chunks + chunk) * 2 + which] = s;
  }
}

template <bool VAND>
__global__ void s4_bwd_fold_kernel(const cf *__restrict__ v, const cf *__restrict__ scratch, cf *__restrict__ dv,
                                   cf *__restrict__ dw, int64_t total, int n_chunks) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  cf s1 = cf(0.f, 0.f), s2 = cf(0.f, 0.f);
  for (int c = 0; c < n_chunks; ++c) {
    s1 = s1 + scratch[(i * n_chunks + c) * 2];
    s2 = s2 + scratch[(i * n_chunks + c) * 2 + 1];
  }
  if (VAND) { s1 = s1 * 2.f; s2 = s2 * 2.f; }
  dv[i] = s1;
  dw[i] = conj(v[i]) * s2;
}

int chunking(int batch, int n, int L, int &l_chunk) {
  const int64_t tiles = (int64_t)batch * ((n + TN - 1) / TN);
  int want = (int)((sm_count_current() * 4 + tiles - 1) / tiles);          // enough CTAs to fill the GPU
  const int max_chunks = (L + 1023) / 1024;                 // at least 1024 positions per CTA
  if (want > max_chunks) want = max_chunks;
  if (want < 1) want = 1;
  l_chunk = (L + want - 1) / want;
  l_chunk = ((l_chunk + BTT - 1) / BTT) * BTT;
  return (L + l_chunk - 1) / l_chunk;
}

int check(const b200_s4_args &a, bool bwd, bool vand) {
  B200_REQUIRE(a.v && a.w && (vand || a.z), B200_ERR_NULL, "s4: v, z, w must be non-null");
  B200_REQUIRE(a.batch > 0 && a.n > 0 && a.seqlen > 0, B200_ERR_SHAPE, "s4: batch, n, seqlen must be positive");
  B200_REQUIRE(a.batch <= 65535, B200_ERR_SHAPE, "s4: batch must be <= 65535");
  if (!bwd) {
    B200_REQUIRE(a.out, B200_ERR_NULL, "s4: out must be non-null");
  } else {
    B200_REQUIRE(a.dout && a.dv && a.dw && a.scratch, B200_ERR_NULL, "s4: dout, dv, dw, scratch must be non-null");
    B200_REQUIRE(a.scratch_bytes >= b200_s4_bwd_scratch_bytes(a.batch, a.n, a.seqlen), B200_ERR_SHAPE,
                 "s4: scratch too small (%lld bytes, need %lld)", (long long)a.scratch_bytes,
                 (long long)b200_s4_bwd_scratch_bytes(a.batch, a.n, a.seqlen));
  }
  return 0;
}

template <bool VAND> int run_bwd(const b200_s4_args &a, cudaStream_t st) {
  int l_chunk;
  const int n_chunks = chunking(a.batch, a.n, a.seqlen, l_chunk);
  dim3 grid((a.n + TN - 1) / TN, n_chunks, a.batch);
  s4_bwd_partial_kernel<VAND><<<grid, BTT, 0, st>>>(
      reinterpret_cast<const cf *>(a.z), reinterpret_cast<const cf *>(a.w), a.dout,
      reinterpret_cast<cf *>(a.scratch), a.n, a.seqlen, l_chunk, n_chunks);
  if (int e = launch_status()) return e;
  const int64_t total = (int64_t)a.batch * a.n;
  s4_bwd_fold_kernel<VAND><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
      reinterpret_cast<const cf *>(a.v), reinterpret_cast<const cf *>(a.scratch), reinterpret_cast<cf *>(a.dv),
      reinterpret_cast<cf *>(a.dw), total, n_chunks);
  return launch_status();
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int64_t b200_s4_bwd_scratch_bytes(int32_t batch, int32_t n, int32_t seqlen) {
  if (batch <= 0 || n <= 0 || seqlen <= 0) return 0;
  int l_chunk;
  const int n_chunks = chunking(batch, n, seqlen, l_chunk);
  return (int64_t)batch * n * n_chunks * 2 * (int64_t)sizeof(cf);
}

int b200_cauchy_fwd(const b200_s4_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "cauchy_fwd: null argument block");
  if (int e = check(*args, false, false)) return e;
  dim3 grid((args->seqlen + CT * FL - 1) / (CT * FL), args->batch);
  cauchy_fwd_kernel<<<grid, CT, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const cf *>(args->v), reinterpret_cast<const cf *>(args->z),
      reinterpret_cast<const cf *>(args->w), reinterpret_cast<cf *>(args->out), args->n, args->seqlen);
  return launch_status();
}

int b200_cauchy_bwd(const b200_s4_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "cauchy_bwd: null argument block");
  if (int e = check(*args, true, false)) return e;
  return run_bwd<false>(*args, reinterpret_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Cauchy backward without any allocation by anybody.
//
// Some users of this library cannot hand it device memory beyond the tensors of
// the call: a plain C or C++ host that links the ABI without a framework
// allocator, or a serving loop that runs under a frozen memory budget where a
// cudaMalloc (which may synchronise the device or fail late) is not acceptable.
// For them the per-chunk partial sums live in a fixed array inside the library
// image.  Every GPU that loads the library holds the array until the process
// exits; its size bounds the problem size.
static __device__ __align__(256) unsigned char g_cauchy_static_scratch[B200_CAUCHY_STATIC_SCRATCH_BYTES];

// In host code the array's name is only a handle; the device address has to be
// asked for, per device, with that device current.
static std::atomic<void *> g_static_scratch_ptr[64];

static int static_scratch_for_current_device(void **out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { set_error("cudaGetDevice: %s", cudaGetErrorString(e)); return (int)e; }
  B200_REQUIRE(dev >= 0 && dev < 64, B200_ERR_UNSUPPORTED, "cauchy_bwd_static: device ordinal %d not supported", dev);
  void *ptr = g_static_scratch_ptr[dev].load(std::memory_order_acquire);
  if (!ptr) {
    e = cudaGetSymbolAddress(&ptr, g_cauchy_static_scratch);
    if (e != cudaSuccess || !ptr) {
      set_error("cudaGetSymbolAddress(static scratch): %s", cudaGetErrorString(e));
      return e != cudaSuccess ? (int)e : B200_ERR_UNSUPPORTED;
    }
    g_static_scratch_ptr[dev].store(ptr, std::memory_order_release);   // same value from every thread
  }
  *out = ptr;
  return 0;
}

int b200_cauchy_bwd_static(const b200_s4_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "cauchy_bwd_static: null argument block");
  const int64_t need = b200_s4_bwd_scratch_bytes(args->batch, args->n, args->seqlen);
  B200_REQUIRE(need <= (int64_t)B200_CAUCHY_STATIC_SCRATCH_BYTES, B200_ERR_TOO_LARGE,
               "cauchy_bwd_static: this problem needs %lld bytes of scratch, the built-in area holds %lld; "
               "use b200_cauchy_bwd with caller-provided scratch",
               (long long)need, (long long)B200_CAUCHY_STATIC_SCRATCH_BYTES);
  b200_s4_args a = *args;
  void *ptr = nullptr;
  if (int e = static_scratch_for_current_device(&ptr)) return e;
  a.scratch = ptr;
  a.scratch_bytes = B200_CAUCHY_STATIC_SCRATCH_BYTES;
  if (int e = check(a, true, false)) return e;
  // Nothing in the area has to start at zero: the first kernel writes every partial-sum slot
  // that the second kernel reads.
  return run_bwd<false>(a, reinterpret_cast<cudaStream_t>(stream));
}

int b200_vand_fwd(const b200_s4_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "vand_fwd: null argument block");
  if (int e = check(*args, false, true)) return e;
  dim3 grid((args->seqlen + FT * VFL - 1) / (FT * VFL), args->batch);
  vand_fwd_kernel<<<grid, FT, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const cf *>(args->v), reinterpret_cast<const cf *>(args->w),
      reinterpret_cast<float *>(args->out), args->n, args->seqlen);
  return launch_status();
}

int b200_vand_bwd(const b200_s4_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "vand_bwd: null argument block");
  if (int e = check(*args, true, true)) return e;
  return run_bwd<true>(*args, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
