// Complex projections around the S5 scan on the 5th-generation tensor cores (tcgen05 + TMEM):
//     out[b] (M x N) = W (M x K) * X[b] (K x N),      complex64, N contiguous,
// the shape of  Bu = B~ u,  y = C~ x  and of the two data gradients  du = B~^H dBu,  dx = C~^H dy
// of lrnnx's simplified_scan_fn / s5_inner_fn (lrnnx/ops/simplified_scan.py:67,87,136,165,401,419,
// 483-524), which lrnnx evaluates with torch.einsum (cuBLAS SIMT cgemm).
//
// Arithmetic.  With X' the (K x 2N) float view of X (re/im interleaved along N),
//     D1 = Re(W) X',   D2 = Im(W) X'     (two real GEMMs sharing the activation tile)
//     out_re[n] = D1[2n] - D2[2n+1],   out_im[n] = D1[2n+1] + D2[2n]
// so the activation is consumed exactly as it lies in memory and only the small weight is split
// into planes.  fp32-class accuracy on TF32 tensor cores comes from the 3xTF32 split
//     a b ~= a_hi b_hi + a_lo b_hi + a_hi b_lo,   x_hi = tf32(x), x_lo = tf32(x - x_hi),
// i.e. six tcgen05.mma per K step.  The weight planes (Re hi, Re lo, Im hi, Im lo) are prepared
// once per call on the host side; the low part of the activation tile is produced inside the
// kernel, in shared memory: it is elementwise, so it is written at the same (swizzled) offsets the
// TMA used for the tile and no layout knowledge is needed.
//
// The tensor core truncates when it adds into its float32 accumulator, an error to one side that
// grows with the length of the chain (4e-6 of the result at K = 512).  So an accumulator lives for
// two stages (32 floats of K) only: in each the small products go in first, then two large ones, and
// the sums of a chain are added up in registers, rounded to nearest, by warps of their own.  Two sets
// of accumulators alternate, so the next chain's products do not wait.  What truncation takes on average is
// given back (a share of 1.3e-7 or less, see below): an error to one side adds up over the scan that follows,
// and sums of positive terms only lose twice that.  Error against 64 bits 1.7e-7 at K = 96, 2.0e-7 at
// K = 1024 (a float32 cuBLAS cgemm with a real x: 1.8e-7 and 4.1e-7).  Chains of one stage would be 10 %
// slower, chains of the whole K 20 times less exact and no faster.
//
// Persistent thread blocks take 128 x 64-complex output tiles in turn: warp 0 issues the TMA loads
// (64-byte swizzled weight tiles, 4-stage ring on mbarriers), warp 1 allocates 512 TMEM columns and
// issues the MMAs, warps 4-7 split the activation tiles, warps 8-15 add up the chains and store.
// The activation is the 128-row operand (MN-major, 128-byte swizzle of 32-byte chunks) and Re(W) over
// Im(W) the 256-row one: an instruction of N = 256 reads half as much shared memory per product as two of
// N = 128 (180 -> 160 us at 8 x 256 x 512 x 4096), and a TMEM lane is a float column of X, so
// the stores are coalesced.  Sizes are free: the weight planes are padded with zeros to the tiles, the
// tensor maps fill with zeros past K and N, and the stores stop at M and N; only the row pitch of x has to
// be a multiple of 16 bytes.  The split of an infinity is no sum (infinity times a zero or opposite low part is
// NaN): outputs that come out as NaN are formed once more by the plain complex sum.  Every mbarrier wait is bounded; an expired wait sets the status word, skips
// the stores and still frees the TMEM.
#include "common.cuh"
#include "dispatch.h"
#include "tc_common.cuh"
#include <cstring>

namespace b200 {
namespace {

using namespace tc;

__device__ int g_cgemm_status = 0;

constexpr int GM = 128;               // weight rows per CTA
constexpr int GN = 128;               // activation floats per CTA (64 complex columns)
constexpr int GK = 16;                // floats of K per stage: one 64-byte swizzle row
constexpr int KPAD = 32;              // the weight planes' K is padded to a multiple of this
constexpr int NSTAGE = 4;
constexpr int TILE = GM * GK * 4;     // 8 KB: a weight-plane tile; an activation tile has the same size
constexpr int STAGE_BYTES = 6 * TILE; // Re hi, Re lo, Im hi, Im lo, X hi, X lo
constexpr int TX_BYTES = 5 * TILE;    // what the TMA delivers per stage (X lo is produced in place)
constexpr int PS = 2;                 // stages per accumulation chain
// Below this K the small products of both stages of a chain go in before the large ones of either: error 1.4e-7
// instead of 1.8e-7 (of a float32 cuBLAS product with a real x at K = 64 and 96), for up to 4 % more time.
constexpr int SHORT_K = 160;
// What truncation takes from a chain, as a share of a sum of random signs (measured against 64 bits, the same at all
// sizes); the weights' low planes are that much larger, the gradient's sums are scaled
__host__ __device__ constexpr float lost(int K) { return K < SHORT_K ? 4.3e-8f : 1.3e-7f; }
constexpr float kLostGrad = 2.3e-7f;  // with what the product of two truncated low parts would have added
constexpr int NTHREADS = 512;
constexpr int TMEM_COLS = 512;        // two sets of two 128-column accumulators
constexpr uint32_t WAIT_LIMIT = 1u << 24;

struct GemmMaps {
  CUtensorMap w;      // (Kp, 4 Mp) float32, box (16, 128): M, K padded to the tiles
  CUtensorMap x;      // (2 N, K, batch) float32, box (32, 16, 1)
};

// weight-plane tile, K-major: rows of 64 bytes, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t k_desc(uint32_t addr) { return smem_desc(addr, 16, 512, 4); }
// activation tile, MN-major: 32-float column groups 2048 bytes apart, 4-row K groups 512 bytes apart
__device__ __forceinline__ uint64_t x_desc(uint32_t addr) { return smem_desc(addr, GK * 128, 512, 1); }
// instruction descriptor: D f32, A and B tf32, A MN-major (the activation), B K-major (256 weight rows), M = 128, N = 256
constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 15) | ((2 * GN >> 3) << 17) | ((GM >> 4) << 24);

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate,
                                         uint32_t idesc = kIdesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0)
      : "memory");
}
// The tensor core truncates a 32-bit operand to TF32, so the high part of x is what it reads from
// the tile as it is; the low part x - trunc(x) is exact in float32 and is rounded to the nearest
// TF32 here (the hardware would truncate it, a one-sided error that adds up over K).  Of an infinity the low part is a
// zero: inf - inf is the canonical NaN 0x7fffffff, which the rounding carries over into -0.
__device__ __forceinline__ float tf32_low(float v) {
  const float r = v - __uint_as_float(__float_as_uint(v) & 0xffffe000u);
  return __uint_as_float((__float_as_uint(r) + 0x1000u) & 0xffffe000u);
}
// What the two kernels share: barriers and the accumulators' two sets.
struct Pipe {
  uint64_t full[NSTAGE], empty[NSTAGE], lo_ready[NSTAGE];      // stage loaded / free again / split
  uint64_t acc_full[2], acc_empty[2];                          // accumulator set complete / read
  uint32_t tmem_base;
  int fail;
  int nan;                                                     // some output came out as NaN
};
__device__ __forceinline__ void pipe_init(Pipe &p, int sum_warps) {
  for (int s = 0; s < NSTAGE; ++s) {
    mbar_init(&p.full[s], 1);
    mbar_init(&p.empty[s], 1);
    mbar_init(&p.lo_ready[s], 4);            // one arrival per splitting warp
  }
  for (int s = 0; s < 2; ++s) {
    mbar_init(&p.acc_full[s], 1);
    mbar_init(&p.acc_empty[s], sum_warps);
  }
  p.fail = 0;
  p.nan = 0;
  mbar_fence_init();
  fence_proxy_async();
}
// n-th use (from 0) of a resource that the other side gives back: the first `free` uses do not wait
__device__ __forceinline__ bool wait_given_back(uint64_t *bar, int n, int slots) {
  return n < slots || mbar_wait(bar, ((n / slots) - 1) & 1, WAIT_LIMIT);
}

template <int R> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// The outputs that a thread has stored as NaN in float column `col` of the GM / 2 rows from m0 on, as plain sums.
__device__ __forceinline__ void plain_tile(const b200_cgemm_args &p, int mt, int m0, int col, int b) {
  if (col >= 2 * p.N) return;
  const int Kp = (p.K + KPAD - 1) / KPAD * KPAD, rows = min(p.M - m0, GM / 2);
  const int64_t plane = (int64_t)mt * GM * Kp;
  const float2 *x = reinterpret_cast<const float2 *>(p.x) + (int64_t)b * p.x_bs + (col >> 1);
  float *orow = reinterpret_cast<float *>(p.out) + ((int64_t)b * p.out_bs + (int64_t)m0 * p.out_ms) * 2 + col;
  for (int i = 0; i < rows; ++i) {
    const float was = orow[(int64_t)i * p.out_ms * 2];
    if (was == was) continue;
    const float *w = reinterpret_cast<const float *>(p.w_planes) + (int64_t)(m0 + i) * Kp;
    float s = 0.f;
    for (int k0 = 0; k0 < p.K && s == s; k0 += 8) {        // a NaN stays one
#pragma unroll
      for (int k = k0; k < k0 + 8; ++k) {
        const float wr = w[k] + w[plane + k], wi = w[2 * plane + k] + w[3 * plane + k];      // the planes reach to Kp
        const float2 v = k < p.K ? x[(int64_t)k * p.x_ks] : make_float2(0.f, 0.f);
        s = (col & 1) ? fmaf(wr, v.y, fmaf(wi, v.x, s)) : fmaf(wr, v.x, fmaf(-wi, v.y, s));
      }
    }
    orow[(int64_t)i * p.out_ms * 2] = s;
  }
}

__global__ void __launch_bounds__(NTHREADS, 1)
cgemm_wx_kernel(const __grid_constant__ GemmMaps maps, const b200_cgemm_args p, const int mt, const int nt, const int nk) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment of the tiles (the swizzle atom) is established by hand: the dynamic
  // shared-memory base is only guaranteed to be 16-byte aligned
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ Pipe pipe;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = mt * nt * p.batch;         // rows of the weight fastest: neighbours share the activation tile
  if (tid == 0) pipe_init(pipe, 8);
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&pipe.tmem_base)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = pipe.tmem_base;

  // Registers: 512 threads are launched with 128 each; 48 + 56 + 2 x 200 = 504 of the four shares of 128 are used
  if (warp < 4) {
    regs_dec<48>();
    if (warp == 0 && lane == 0) {
    // ------------------------------------------------------------------ TMA producer
      int g = 0;                               // stages so far
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const int m0 = t % mt * GM, n0 = t / mt % nt * GN, b = t / (mt * nt);
        for (int ks = 0; ks < nk; ++ks, ++g) {
          const int s = g % NSTAGE;
          if (!wait_given_back(&pipe.empty[s], g, NSTAGE)) { ok = false; break; }
          unsigned char *st = smem + (size_t)s * STAGE_BYTES;
          mbar_expect_tx(&pipe.full[s], TX_BYTES);
          const int k0 = ks * GK;
#pragma unroll
          for (int pl = 0; pl < 4; ++pl)        // tiles Re hi | Im hi | Re lo | Im lo, planes Re hi, Re lo, Im hi, Im lo
            tma_2d(st + pl * TILE, &maps.w, k0, ((pl & 1) * 2 + (pl >> 1)) * mt * GM + m0, &pipe.full[s]);
#pragma unroll
          for (int j = 0; j < GN / 32; ++j) tma_3d(st + 4 * TILE + j * GK * 128, &maps.x, n0 + 32 * j, k0, b, &pipe.full[s]);
        }
      }
      if (!ok) atomicExch(&pipe.fail, 1);
    } else if (warp == 1 && lane == 0) {
    // ------------------------------------------------------------------ MMA issuer
      int g = 0, ch = 0;                       // stages, chains so far
      bool ok = true;
      const bool small_first = p.K < SHORT_K;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        for (int ks = 0; ks < nk && ok; ks += PS, ++ch) {
          const int n = min(PS, nk - ks);       // stages of this chain
          const uint32_t d = tmem_base + (ch & 1) * 2 * GN;       // columns: 128 of Re(W) X', 128 of Im(W) X'
          const auto large = [&](int s) {
            const uint32_t st = smem_u32(smem + (size_t)s * STAGE_BYTES);
#pragma unroll
            for (int kk = 0; kk < GK / 8; ++kk) mma_tf32(d, x_desc(st + 4 * TILE + kk * 1024), k_desc(st + 0 * TILE + kk * 32), 1u);
            mma_commit(&pipe.empty[s]);         // the stage may be refilled once these MMAs have read it
          };
          if (!wait_given_back(&pipe.acc_empty[ch & 1], ch, 2)) { ok = false; break; }
          for (int i = 0; i < n; ++i) {
            const int s = (g + i) % NSTAGE;
            const uint32_t ph = ((g + i) / NSTAGE) & 1;
            if (!mbar_wait(&pipe.full[s], ph, WAIT_LIMIT) || !mbar_wait(&pipe.lo_ready[s], ph, WAIT_LIMIT)) { ok = false; break; }
            tc_fence_after();
            // the small products first: what is truncated while they add up is small as well
            const uint32_t st = smem_u32(smem + (size_t)s * STAGE_BYTES);
#pragma unroll
            for (int kk = 0; kk < GK / 8; ++kk) {
              mma_tf32(d, x_desc(st + 5 * TILE + kk * 1024), k_desc(st + 0 * TILE + kk * 32), kk > 0 || i > 0 ? 1u : 0u);
              mma_tf32(d, x_desc(st + 4 * TILE + kk * 1024), k_desc(st + 2 * TILE + kk * 32), 1u);
            }
            if (!small_first) large(s);
          }
          if (!ok) break;
          if (small_first)
            for (int i = 0; i < n; ++i) large((g + i) % NSTAGE);
          g += n;
          mma_commit(&pipe.acc_full[ch & 1]);
        }
      }
      if (!ok) atomicExch(&pipe.fail, 1);
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ activation split
    regs_dec<56>();
    const int et = tid - 128;                   // 0..127
    int g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      for (int ks = 0; ks < nk; ++ks, ++g) {
        const int s = g % NSTAGE;
        if (!mbar_wait(&pipe.full[s], (g / NSTAGE) & 1, WAIT_LIMIT)) { ok = false; break; }
        const float4 *hi = reinterpret_cast<const float4 *>(smem + (size_t)s * STAGE_BYTES + 4 * TILE);
        float4 *lo = reinterpret_cast<float4 *>(smem + (size_t)s * STAGE_BYTES + 5 * TILE);
#pragma unroll
        for (int i = 0; i < TILE / 16 / 128; ++i) {
          const float4 v = hi[i * 128 + et];
          lo[i * 128 + et] = make_float4(tf32_low(v.x), tf32_low(v.y), tf32_low(v.z), tf32_low(v.w));
        }
        fence_proxy_async();                    // generic-proxy writes -> visible to the tensor core's reads
        __syncwarp();
        if (lane == 0) mbar_arrive(&pipe.lo_ready[s]);
      }
    }
    if (!ok) atomicExch(&pipe.fail, 1);
  } else {
    // ------------------------------------------------------------------ sums over the chains, stores
    regs_inc<200>();
    // a TMEM lane is a float column of the activation, a TMEM column a weight row
    const int q = warp & 3, h = (warp - 8) >> 2;   // the quarter of the TMEM lanes that this warp may read, half of the rows
    int g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      const int m0 = t % mt * GM + h * (GM / 2), col = t / mt % nt * GN + q * 32 + lane, b = t / (mt * nt);
      float acc1[GM / 2], acc2[GM / 2];
#pragma unroll
      for (int i = 0; i < GM / 2; ++i) acc1[i] = acc2[i] = 0.f;
      for (int ks = 0; ks < nk; ks += PS, ++g) {
        if (!mbar_wait(&pipe.acc_full[g & 1], (g >> 1) & 1, WAIT_LIMIT)) { ok = false; break; }
        tc_fence_after();
        const uint32_t ta = tmem_base + (g & 1) * 2 * GN + ((uint32_t)(q * 32) << 16) + h * (GM / 2);
#pragma unroll
        for (int c = 0; c < GM / 64; ++c) {
          float v[32];
          tmem_ld32(ta + c * 32, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc1[c * 32 + j] += v[j];
          tmem_ld32(ta + GM + c * 32, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc2[c * 32 + j] += v[j];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pipe.acc_empty[g & 1]);
      }
      if (ok) {
        // even lanes hold the real parts of X's columns, odd lanes the imaginary parts: the other one's Im(W) sum
        // completes the product, and a warp stores 16 complex elements of a row at a time
        float *orow = reinterpret_cast<float *>(p.out) + ((int64_t)b * p.out_bs + (int64_t)m0 * p.out_ms) * 2 + col;
        const float sign = (lane & 1) ? 1.f : -1.f;
        const int rows = p.M - m0;
        const bool in = col < 2 * p.N;
        float any = 0.f;                                // NaN if an output is (or infinities of both signs are among them)
#pragma unroll
        for (int i = 0; i < GM / 2; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, acc2[i], 1), v = fmaf(sign, other, acc1[i]);
          any += v;
          if (i < rows && in) orow[(int64_t)i * p.out_ms * 2] = v;
        }
        if (any != any) *(volatile int *)&pipe.nan = 1;
      }
    }
    if (!ok) atomicExch(&pipe.fail, 1);
    if (*(volatile int *)&pipe.nan && ok)               // after all the tiles, where it takes no registers from them
      for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        plain_tile(p, mt, t % mt * GM + h * (GM / 2), t / mt % nt * GN + q * 32 + lane, t / (mt * nt));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
  if (tid == 0 && pipe.fail) atomicExch(&g_cgemm_status, 5);
}

// ---------------------------------------------------------------------------------------------
// Weight gradients of the projections:  dW (M x N) = sum over batch and time of G[b] U[b]^H,
// G (batch, M, L), U (batch, N, L) complex64 with L contiguous: dB~ = sum dBu u^H, dC~ = sum dy x^H
// (lrnnx/ops/simplified_scan.py:139,168,495,520).  Both operands are K-major here (the contraction
// runs along their contiguous dimension), and with g', u' the float views interleaved along L
//     Re dW = g' . u',     Im dW = g' . w',   w'[2l] = -u'[2l+1],  w'[2l+1] = u'[2l]
// so the imaginary part needs a pair-swapped, sign-flipped copy of the U tile.  The swap stays
// inside 16-byte chunks, so like the TF32 low parts it is produced in shared memory at the tile's
// own (swizzled) offsets.  Six tiles per stage: G, U from the TMA; G_lo, U_lo, W, W_lo from the
// transforming warps.  As above an accumulator lives for two stages, and eight warps with 64 columns
// of both results each add the chains up in registers.  The long contraction (batch x 2L floats) is
// cut over grid.z so that every SM has a piece; a thread block adds its 128 x 128 result to the
// zero-filled output with float32 vector reductions.  Rows past M or N belong to no output, steps
// past L are zeros.
constexpr uint32_t kIdescKK = kIdesc & ~(1u << 15);      // both operands K-major

struct GradMaps {
  CUtensorMap g;      // (2 L, batch M) float32, box (16, 128)
  CUtensorMap u;      // (2 L, batch N) float32, box (16, 128)
};

// This block's part (stages s_begin .. s_end) of the sum for row m and columns n, n + 32 of the output, as a plain sum, for
// the rows m + r whose bit is set in the column's mask.
__device__ __forceinline__ void plain_sums(const b200_cgemm_grad_args &p, uint32_t set0, uint32_t set1, int m, int n, int s_begin, int s_end) {
  const int per_batch = (2 * p.L + GK - 1) / GK;
  for (uint64_t set = set0 | (uint64_t)set1 << 32; set; set &= set - 1) {
    const int i = __ffsll((long long)set) - 1, mm = m + (i & 31), nn = n + (i & 32);
    float re = 0.f, im = 0.f;
    for (int s = s_begin; s < s_end && (re == re || im == im); ++s) {
      const int b = s / per_batch, l0 = s % per_batch * (GK / 2);
      const float2 *g = reinterpret_cast<const float2 *>(p.g) + ((int64_t)b * p.M + mm) * p.g_rs + l0;
      const float2 *u = reinterpret_cast<const float2 *>(p.u) + ((int64_t)b * p.N + nn) * p.u_rs + l0;
#pragma unroll
      for (int l = 0; l < GK / 2; ++l) {
        const float2 x = l < p.L - l0 ? g[l] : make_float2(0.f, 0.f), y = l < p.L - l0 ? u[l] : make_float2(0.f, 0.f);
        re = fmaf(x.x, y.x, fmaf(x.y, y.y, re));
        im = fmaf(x.y, y.x, fmaf(-x.x, y.y, im));
      }
    }
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(reinterpret_cast<float *>(p.out) + ((int64_t)mm * p.N + nn) * 2), "f"(re), "f"(im)
                 : "memory");
  }
}

__global__ void __launch_bounds__(NTHREADS, 1)
cgemm_ggh_kernel(const __grid_constant__ GradMaps maps, const b200_cgemm_grad_args p, const int stages_per_cta) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ Pipe pipe;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * GN, m0 = blockIdx.y * GM;
  const int per_batch = (2 * p.L + GK - 1) / GK;           // stages per batch entry
  const int total = p.batch * per_batch;
  const int s_begin = blockIdx.z * stages_per_cta;
  const int nk = max(0, min(stages_per_cta, total - s_begin));
  // tile slots of a stage: 0 G, 1 G_lo, 2 U, 3 W, 4 U_lo, 5 W_lo: U | W and U_lo | W_lo are operands of 256 rows
  if (tid == 0) pipe_init(pipe, 8);
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&pipe.tmem_base)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = pipe.tmem_base;

  // Registers: 512 threads are launched with 128 each; 48 + 64 + 2 x 184 = 480 of the four shares of 128 are used
  if (warp < 4) {
    regs_dec<48>();
    if (warp == 0 && lane == 0) {
      bool ok = true;
      for (int ks = 0; ks < nk; ++ks) {
        const int s = ks % NSTAGE;
        if (!wait_given_back(&pipe.empty[s], ks, NSTAGE)) { ok = false; break; }
        unsigned char *st = smem + (size_t)s * STAGE_BYTES;
        mbar_expect_tx(&pipe.full[s], 2 * TILE);
        const int sg = s_begin + ks;
        const int b = sg / per_batch, l0 = (sg % per_batch) * GK;
        tma_2d(st + 0 * TILE, &maps.g, l0, b * p.M + m0, &pipe.full[s]);
        tma_2d(st + 2 * TILE, &maps.u, l0, b * p.N + n0, &pipe.full[s]);
      }
      if (!ok) atomicExch(&pipe.fail, 1);
    } else if (warp == 1 && lane == 0) {
      bool ok = true;
      for (int ks = 0; ks < nk; ++ks) {
        const int s = ks % NSTAGE;
        const uint32_t ph = (ks / NSTAGE) & 1;
        const int ch = ks / PS;
        const uint32_t d = tmem_base + (ch & 1) * 2 * GN;        // columns: 128 real parts, 128 imaginary parts
        if (!mbar_wait(&pipe.full[s], ph, WAIT_LIMIT) || !mbar_wait(&pipe.lo_ready[s], ph, WAIT_LIMIT) ||
            (ks % PS == 0 && !wait_given_back(&pipe.acc_empty[ch & 1], ch, 2))) { ok = false; break; }
        tc_fence_after();
        const uint32_t st = smem_u32(smem + (size_t)s * STAGE_BYTES);
#pragma unroll
        for (int kk = 0; kk < GK / 8; ++kk) {
          mma_tf32(d, k_desc(st + 1 * TILE + kk * 32), k_desc(st + 2 * TILE + kk * 32), kk > 0 || ks % PS != 0 ? 1u : 0u, kIdescKK);
          mma_tf32(d, k_desc(st + 0 * TILE + kk * 32), k_desc(st + 4 * TILE + kk * 32), 1u, kIdescKK);
        }
#pragma unroll
        for (int kk = 0; kk < GK / 8; ++kk)
          mma_tf32(d, k_desc(st + 0 * TILE + kk * 32), k_desc(st + 2 * TILE + kk * 32), 1u, kIdescKK);
        mma_commit(&pipe.empty[s]);
        if (ks % PS == PS - 1 || ks == nk - 1) mma_commit(&pipe.acc_full[ch & 1]);
      }
      if (!ok) atomicExch(&pipe.fail, 1);
    }
  } else if (warp < 8) {
    regs_dec<64>();
    const int et = tid - 128;
    bool ok = true;
    for (int ks = 0; ks < nk; ++ks) {
      const int s = ks % NSTAGE;
      if (!mbar_wait(&pipe.full[s], (ks / NSTAGE) & 1, WAIT_LIMIT)) { ok = false; break; }
      float4 *t = reinterpret_cast<float4 *>(smem + (size_t)s * STAGE_BYTES);
      constexpr int T4 = TILE / 16;           // float4 per tile
#pragma unroll
      for (int i = 0; i < T4 / 128; ++i) {
        const int o = i * 128 + et;
        const float4 g = t[o], u = t[2 * T4 + o];
        t[T4 + o] = make_float4(tf32_low(g.x), tf32_low(g.y), tf32_low(g.z), tf32_low(g.w));
        const float4 ul = make_float4(tf32_low(u.x), tf32_low(u.y), tf32_low(u.z), tf32_low(u.w));
        t[4 * T4 + o] = ul;
        t[3 * T4 + o] = make_float4(-u.y, u.x, -u.w, u.z);
        t[5 * T4 + o] = make_float4(-ul.y, ul.x, -ul.w, ul.z);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pipe.lo_ready[s]);
    }
    if (!ok) atomicExch(&pipe.fail, 1);
  } else {
    regs_inc<184>();
    const int q = warp & 3, h = (warp - 8) >> 2;           // quarter of the TMEM lanes, half of the columns
    bool ok = true;
    float re[GN / 2], im[GN / 2];
#pragma unroll
    for (int i = 0; i < GN / 2; ++i) re[i] = im[i] = 0.f;
    for (int ch = 0; ch * PS < nk; ++ch) {
      if (!mbar_wait(&pipe.acc_full[ch & 1], (ch >> 1) & 1, WAIT_LIMIT)) { ok = false; break; }
      tc_fence_after();
      const uint32_t ta = tmem_base + (ch & 1) * 2 * GN + ((uint32_t)(q * 32) << 16) + h * (GN / 2);
#pragma unroll
      for (int c = 0; c < GN / 64; ++c) {
        float v1[32], v2[32];
        tmem_ld32x2(ta + c * 32, ta + GN + c * 32, v1, v2);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          re[c * 32 + j] += v1[j];
          im[c * 32 + j] += v2[j];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pipe.acc_empty[ch & 1]);
    }
    if (!ok) atomicExch(&pipe.fail, 1);
    if (ok && nk > 0 && pipe.fail == 0) {
      // A thread holds one output row (its TMEM lane).  32 columns at a time are turned through shared memory so
      // that a warp adds 32 consecutive complex elements of one row per instruction.  The stage buffers are free:
      // the last acc_full said that every MMA has read them and nothing is in flight.
      float2 *turn = reinterpret_cast<float2 *>(smem) + (size_t)(warp - 8) * 32 * 33;
      uint32_t nan[GN / 64];
#pragma unroll
      for (int c = 0; c < GN / 64; ++c) {
        nan[c] = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) turn[lane * 33 + j] =
            make_float2(fmaf(re[c * 32 + j], kLostGrad, re[c * 32 + j]), fmaf(im[c * 32 + j], kLostGrad, im[c * 32 + j]));
        __syncwarp();
        const int n = n0 + h * (GN / 2) + c * 32 + lane;
#pragma unroll 4
        for (int r = 0; r < 32; ++r) {
          const float2 v = turn[r * 33 + lane];
          const int m = m0 + q * 32 + r;
          if (m >= p.M || n >= p.N) continue;
          if (v.x != v.x || v.y != v.y) nan[c] |= 1u << r;
          else
            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(reinterpret_cast<float *>(p.out) + ((int64_t)m * p.N + n) * 2),
                         "f"(v.x), "f"(v.y)
                         : "memory");
        }
        __syncwarp();
      }
      if (nan[0] | nan[1]) plain_sums(p, nan[0], nan[1], m0 + q * 32, n0 + h * (GN / 2) + lane, s_begin, s_begin + nk);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
  if (tid == 0 && pipe.fail) atomicExch(&g_cgemm_status, 6);
}

// v rounded to the nearest TF32; a NaN stays one (its bits would carry over into a zero) and what would round to
// infinity is truncated
__device__ __forceinline__ float tf32_high(float v) {
  const uint32_t u = __float_as_uint(v), r = (u + 0x1000u) & 0xffffe000u;
  if (v != v) return __uint_as_float(0x7fc00000u);
  return __uint_as_float((r & 0x7fffffffu) == 0x7f800000u ? u & 0xffffe000u : r);
}

// Weight planes for cgemm_wx_kernel: (4, Mp, Kp) float32 = tf32(Re W), tf32(Re W - that), and the same
// for Im W, from a complex64 matrix addressed by element strides (a transposed view costs nothing)
// and optionally conjugated; zeros in the rows and columns that pad W to whole tiles.
__global__ void cgemm_planes_kernel(const float2 *w, int M, int K, int Mp, int Kp, int64_t rs, int64_t cs, int conj, float *planes) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t MK = (int64_t)Mp * Kp;
  if (i >= MK) return;
  const int m = (int)(i / Kp), k = (int)(i % Kp);
  float2 v = m < M && k < K ? w[(int64_t)m * rs + (int64_t)k * cs] : make_float2(0.f, 0.f);
  if (conj) v.y = -v.y;
  const float rh = tf32_high(v.x), ih = tf32_high(v.y);
  // of an infinity or a NaN: the canonical NaN, which becomes -0 below
  const float rl = fmaf(lost(K), v.x, v.x - rh), il = fmaf(lost(K), v.y, v.y - ih);
  planes[i] = rh;
  planes[MK + i] = __uint_as_float((__float_as_uint(rl) + 0x1000u) & 0xffffe000u);
  planes[2 * MK + i] = ih;
  planes[3 * MK + i] = __uint_as_float((__float_as_uint(il) + 0x1000u) & 0xffffe000u);
}

int up_to(int n, int unit) { return (n + unit - 1) / unit * unit; }

// (inner, rows[, batch]) float32; pitches in bytes
bool make_map(CUtensorMap *m, const void *base, uint64_t inner, uint64_t rows, uint64_t row_bytes, uint32_t box_inner, uint32_t box_rows,
              CUtensorMapSwizzle swizzle, uint64_t batch = 0, uint64_t batch_bytes = 0) {
  EncodeTiledFn enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {inner, rows, batch};
  const cuuint64_t strides[2] = {row_bytes, batch_bytes};
  const cuuint32_t box[3] = {box_inner, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, batch ? 3 : 2, const_cast<void *>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

int cgemm_status_read() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_cgemm_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace b200

using namespace b200;


extern "C" int b200_cgemm_grad(const b200_cgemm_grad_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "cgemm_grad: null argument block");
  const b200_cgemm_grad_args &a = *args;
  B200_REQUIRE(a.g && a.u && a.out, B200_ERR_NULL, "cgemm_grad: g, u, out must be non-null");
  B200_REQUIRE(a.batch > 0 && a.M > 0 && a.N > 0 && a.L > 0, B200_ERR_SHAPE, "cgemm_grad: sizes must be positive");
  B200_REQUIRE(a.g_rs || a.u_rs || (a.M % 128 == 0 && a.N % 128 == 0 && a.L % 16 == 0), B200_ERR_SHAPE,
               "cgemm_grad: without row pitches M and N must be multiples of 128, L of 16 (got M=%d N=%d L=%d)", a.M, a.N, a.L);
  // rows of all batch entries in one run: the batch pitch is M (N) row pitches
  const int64_t g_rs = a.g_rs ? a.g_rs : a.L, u_rs = a.u_rs ? a.u_rs : a.L;
  B200_REQUIRE(g_rs >= a.L && u_rs >= a.L && g_rs % 2 == 0 && u_rs % 2 == 0, B200_ERR_SHAPE,
               "cgemm_grad: row pitches must be even and at least L (L=%d, pitches %lld, %lld)", a.L, (long long)g_rs, (long long)u_rs);
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a.g) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.u) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(a.out) & 7) == 0,
               B200_ERR_ALIGN, "cgemm_grad: operands must be 16-byte aligned");
  const int64_t total = (int64_t)a.batch * ((2 * (int64_t)a.L + GK - 1) / GK);
  B200_REQUIRE((int64_t)a.batch * a.M < (int64_t(1) << 31) && (int64_t)a.batch * a.N < (int64_t(1) << 31) && total < (int64_t(1) << 31) &&
                   2 * (int64_t)a.L < (int64_t(1) << 31) - GK,
               B200_ERR_SHAPE, "cgemm_grad: batch * rows or batch * L too large");
  GradMaps maps;
  memset(&maps, 0, sizeof(maps));
  B200_REQUIRE(make_map(&maps.g, a.g, 2ull * a.L, (uint64_t)a.batch * a.M, 8ull * g_rs, GK, GM, CU_TENSOR_MAP_SWIZZLE_64B) &&
                   make_map(&maps.u, a.u, 2ull * a.L, (uint64_t)a.batch * a.N, 8ull * u_rs, GK, GN, CU_TENSOR_MAP_SWIZZLE_64B),
               B200_ERR_UNSUPPORTED, "cgemm_grad: tensor-map encoding failed");
  const int smem = NSTAGE * STAGE_BYTES + 1024;
  cudaError_t e = cudaFuncSetAttribute(cgemm_ggh_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return (int)e; }
  // As many pieces of the contraction as give every SM a thread block, of at least 16 stages each: a piece ends
  // with 128 KB of reductions
  const int nt = (a.N + GN - 1) / GN, mt = (a.M + GM - 1) / GM;
  int64_t pieces = sm_count_current() / ((int64_t)nt * mt);
  if (pieces > (total + 15) / 16) pieces = (total + 15) / 16;
  if (pieces < 1) pieces = 1;
  const int64_t per = (total + pieces - 1) / pieces;
  const dim3 grid((unsigned)nt, (unsigned)mt, (unsigned)((total + per - 1) / per));
  b200_cgemm_grad_args k = a;
  k.g_rs = g_rs;
  k.u_rs = u_rs;
  cgemm_ggh_kernel<<<grid, NTHREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(maps, k, (int)per);
  return launch_status();
}

extern "C" int b200_cgemm_planes(const b200_cgemm_planes_args *args, void *stream) {
  B200_REQUIRE(args && args->w && args->planes, B200_ERR_NULL, "cgemm_planes: w and planes must be non-null");
  B200_REQUIRE(args->M > 0 && args->K > 0, B200_ERR_SHAPE, "cgemm_planes: sizes must be positive");
  const int Mp = args->padded ? up_to(args->M, GM) : args->M, Kp = args->padded ? up_to(args->K, KPAD) : args->K;
  const int64_t n = (int64_t)Mp * Kp;
  cgemm_planes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2 *>(args->w), args->M, args->K, Mp, Kp, args->w_rs, args->w_cs, args->conj,
      reinterpret_cast<float *>(args->planes));
  return launch_status();
}

extern "C" int b200_cgemm_wx(const b200_cgemm_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "cgemm_wx: null argument block");
  const b200_cgemm_args &a = *args;
  B200_REQUIRE(a.w_planes && a.x && a.out, B200_ERR_NULL, "cgemm_wx: w_planes, x, out must be non-null");
  B200_REQUIRE(a.batch > 0 && a.M > 0 && a.K > 0 && a.N > 0, B200_ERR_SHAPE, "cgemm_wx: sizes must be positive");
  B200_REQUIRE(a.padded || (a.M % 128 == 0 && a.K % 32 == 0 && a.N % 64 == 0), B200_ERR_SHAPE,
               "cgemm_wx: without padded planes M must be a multiple of 128, K of 32, N of 64 (got M=%d K=%d N=%d)", a.M, a.K, a.N);
  B200_REQUIRE(a.padded || (a.x_ks == a.N && a.x_bs == (int64_t)a.K * a.N && a.out_ms % 2 == 0 && a.out_bs % 2 == 0 &&
                            (reinterpret_cast<uintptr_t>(a.out) & 15) == 0),
               B200_ERR_UNSUPPORTED, "cgemm_wx: without padded planes x must be a dense (batch, K, N) tensor, out 16-byte aligned");
  B200_REQUIRE(a.x_ks >= a.N && a.x_ks % 2 == 0 && a.x_bs >= 0 && a.x_bs % 2 == 0, B200_ERR_SHAPE,
               "cgemm_wx: the row pitch of x must be even and at least N, its batch pitch even (N=%d, pitches %lld, %lld)", a.N,
               (long long)a.x_ks, (long long)a.x_bs);
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 7) == 0 &&
                   (reinterpret_cast<uintptr_t>(a.w_planes) & 15) == 0,
               B200_ERR_ALIGN, "cgemm_wx: x and the planes must be 16-byte aligned, out 8-byte aligned");
  const int Mp = up_to(a.M, GM), Kp = up_to(a.K, KPAD);
  const int mt = Mp / GM;
  const int64_t nt = (2 * (int64_t)a.N + GN - 1) / GN, tiles = nt * mt * a.batch;
  B200_REQUIRE(tiles < (int64_t(1) << 30) && 2 * (int64_t)a.N < (int64_t(1) << 31) - GN, B200_ERR_SHAPE, "cgemm_wx: sizes too large");
  GemmMaps maps;
  memset(&maps, 0, sizeof(maps));
  B200_REQUIRE(make_map(&maps.w, a.w_planes, (uint64_t)Kp, 4ull * Mp, (uint64_t)Kp * 4, GK, GM, CU_TENSOR_MAP_SWIZZLE_64B) &&
                   make_map(&maps.x, a.x, 2ull * a.N, (uint64_t)a.K, 8ull * a.x_ks, 32, GK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, (uint64_t)a.batch,
                            8ull * (a.batch > 1 ? a.x_bs : a.x_ks * (int64_t)a.K)),
               B200_ERR_UNSUPPORTED, "cgemm_wx: tensor-map encoding failed");
  const int smem = NSTAGE * STAGE_BYTES + 1024;
  cudaError_t e = cudaFuncSetAttribute(cgemm_wx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return (int)e; }
  const int sms = sm_count_current();
  cgemm_wx_kernel<<<(unsigned)(tiles < sms ? tiles : sms), NTHREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      maps, a, mt, (int)nt, (a.K + GK - 1) / GK);
  return launch_status();
}
