// Selective scan with one state per channel and constant B and C, float32: the RG-LRU and S7 layers
// (lrnnx/ops/rglru_scan.py:28-144, lrnnx/ops/s7_scan.py:28-180 call the extension this way).
//
// With a single state nothing is reused (12 bytes a step forward, 20 backward), and what a step costs is instructions: the
// coefficient, the scans and the way through shared memory (IPC 3.5 of 4 forward, 2.5 backward; DRAM 27 %).  A thread block owns a row and takes 2048 steps (one checkpoint chunk) at a
// time, 256 per warp, 8 consecutive ones per lane; rows of up to 256, 512 and 1024 steps get 1, 2 and 4 warps.
// Rows are read and written by coalesced 4-byte elements and turned to 8 steps per lane through a conflict-free
// row in shared memory: any length and alignment.  Thread-serial scan of 8 steps, warp-shuffle scan of the
// lanes, a short fold over the warps.  The backward rebuilds the states from the checkpoint before the chunk and
// runs the adjoint in the same pass: g_t = dy_t B C + q_t, q_{t-1} = a_t g_t.
// Measured, 4 x 1024 rows x 2048 steps: forward 32 us, backward 61 us (the one-warp-per-row coverage kernels: 151 and
// 378 us; the bytes alone: 15 and 25 us at the copy rate).  The exponential beside expm1 is 2 us of each.
// The RG-LRU input gain sqrt(1 - a^2) is taken from expm1, which keeps it exact where a is close to 1; the transition
// itself is the exponential where it is small (dA is divided by A, so a's error counts relative to a).
#include "common.cuh"
#include "dispatch.h"

namespace b200 {
namespace {

constexpr int RI = 8;                     // steps per lane
constexpr int RSTEPS = 32 * RI;           // steps per warp
constexpr int RROW = RSTEPS + 16;         // floats of a warp's row in shared memory

// a 256-step row lies as pieces of 4 steps, even pieces first, odd ones 16 banks off: a lane's two
// pieces and 32 consecutive elements are both free of bank conflicts
__device__ __forceinline__ int elem_at(int i) {
  const int piece = i >> 2;
  return (piece & 1) * (RSTEPS / 2 + 16) + (piece >> 1) * 4 + (i & 3);
}
__device__ __forceinline__ void fetch(const float *row, int t0, int L, int lane, float (&r)[RI]) {
#pragma unroll
  for (int k = 0; k < RI; ++k) r[k] = t0 + lane + 32 * k < L ? row[t0 + lane + 32 * k] : 0.f;
}
__device__ __forceinline__ void to_lanes(float *buf, int lane, float (&r)[RI]) {
#pragma unroll
  for (int k = 0; k < RI; ++k) buf[elem_at(lane + 32 * k)] = r[k];
  __syncwarp();
  const float4 x = *reinterpret_cast<const float4 *>(buf + 4 * lane), y = *reinterpret_cast<const float4 *>(buf + RSTEPS / 2 + 16 + 4 * lane);
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w; r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
  __syncwarp();
}
__device__ __forceinline__ void store(float *row, int t0, int L, float *buf, int lane, const float (&v)[RI]) {
  *reinterpret_cast<float4 *>(buf + 4 * lane) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4 *>(buf + RSTEPS / 2 + 16 + 4 * lane) = make_float4(v[4], v[5], v[6], v[7]);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < RI; ++k)
    if (t0 + lane + 32 * k < L) row[t0 + lane + 32 * k] = buf[elem_at(lane + 32 * k)];
  __syncwarp();
}

// e = exp(x) and m = exp(x) - 1, each accurate relative to itself.  For |x| <= 1 m is the Taylor series to x^10
// (truncation below 4e-8 of m) and e = 1 + m, at least 0.36, loses half a unit of 1.  Elsewhere nothing cancels in
// m = e - 1, but 1 + m would keep only e's bits above 2^-24: there e itself is the exponential.
__device__ __forceinline__ void exp_expm1(float x, float &e, float &m) {
  const float big = expf(x);
  float s = fmaf(x, 1.f / 10.f, 1.f);
#pragma unroll
  for (int k = 9; k >= 2; --k) s = fmaf(x * (1.f / k), s, 1.f);
  const bool near0 = fabsf(x) <= 1.f;
  m = near0 ? x * s : big - 1.f;
  e = near0 ? 1.f + m : big;
}

// transition a, input gain k
template <int DM> __device__ __forceinline__ void coef(float logA, float d, float &a, float &k) {
  if constexpr (DM == B200_DISC_RGLRU) {          // a = A^d, k = sqrt(1 - a^2)
    float m;
    exp_expm1(d * logA, a, m);
    k = sqrtf(-m * (2.f + m));
  } else {                                        // S7: a = 1 - 1 / (d^2 + 1/2), k = 1
    a = 1.f - 1.f / (d * d + 0.5f);
    k = 1.f;
  }
}

// composition of the lanes' maps h -> P h + H, lane 0 first: on return (P, H) is the map of lanes 0 .. lane - 1
// and (Pt, Ht) that of the whole warp
__device__ __forceinline__ void scan_up(float &P, float &H, float &Pt, float &Ht, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float p = __shfl_up_sync(0xffffffffu, P, off), h = __shfl_up_sync(0xffffffffu, H, off);
    if (lane >= off) { H = fmaf(P, h, H); P *= p; }
  }
  Pt = __shfl_sync(0xffffffffu, P, 31);
  Ht = __shfl_sync(0xffffffffu, H, 31);
  P = __shfl_up_sync(0xffffffffu, P, 1);
  H = __shfl_up_sync(0xffffffffu, H, 1);
  if (lane == 0) { P = 1.f; H = 0.f; }
}
__device__ __forceinline__ void scan_down(float &P, float &H, float &Pt, float &Ht, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float p = __shfl_down_sync(0xffffffffu, P, off), h = __shfl_down_sync(0xffffffffu, H, off);
    if (lane + off < 32) { H = fmaf(P, h, H); P *= p; }
  }
  Pt = __shfl_sync(0xffffffffu, P, 0);
  Ht = __shfl_sync(0xffffffffu, H, 0);
  P = __shfl_down_sync(0xffffffffu, P, 1);
  H = __shfl_down_sync(0xffffffffu, H, 1);
  if (lane == 31) { P = 1.f; H = 0.f; }
}

template <int DM, int NW>
__global__ void __launch_bounds__(NW * 32) selscan_row1_fwd_kernel(const b200_selscan_fwd_args p) {
  __shared__ __align__(16) float buf_all[NW][RROW];
  __shared__ float2 agg[2][NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x;
  const int b = (int)(row / p.dim), d = (int)(row % p.dim);
  const int L = p.seqlen, n_chunks = (L + kChunk - 1) / kChunk;
  const float *up = reinterpret_cast<const float *>(p.u) + (int64_t)b * p.u_bs + (int64_t)d * p.u_ds;
  const float *dp = reinterpret_cast<const float *>(p.delta) + (int64_t)b * p.delta_bs + (int64_t)d * p.delta_ds;
  float *op = reinterpret_cast<float *>(p.out) + (int64_t)b * p.out_bs + (int64_t)d * p.out_ds;
  float2 *xp = reinterpret_cast<float2 *>(p.x) + row * n_chunks;
  const float logA = DM == B200_DISC_RGLRU ? logf(reinterpret_cast<const float *>(p.A)[(int64_t)d * p.A_ds]) : 0.f;
  const float cfix = reinterpret_cast<const float *>(p.B)[(int64_t)d * p.B_gs] * reinterpret_cast<const float *>(p.C)[(int64_t)d * p.C_gs];
  float *buf = buf_all[warp];
  float hc = 0.f, Pc = 1.f;               // state entering the chunk, product of a so far
  float u[RI], dl[RI];
  fetch(up, warp * RSTEPS, L, lane, u);
  fetch(dp, warp * RSTEPS, L, lane, dl);
  for (int c = 0; c < n_chunks; ++c) {
    const int t0 = c * kChunk + warp * RSTEPS;
    to_lanes(buf, lane, u);
    to_lanes(buf, lane, dl);
    float a[RI], h[RI];
    float P = 1.f, H = 0.f;
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      float k;
      coef<DM>(logA, dl[i], a[i], k);
      h[i] = k * u[i];
      if (t0 + lane * RI + i >= L) { a[i] = 1.f; h[i] = 0.f; }
      H = fmaf(a[i], H, h[i]);
      P *= a[i];
    }
    if (c + 1 < n_chunks) {               // the next chunk's rows travel during the scans and the stores
      fetch(up, t0 + kChunk, L, lane, u);
      fetch(dp, t0 + kChunk, L, lane, dl);
    }
    float Pt, Ht;
    scan_up(P, H, Pt, Ht, lane);
    if (lane == 0) agg[c & 1][warp] = make_float2(Pt, Ht);
    __syncthreads();
    float hw = hc, hn = hc, pn = Pc;      // state entering this warp's steps; state and product after the chunk
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float2 v = agg[c & 1][w];
      if (w == warp) hw = hn;
      hn = fmaf(v.x, hn, v.y);
      pn *= v.x;
    }
    float s = fmaf(P, hw, H);
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      s = fmaf(a[i], s, h[i]);
      h[i] = s * cfix;
    }
    store(op, t0, L, buf, lane, h);
    hc = hn;
    Pc = pn;
    if (threadIdx.x == 0) xp[c] = make_float2(Pc, hc);
  }
}

template <int DM, int NW>
__global__ void __launch_bounds__(NW * 32) selscan_row1_bwd_kernel(const b200_selscan_bwd_args q) {
  const b200_selscan_fwd_args &p = q.f;
  __shared__ __align__(16) float buf_all[NW][RROW];
  __shared__ float2 agg[2][NW], ragg[2][NW], sums[NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x;
  const int b = (int)(row / p.dim), d = (int)(row % p.dim);
  const int L = p.seqlen, n_chunks = (L + kChunk - 1) / kChunk;
  const float *up = reinterpret_cast<const float *>(p.u) + (int64_t)b * p.u_bs + (int64_t)d * p.u_ds;
  const float *dp = reinterpret_cast<const float *>(p.delta) + (int64_t)b * p.delta_bs + (int64_t)d * p.delta_ds;
  const float *gp = reinterpret_cast<const float *>(q.dout) + (int64_t)b * q.dout_bs + (int64_t)d * q.dout_ds;
  float *dup = reinterpret_cast<float *>(q.du) + (int64_t)b * q.du_bs + (int64_t)d * q.du_ds;
  float *ddp = reinterpret_cast<float *>(q.ddelta) + (int64_t)b * q.ddelta_bs + (int64_t)d * q.ddelta_ds;
  const float2 *xp = reinterpret_cast<const float2 *>(p.x) + row * n_chunks;
  const float A = reinterpret_cast<const float *>(p.A)[(int64_t)d * p.A_ds];
  const float logA = DM == B200_DISC_RGLRU ? logf(A) : 0.f;
  const float Bv = reinterpret_cast<const float *>(p.B)[(int64_t)d * p.B_gs], Cv = reinterpret_cast<const float *>(p.C)[(int64_t)d * p.C_gs];
  const float cfix = Bv * Cv;
  float *buf = buf_all[warp];
  float qc = 0.f;                          // a g of the first step of the chunk after
  float accA = 0.f, accBC = 0.f;
  float u[RI], dl[RI], dy[RI];
  {
    const int t0 = (n_chunks - 1) * kChunk + warp * RSTEPS;
    fetch(up, t0, L, lane, u);
    fetch(dp, t0, L, lane, dl);
    fetch(gp, t0, L, lane, dy);
  }
  for (int c = n_chunks - 1; c >= 0; --c) {
    const int t0 = c * kChunk + warp * RSTEPS;
    const float hc = c > 0 ? xp[c - 1].y : 0.f;
    to_lanes(buf, lane, u);
    to_lanes(buf, lane, dl);
    to_lanes(buf, lane, dy);
    float a[RI], k[RI], g[RI], hp[RI], uu[RI], dd[RI];
    float P = 1.f, H = 0.f, Q = 1.f, G = 0.f;
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      coef<DM>(logA, dl[i], a[i], k[i]);
      if (t0 + lane * RI + i >= L) { a[i] = 1.f; k[i] = 0.f; }
      uu[i] = u[i];
      dd[i] = dl[i];
      g[i] = dy[i];
      H = fmaf(a[i], H, k[i] * u[i]);
      P *= a[i];
    }
#pragma unroll
    for (int i = RI - 1; i >= 0; --i) G = a[i] * fmaf(g[i], cfix, G);
    Q = P;
    if (c > 0) {
      fetch(up, t0 - kChunk, L, lane, u);
      fetch(dp, t0 - kChunk, L, lane, dl);
      fetch(gp, t0 - kChunk, L, lane, dy);
    }
    float Pt, Ht, Qt, Gt;
    scan_up(P, H, Pt, Ht, lane);
    scan_down(Q, G, Qt, Gt, lane);
    if (lane == 0) {
      agg[c & 1][warp] = make_float2(Pt, Ht);
      ragg[c & 1][warp] = make_float2(Qt, Gt);
    }
    __syncthreads();
    float hw = hc, qw = qc, qn = qc;
#pragma unroll
    for (int w = 0; w < NW; ++w)
      if (w < warp) { const float2 v = agg[c & 1][w]; hw = fmaf(v.x, hw, v.y); }
#pragma unroll
    for (int w = NW - 1; w >= 0; --w) {
      const float2 v = ragg[c & 1][w];
      if (w == warp) qw = qn;
      qn = fmaf(v.x, qn, v.y);
    }
    qc = qn;
    float s = fmaf(P, hw, H);
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      hp[i] = s;
      s = fmaf(a[i], s, k[i] * uu[i]);
      accBC = fmaf(g[i], s, accBC);
    }
    float qq = fmaf(Q, qw, G);
#pragma unroll
    for (int i = RI - 1; i >= 0; --i) {
      const float gg = fmaf(g[i], cfix, qq);
      qq = a[i] * gg;
      float dv = 0.f;
      if constexpr (DM == B200_DISC_RGLRU) {
        if (dd[i] > 0.f) {
          const float Ga = gg * (hp[i] - a[i] * uu[i] * __fdividef(1.f, k[i])) * a[i];
          dv = Ga * logA;
          if (t0 + lane * RI + i < L) accA = fmaf(Ga, dd[i], accA);
        }
      } else {
        const float sq = fmaf(dd[i], dd[i], 0.5f);
        dv = gg * hp[i] * __fdividef(2.f * dd[i], sq * sq);
      }
      g[i] = gg * k[i];                    // du
      dd[i] = dv;
    }
    store(dup, t0, L, buf, lane, g);
    store(ddp, t0, L, buf, lane, dd);
  }
  accA = warp_sum(accA);
  accBC = warp_sum(accBC);
  if (lane == 0) sums[warp] = make_float2(accA, accBC);
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < NW; ++w) { accA += sums[w].x; accBC += sums[w].y; }
    if (DM == B200_DISC_RGLRU) atomicAdd(reinterpret_cast<float *>(q.dA) + (int64_t)d * q.dA_ds, accA / A);
    atomicAdd(reinterpret_cast<float *>(q.dB) + (int64_t)d * q.dB_gs, accBC * Cv);
    atomicAdd(reinterpret_cast<float *>(q.dC) + (int64_t)d * q.dC_gs, accBC * Bv);
  }
}

#define B200_ROW1(KERNEL, ARGS)                                                                                    \
  const int L = f.seqlen;                                                                                          \
  const unsigned rows = (unsigned)((int64_t)f.batch * f.dim);                                                      \
  if (f.method == B200_DISC_RGLRU) {                                                                               \
    if (L <= RSTEPS) KERNEL<B200_DISC_RGLRU, 1><<<rows, 32, 0, st>>>(ARGS);                                        \
    else if (L <= 2 * RSTEPS) KERNEL<B200_DISC_RGLRU, 2><<<rows, 64, 0, st>>>(ARGS);                               \
    else if (L <= 4 * RSTEPS) KERNEL<B200_DISC_RGLRU, 4><<<rows, 128, 0, st>>>(ARGS);                              \
    else KERNEL<B200_DISC_RGLRU, 8><<<rows, 256, 0, st>>>(ARGS);                                                   \
  } else {                                                                                                         \
    if (L <= RSTEPS) KERNEL<B200_DISC_S7, 1><<<rows, 32, 0, st>>>(ARGS);                                           \
    else if (L <= 2 * RSTEPS) KERNEL<B200_DISC_S7, 2><<<rows, 64, 0, st>>>(ARGS);                                  \
    else if (L <= 4 * RSTEPS) KERNEL<B200_DISC_S7, 4><<<rows, 128, 0, st>>>(ARGS);                                 \
    else KERNEL<B200_DISC_S7, 8><<<rows, 256, 0, st>>>(ARGS);                                                      \
  }                                                                                                                \
  return launch_status();

}  // namespace

bool selscan_row1_supported(const b200_selscan_fwd_args &a) {
  return (a.method == B200_DISC_RGLRU || a.method == B200_DISC_S7) && a.dstate == 1 && !a.is_complex && a.dtype == B200_F32 &&
         !a.var_B && !a.var_C && !a.D && !a.z && !a.delta_bias && !a.deltaA && !a.delta_softplus &&
         (reinterpret_cast<uintptr_t>(a.x) & 7) == 0 && (int64_t)a.batch * a.dim < (int64_t)1 << 31;
}

int selscan_row1_fwd(const b200_selscan_fwd_args &f, cudaStream_t st) { B200_ROW1(selscan_row1_fwd_kernel, f) }
int selscan_row1_bwd(const b200_selscan_bwd_args &q, cudaStream_t st) {
  const b200_selscan_fwd_args &f = q.f;
  B200_ROW1(selscan_row1_bwd_kernel, q)
}

}  // namespace b200
