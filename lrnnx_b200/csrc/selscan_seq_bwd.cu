// State-parallel selective scan, backward (same shape class as selscan_seq.cu).
//
// With h_t = a_t h_{t-1} + delta_t u_t B_t, y_t = C_t . h_t and dy_t the gradient arriving at y_t, the
// adjoint is g_t = C_t dy_t + q_t, q_{t-1} = a_t g_t.  Two launches:
//   1. selscan_seq_pre_kernel: thread blocks of two kinds, in one grid because either alone leaves
//      most issue slots empty.  Some walk the sequence backward, as the forward kernel walks it
//      forward, and write the q entering every block of 4 steps from the right; the others start
//      from the states that the forward call saved and write the state entering every block.
//   2. selscan_seq_bwd_kernel: every block of 4 steps is now independent.  A thread block owns 128
//      steps and loops over channels; a warp owns four states and a lane 4 steps, so B, C and the
//      dB / dC sums over the channels stay in registers from the first channel to the last (they
//      are the sums that a kernel which owns channels has to push through shared memory or
//      shuffles at every step).  delta, delta u and dy of 4 channels at a time are prepared once by
//      all threads; the sums over the states (for du and ddelta) meet in shared memory.
// Measured, batch 8 x 1536 channels x 2048 steps, bf16, gated: 280 + 415 us (a kernel that owns channels and scans
// across lanes: 845 us).  The first launch is bound by the shared-memory pipe (93 %; SFU 76 %), the second by latency
// (12 warps per SM, IPC 1.9 of 4, FMA pipe 44 %).  Blocks of 4 steps rather than 8: with 8 a lane needs 255 registers,
// two warps per scheduler are left and the second launch takes 600 us, for 90 us less in the first.
// Gradients of A, B, C, D and delta_bias leave by float32 atomics, one per (n, t) and run of
// channels for B and C, one per (channel, n) and 128 steps for A.
// Results match csrc/selective_scan/selective_scan_backward.cuh:86-845 of lrnnx.
#include "selscan_seq.cuh"

namespace b200 {
namespace {
using namespace seq;

constexpr int FW = 4;             // warps per thread block of the walks
constexpr int TB = kSeqBlock;     // steps per block of their recurrences
constexpr int CROW = 20;          // floats per timestep row of their C | B tile (16 + 4 of padding)

// 4 steps of a row as they come from memory.  VEC: one access of 4 elements, kept packed (taking the
// elements apart right after the load would wait for it)
template <typename T, bool VEC> struct Quad {
  T v[4];
  __device__ __forceinline__ void load(const T *p, int left) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = left > j ? p[j] : from_f<T>(0.f);
  }
  __device__ __forceinline__ void load4(const T *p) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = p[j];
  }
  __device__ __forceinline__ float get(int j) const { return to_f(v[j]); }
};
template <typename T> struct Quad<T, true> {
  static constexpr int W = (int)sizeof(T);          // 32-bit words
  uint32_t w[W];
  __device__ __forceinline__ void load4(const T *p) {
    if constexpr (W == 4) {
      const uint4 x = *reinterpret_cast<const uint4 *>(p);
      w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
    } else {
      const uint2 x = *reinterpret_cast<const uint2 *>(p);
      w[0] = x.x; w[1] = x.y;
    }
  }
  __device__ __forceinline__ void load(const T *p, int left) {
    if (left >= 4) { load4(p); return; }
#pragma unroll
    for (int j = 0; j < W; ++j) w[j] = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (left > j) {
        if constexpr (W == 4) w[j] = reinterpret_cast<const uint32_t *>(p)[j];
        else w[j >> 1] |= (uint32_t)reinterpret_cast<const unsigned short *>(p)[j] << (16 * (j & 1));
      }
  }
  __device__ __forceinline__ float get(int j) const {
    if constexpr (W == 4) return __uint_as_float(w[j]);
    else return to_f(reinterpret_cast<const T *>(&w[j >> 1])[j & 1]);
  }
};
// ------------------------------------------------- states and adjoints at the block boundaries
// what the launch needs beyond the call's arguments
struct SeqPre {
  float4 *hs, *qs;       // (batch, dim, 4 quarters of the states, seq_blocks(seqlen))
  float4 *carry;         // (batch, dim, 4): the adjoint that leaves the window to the left
  int t0, total;         // the call's arguments are steps t0 .. t0 + seqlen of this many; x and stage_h those of all
  int piece;             // steps per independently started piece of the states' walk
  int tiles;             // thread blocks that a batch row takes
  int adj;               // thread blocks of the first kind: one per tile and batch row, then one per piece
};

constexpr int PRE_FIX = (2 * QT * CROW + FW * QT * DROW) * (int)sizeof(float);     // tiles of the walks, bytes
// ADJ: the walk backward over {delta, dy} and C; otherwise the walk forward over {delta, delta u} and B
template <typename T, bool ADJ, bool ALN, bool Z>
__device__ __forceinline__ void seq_walk(const b200_selscan_bwd_args &a, const SeqPre &x, int tile, int piece, unsigned char *smem) {
  const b200_selscan_fwd_args &p = a.f;
  constexpr bool GZ = ADJ && Z;                                  // dy needs the gate
  constexpr int RAW = QCH * QT * (int)sizeof(T), NRAW = Z ? 3 : 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *mt = reinterpret_cast<float *>(smem);                   // [2][QT * CROW]: C or B of a stage, float32, [t][n]
  float *dd = mt + 2 * QT * CROW + warp * QT * DROW;             // {delta, dy or delta u} per (t, channel)
  unsigned char *raw = smem + PRE_FIX + (ALN ? warp * 2 * NRAW * RAW : 0);
  const int c = lane & 7, q = lane >> 3;                         // recurrence: channel, quarter of the states
  const int cpg = p.dim / p.n_groups;
  const int tpg = (cpg + FW * QCH - 1) / (FW * QCH);
  const int b = tile / (p.n_groups * tpg), g = tile / tpg % p.n_groups;
  const int cin = (tile % tpg * FW + warp) * QCH;                // first channel of this warp within the group
  const int nch = min(cpg - cin, QCH);                           // <= 0: the warp only helps with the C | B tile
  const int d0 = g * cpg + cin, dl = nch > 0 ? d0 : g * cpg;
  const int t_begin = ADJ ? 0 : piece * x.piece, L = ADJ ? p.seqlen : min(p.seqlen, t_begin + x.piece);
  const int nst = (L - t_begin + QT - 1) / QT;
  const int t_first = ADJ ? (nst - 1) * QT : t_begin;            // first step of the first stage walked
  const int dir = ADJ ? -QT : QT;

  // ---- operands: delta, then dout (and z) or u
  const void *vp = ADJ ? a.dout : p.u;
  const int64_t v_bs = ADJ ? a.dout_bs : p.u_bs, v_ds = ADJ ? a.dout_ds : p.u_ds;
  RowCopy<T> cd, cv, cz;
  T rd[ALN ? 1 : QCH], rv[ALN ? 1 : QCH], rz[ALN ? 1 : QCH];
  const T *Dp = nullptr, *Vp = nullptr, *Zp = nullptr;
  if constexpr (ALN) {
    cd.init(p.delta, p.delta_bs, p.delta_ds, b, dl, lane, nch, t_first);
    cv.init(vp, v_bs, v_ds, b, dl, lane, nch, t_first);
    if (GZ) cz.init(p.z, p.z_bs, p.z_ds, b, dl, lane, nch, t_first);
  } else {
    Dp = reinterpret_cast<const T *>(p.delta) + (int64_t)b * p.delta_bs + (int64_t)dl * p.delta_ds + t_first + lane;
    Vp = reinterpret_cast<const T *>(vp) + (int64_t)b * v_bs + (int64_t)dl * v_ds + t_first + lane;
    if (GZ) Zp = reinterpret_cast<const T *>(p.z) + (int64_t)b * p.z_bs + (int64_t)dl * p.z_ds + t_first + lane;
  }
  // C | B: a thread takes 4 steps of one of the 16 rows
  const int mrow = threadIdx.x & 15, mt0 = (threadIdx.x >> 4) * 4;
  const T *Mp = reinterpret_cast<const T *>(ADJ ? p.C : p.B) + (int64_t)b * (ADJ ? p.C_bs : p.B_bs) + (int64_t)g * (ADJ ? p.C_gs : p.B_gs) +
                (int64_t)mrow * (ADJ ? p.C_ns : p.B_ns) + t_first + mt0;
  Quad<T, ALN> rm;
  auto load_stage = [&](int s) {                                 // s-th stage walked
    const int left = L - (t_first + s * dir);
    rm.load(Mp, left - mt0);
    Mp += dir;
    if constexpr (ALN) {
      const int mine = left - (lane % PPR<T>) * EPC<T>;
      unsigned char *dst = raw + (s & 1) * NRAW * RAW;
      cd.fetch(dst, lane, nch, mine);
      cv.fetch(dst + RAW, lane, nch, mine);
      cd.p += dir;
      cv.p += dir;
      if constexpr (GZ) {
        cz.fetch(dst + 2 * RAW, lane, nch, mine);
        cz.p += dir;
      }
      cp_commit();
    } else {
      const bool ok = lane < left;
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        const bool oki = ok && i < nch;
        rd[i] = oki ? Dp[(int64_t)i * p.delta_ds] : from_f<T>(0.f);
        rv[i] = oki ? Vp[(int64_t)i * v_ds] : from_f<T>(0.f);
        if (GZ) rz[i] = oki ? Zp[(int64_t)i * p.z_ds] : from_f<T>(0.f);
      }
      Dp += dir;
      Vp += dir;
      if (GZ) Zp += dir;
    }
  };
  load_stage(0);

  float2 A2[2];
  {
    const float *A = reinterpret_cast<const float *>(p.A) + (int64_t)(dl + min(c, max(nch - 1, 0))) * p.A_ds;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      A2[j] = make_float2(decay2(A[(int64_t)(QS * q + 2 * j) * p.A_ns]), decay2(A[(int64_t)(QS * q + 2 * j + 1) * p.A_ns]));
  }
  float bias[QCH];
#pragma unroll
  for (int i = 0; i < QCH; ++i) bias[i] = p.delta_bias && i < nch ? reinterpret_cast<const float *>(p.delta_bias)[dl + i] : 0.f;
  const bool mine = c < nch;
  const int64_t row = (int64_t)b * p.dim + d0 + c;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);                    // the state, or q
  if (mine) {
    const int64_t o = QS * q;
    const int t = x.t0 + t_begin;                                // a multiple of the piece
    if (ADJ) {
      if (x.t0 + p.seqlen < x.total) v = x.carry[row * 4 + q];
      else if (a.q_in) v = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(a.q_in) + row * QN + o);
    } else if (t == 0) {
      if (a.h_in) v = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(a.h_in) + row * QN + o);
    } else if (p.stage_h) {
      const int64_t n_stages = (x.total + p.stage_len - 1) / p.stage_len;
      v = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.stage_h) + (row * n_stages + t / p.stage_len - 1) * QN + o);
    } else {
      const int64_t n_chunks = (x.total + kChunk - 1) / kChunk;
      const float4 *xr = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p.x) + (row * n_chunks + t / kChunk - 1) * 2 * QN + 2 * o);
      v = make_float4(xr[0].y, xr[0].w, xr[1].y, xr[1].w);
    }
  }
  float2 s0 = make_float2(v.x, v.y), s1 = make_float2(v.z, v.w), o0 = s0, o1 = s1;
  // this lane's part of the stage's 8 blocks of 4 steps
  float4 *out = (ADJ ? x.qs : x.hs) + (row * 4 + q) * seq_blocks(p.seqlen) + t_first / kSeqBlock;

  for (int s = 0; s < nst; ++s) {
    const bool live = t_first + s * dir + lane < L;
    float *m = mt + (s & 1) * QT * CROW;
    // ---- preparation: lane = timestep
#pragma unroll
    for (int j = 0; j < 4; ++j) m[(mt0 + j) * CROW + mrow] = rm.get(j);
    float dv[QCH], w[QCH];
    if constexpr (ALN) {
      const T *src = reinterpret_cast<const T *>(raw + (s & 1) * NRAW * RAW);
      cp_wait<0>();
      __syncwarp();
#pragma unroll
      for (int i = 0; i < QCH; ++i) dv[i] = to_f(src[i * QT + lane]);
#pragma unroll
      for (int i = 0; i < QCH; ++i) w[i] = to_f(src[QCH * QT + i * QT + lane]);
      if constexpr (GZ) {
#pragma unroll
        for (int i = 0; i < QCH; ++i) {
          const float z = to_f(src[2 * QCH * QT + i * QT + lane]);
          w[i] *= z * sigm(z);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        dv[i] = to_f(rd[i]);
        w[i] = to_f(rv[i]);
        if (GZ) {
          const float z = to_f(rz[i]);
          w[i] *= z * sigm(z);
        }
      }
    }
    if (s + 1 < nst) load_stage(s + 1);
#pragma unroll
    for (int i = 0; i < QCH; ++i) dv[i] += bias[i];
    if (p.delta_softplus) {
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        float e;
        dv[i] = softplus_e(dv[i], e);
      }
    }
#pragma unroll
    for (int i = 0; i < QCH; ++i) {
      const float d = live ? dv[i] : 0.f;                        // past the end: a = 1, and dy = u = 0
      *reinterpret_cast<float2 *>(dd + lane * DROW + 2 * i) = make_float2(d, ADJ ? w[i] : d * w[i]);
    }
    __syncthreads();      // the stage's C | B tile is complete; the other buffer's readers are a barrier behind
    // ---- the recurrence: lane = (channel, four states)
    if (nch > 0) {
#pragma unroll
      for (int k = 0; k < QT / TB; ++k) {
        const int blk = ADJ ? QT / TB - 1 - k : k;
        // entering a block: the boundaries of two neighbouring blocks are written together
        if ((k & 1) == 0) { o0 = s0; o1 = s1; }
        else if (mine) {
          if (ADJ) st_states(out + blk, s0, s1, o0, o1);
          else st_states(out + blk - 1, o0, o1, s0, s1);
        }
        float2 vd[TB];
        float4 vm[TB];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
          vd[i] = *reinterpret_cast<const float2 *>(dd + (blk * TB + i) * DROW + 2 * c);
          vm[i] = *reinterpret_cast<const float4 *>(m + (blk * TB + i) * CROW + QS * q);
        }
        float2 a0[TB], a1[TB];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
          const float2 d2 = make_float2(vd[i].x, vd[i].x);
          a0[i] = ex2f2(__fmul2_rn(d2, A2[0]));
          a1[i] = ex2f2(__fmul2_rn(d2, A2[1]));
        }
#pragma unroll
        for (int j = 0; j < TB; ++j) {
          const int i = ADJ ? TB - 1 - j : j;
          const float2 w2 = make_float2(vd[i].y, vd[i].y), m0 = make_float2(vm[i].x, vm[i].y), m1 = make_float2(vm[i].z, vm[i].w);
          if (ADJ) {
            s0 = __fmul2_rn(a0[i], __ffma2_rn(m0, w2, s0));
            s1 = __fmul2_rn(a1[i], __ffma2_rn(m1, w2, s1));
          } else {
            s0 = __ffma2_rn(a0[i], s0, __fmul2_rn(w2, m0));
            s1 = __ffma2_rn(a1[i], s1, __fmul2_rn(w2, m1));
          }
        }
      }
    }
    out += dir / kSeqBlock;
    __syncwarp();
  }
  if (ADJ && mine && x.t0 > 0) x.carry[row * 4 + q] = make_float4(s0.x, s0.y, s1.x, s1.y);
}

template <typename T, bool ALN, bool Z>
__global__ void __launch_bounds__(FW * 32, 5) selscan_seq_pre_kernel(const b200_selscan_bwd_args a, const SeqPre x) {
  extern __shared__ __align__(16) unsigned char smem_pre[];
  const int blk = (int)blockIdx.x;
  if (blk < x.adj) seq_walk<T, true, ALN, Z>(a, x, blk, 0, smem_pre);
  else seq_walk<T, false, ALN, Z>(a, x, (blk - x.adj) % x.adj, (blk - x.adj) / x.adj, smem_pre);
}

// ---------------------------------------------------------------------------------- gradients
constexpr int BW = 4;                       // warps per thread block = quarters of the states; also channels between two barriers
constexpr int KB = kSeqBlock;               // steps per lane
constexpr int BT = 32 * KB;                 // steps per thread block
constexpr int BCTA = 3;                     // resident thread blocks per SM that the registers allow

struct BwdSmem {
  float dl[BW][BT], du[BW][BT], dy[BW][BT];           // delta, delta u, dy of 4 channels
  float uu[BW][BT], sg[BW][BT];                       // u and the derivative of softplus, for the thread that wrote them
  float ss[BW][BW][2][BT];                            // [channel][warp]: sum over the warp's states of g B and of A2 w
  float4 st[2][BW][2][BW][32];                        // [buffer][channel][state, adjoint][warp][lane], a batch of channels ahead
  float da[BW][32][20];                               // [warp][lane]: 4 channels x 4 states of dA
  float A2[2][BW][QN];
};

template <typename T, bool VEC> __device__ __forceinline__ void st4(T *p, const float (&v)[4], int left) {
  if (VEC && left >= 4) {
    struct alignas(4 * sizeof(T)) { T v[4]; } r;
#pragma unroll
    for (int j = 0; j < 4; ++j) r.v[j] = from_f<T>(v[j]);
    if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4 *>(p) = reinterpret_cast<const uint4 &>(r);
    else *reinterpret_cast<uint2 *>(p) = reinterpret_cast<const uint2 &>(r);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (left > j) p[j] = from_f<T>(v[j]);
}
template <typename T, bool Z, bool VEC>
__global__ void __launch_bounds__(BW * 32, BCTA)
selscan_seq_bwd_kernel(const b200_selscan_bwd_args a, const float4 *__restrict__ hs, const float4 *__restrict__ qs, const int batches) {
  const b200_selscan_fwd_args &p = a.f;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BwdSmem &sm = *reinterpret_cast<BwdSmem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // uniform, and known to be
  const int L = p.seqlen;
  const int nwin = (L + BT - 1) / BT;
  const int nblk = seq_blocks(L);
  const int cpg = p.dim / p.n_groups;
  const int bw = (int)blockIdx.x, bg = bw / nwin;             // (batch row, group, window of 128 steps)
  const int b = bg / p.n_groups, g = bg % p.n_groups;
  const int i_begin = blockIdx.y * batches * BW, i_end = min(cpg, i_begin + batches * BW);      // channels within the group
  const int tw = (bw % nwin) * BT;                            // first step of the window
  const int t0 = tw + KB * lane, left = L - t0;               // the lane's 4 steps
  // recurrence: the warp's states 4 warp .. 4 warp + 3 of every channel; otherwise: all of channel `warp` of 4

  // B and C of the lane's steps and the warp's states stay in registers for all channels; they come
  // (and dB, dC leave) through shared memory, a coalesced row at a time
  float2 B0[KB], B1[KB], C0[KB], C1[KB], dB0[KB], dB1[KB], dC0[KB], dC1[KB];
  float *own = &sm.ss[0][warp][0][0];                         // a row of this warp's, and no other's
  const auto row_of = [&](const void *base, int64_t bs, int64_t gs, int64_t ns, int n) {
    const T *src = reinterpret_cast<const T *>(base) + (int64_t)b * bs + (int64_t)g * gs + (int64_t)n * ns;
#pragma unroll
    for (int k = 0; k < KB; ++k) own[lane + 32 * k] = tw + lane + 32 * k < L ? to_f(src[tw + lane + 32 * k]) : 0.f;
    __syncwarp();
    const float4 v = *reinterpret_cast<const float4 *>(own + 4 * lane);
    __syncwarp();
    return v;
  };
  const auto pairs_of = [&](const void *base, int64_t bs, int64_t gs, int64_t ns, int n, float2 (&v)[KB]) {
    const float4 x = row_of(base, bs, gs, ns, n), y = row_of(base, bs, gs, ns, n + 1);
    v[0] = make_float2(x.x, y.x); v[1] = make_float2(x.y, y.y); v[2] = make_float2(x.z, y.z); v[3] = make_float2(x.w, y.w);
  };
  pairs_of(p.B, p.B_bs, p.B_gs, p.B_ns, QS * warp, B0);
  pairs_of(p.B, p.B_bs, p.B_gs, p.B_ns, QS * warp + 2, B1);
  pairs_of(p.C, p.C_bs, p.C_gs, p.C_ns, QS * warp, C0);
  pairs_of(p.C, p.C_bs, p.C_gs, p.C_ns, QS * warp + 2, C1);
#pragma unroll
  for (int t = 0; t < KB; ++t) dB0[t] = dB1[t] = dC0[t] = dC1[t] = make_float2(0.f, 0.f);

  // this thread's steps in channel i + warp of an activation; the channel may lie past the group's end:
  // then nothing is read or written
  const int64_t lane_bytes = (int64_t)t0 * (int)sizeof(T);
  const auto at = [&](const void *base, int64_t bs, int64_t ds, int i) {
    const char *r = reinterpret_cast<const char *>(base) + b * bs * (int)sizeof(T);
    return reinterpret_cast<T *>(const_cast<char *>(r + ((int64_t)(g * cpg + i + warp) * (int)(ds * (int)sizeof(T)) + lane_bytes)));
  };
  const float *bp = reinterpret_cast<const float *>(p.delta_bias), *Dvp = reinterpret_cast<const float *>(p.D);

  Quad<T, VEC> rd, ru, rg, rz, ro;
  float rbias = 0.f, rA = 0.f, rD = 0.f;
  auto load_rows = [&](int i) {
    const int n = i + warp < i_end ? left : 0;
    const T *pd = at(p.delta, p.delta_bs, p.delta_ds, i), *pu = at(p.u, p.u_bs, p.u_ds, i), *pg = at(a.dout, a.dout_bs, a.dout_ds, i);
    const T *pz = Z ? at(p.z, p.z_bs, p.z_ds, i) : nullptr, *po = Z ? at(p.out, p.out_bs, p.out_ds, i) : nullptr;
    if (n >= 4) {
      rd.load4(pd);
      ru.load4(pu);
      rg.load4(pg);
      if (Z) { rz.load4(pz); ro.load4(po); }
    } else {
      rd.load(pd, n);
      ru.load(pu, n);
      rg.load(pg, n);
      if (Z) { rz.load(pz, n); ro.load(po, n); }
    }
    rbias = bp && i + warp < i_end ? bp[g * cpg + i + warp] : 0.f;
    rD = Dvp && i + warp < i_end ? Dvp[g * cpg + i + warp] : 0.f;
    if (tid < BW * QN && i + tid / QN < i_end)
      rA = decay2(reinterpret_cast<const float *>(p.A)[(int64_t)(g * cpg + i + tid / QN) * p.A_ds + (int64_t)(tid % QN) * p.A_ns]);
  };
  auto prep = [&](int i, int buf) {
    const int n = i + warp < i_end ? left : 0;
    float d[4], u[4], s[4], y[4], du[4], dz[4], oz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      u[j] = ru.get(j);
      y[j] = rg.get(j);
      d[j] = rd.get(j) + rbias;
      s[j] = 1.f;
    }
    if (p.delta_softplus) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x = d[j];
        float e;
        d[j] = softplus_e(x, e);
        s[j] = x > 20.f ? 1.f : e * rcpf(1.f + e);
      }
    }
    if (Z) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float z = rz.get(j), o = ro.get(j);
        const float sz = sigm(z), zs = z * sz;
        dz[j] = y[j] * o * (sz + zs * (1.f - sz));
        oz[j] = o * zs;
        y[j] *= zs;
      }
      st4<T, VEC>(at(a.dz, a.dz_bs, a.dz_ds, i), dz, n);
      if (p.out_z) st4<T, VEC>(at(p.out_z, p.out_z_bs, p.out_z_ds, i), oz, n);
    }
    if (n < 4) {                             // outside: a = 1, and u = dy = 0
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j >= n) d[j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) du[j] = d[j] * u[j];
    *reinterpret_cast<float4 *>(&sm.dl[warp][4 * lane]) = make_float4(d[0], d[1], d[2], d[3]);
    *reinterpret_cast<float4 *>(&sm.du[warp][4 * lane]) = make_float4(du[0], du[1], du[2], du[3]);
    *reinterpret_cast<float4 *>(&sm.dy[warp][4 * lane]) = make_float4(y[0], y[1], y[2], y[3]);
    *reinterpret_cast<float4 *>(&sm.uu[warp][4 * lane]) = make_float4(u[0], u[1], u[2], u[3]);
    *reinterpret_cast<float4 *>(&sm.sg[warp][4 * lane]) = make_float4(s[0], s[1], s[2], s[3]);
    if (tid < BW * QN) sm.A2[buf][tid / QN][tid % QN] = rA;
  };
  // states and adjoints: (batch, dim, 4 quarters of the states, blocks); a lane reads only what it fetched itself
  const int64_t sd = left > 0 ? (int64_t)4 * nblk : 0;
  const int64_t so = left > 0 ? (((int64_t)b * p.dim + g * cpg + i_begin) * 4 + warp) * nblk + t0 / KB : 0;
  const float4 *hp = hs + so, *qp = qs + so;
  auto load_states = [&](int i, int buf) {           // of the next BW channels
#pragma unroll
    for (int k = 0; k < BW; ++k) {
      const int n = left > 0 && i + k < i_end ? 16 : 0;
      cp16(&sm.st[buf][k][0][warp][lane], n ? hp : hs, n);          // copies of 0 bytes name a mapped address too
      cp16(&sm.st[buf][k][1][warp][lane], n ? qp : qs, n);
      hp += sd;
      qp += sd;
    }
    cp_commit();
  };

  load_rows(i_begin);
  load_states(i_begin, 0);
  prep(i_begin, 0);
  __syncthreads();
  for (int i = i_begin, buf = 0; i < i_end; i += BW, buf ^= 1) {
    cp_wait<0>();
    const float Dv = rD;
    if (i + BW < i_end) {
      load_rows(i + BW);
      load_states(i + BW, buf ^ 1);
    }
    // ---- the recurrences of 4 channels over the lane's 4 steps, from the state and the adjoint that enter them
#pragma unroll
    for (int k = 0; k < BW; ++k) {
      const float4 vh = sm.st[buf][k][0][warp][lane], vq = sm.st[buf][k][1][warp][lane];
      const float4 vA = *reinterpret_cast<const float4 *>(&sm.A2[buf][k][QS * warp]);
      const float4 vd = *reinterpret_cast<const float4 *>(&sm.dl[k][4 * lane]);
      const float4 vu = *reinterpret_cast<const float4 *>(&sm.du[k][4 * lane]);
      const float4 vy = *reinterpret_cast<const float4 *>(&sm.dy[k][4 * lane]);
      const float d[4] = {vd.x, vd.y, vd.z, vd.w}, u[4] = {vu.x, vu.y, vu.z, vu.w}, y[4] = {vy.x, vy.y, vy.z, vy.w};
      const float2 A0 = make_float2(vA.x, vA.y), A1 = make_float2(vA.z, vA.w);
      float2 H0[KB + 1], H1[KB + 1], w0[KB], w1[KB];
      H0[0] = make_float2(vh.x, vh.y);
      H1[0] = make_float2(vh.z, vh.w);
      float2 q0 = make_float2(vq.x, vq.y), q1 = make_float2(vq.z, vq.w);
#pragma unroll
      for (int t = 0; t < KB; ++t) {
        const float2 d2 = make_float2(d[t], d[t]), u2 = make_float2(u[t], u[t]);
        w0[t] = ex2f2(__fmul2_rn(d2, A0));
        w1[t] = ex2f2(__fmul2_rn(d2, A1));
        H0[t + 1] = __ffma2_rn(w0[t], H0[t], __fmul2_rn(u2, B0[t]));
        H1[t + 1] = __ffma2_rn(w1[t], H1[t], __fmul2_rn(u2, B1[t]));
      }
      float2 s0 = make_float2(0.f, 0.f), s1 = s0;
      float gB[KB], gA[KB];
#pragma unroll
      for (int t = KB - 1; t >= 0; --t) {
        const float2 d2 = make_float2(d[t], d[t]), u2 = make_float2(u[t], u[t]), y2 = make_float2(y[t], y[t]);
        const float2 g0 = __ffma2_rn(C0[t], y2, q0), g1 = __ffma2_rn(C1[t], y2, q1);
        dC0[t] = __ffma2_rn(H0[t + 1], y2, dC0[t]);
        dC1[t] = __ffma2_rn(H1[t + 1], y2, dC1[t]);
        dB0[t] = __ffma2_rn(g0, u2, dB0[t]);
        dB1[t] = __ffma2_rn(g1, u2, dB1[t]);
        q0 = __fmul2_rn(w0[t], g0);
        q1 = __fmul2_rn(w1[t], g1);
        const float2 x0 = __fmul2_rn(q0, H0[t]), x1 = __fmul2_rn(q1, H1[t]);
        s0 = __ffma2_rn(d2, x0, s0);
        s1 = __ffma2_rn(d2, x1, s1);
        const float2 xB = __ffma2_rn(g1, B1[t], __fmul2_rn(g0, B0[t])), xA = __ffma2_rn(x1, A1, __fmul2_rn(x0, A0));
        gB[t] = xB.x + xB.y;
        gA[t] = xA.x + xA.y;
      }
      *reinterpret_cast<float4 *>(&sm.ss[k][warp][0][4 * lane]) = make_float4(gB[0], gB[1], gB[2], gB[3]);
      *reinterpret_cast<float4 *>(&sm.ss[k][warp][1][4 * lane]) = make_float4(gA[0], gA[1], gA[2], gA[3]);
      *reinterpret_cast<float4 *>(&sm.da[warp][lane][4 * k]) = make_float4(s0.x, s0.y, s1.x, s1.y);
    }
    __syncthreads();
    // ---- du, ddelta of the thread's 4 steps
    {
      const int n = i + warp < i_end ? left : 0;
      float2 b0 = make_float2(0.f, 0.f), b1 = b0, a0 = b0, a1 = b0;
#pragma unroll
      for (int w = 0; w < BW; ++w) {
        const float4 x = *reinterpret_cast<const float4 *>(&sm.ss[warp][w][0][4 * lane]), z = *reinterpret_cast<const float4 *>(&sm.ss[warp][w][1][4 * lane]);
        b0 = __fadd2_rn(b0, make_float2(x.x, x.y));
        b1 = __fadd2_rn(b1, make_float2(x.z, x.w));
        a0 = __fadd2_rn(a0, make_float2(z.x, z.y));
        a1 = __fadd2_rn(a1, make_float2(z.z, z.w));
      }
      const float gB[4] = {b0.x, b0.y, b1.x, b1.y}, gA[4] = {a0.x, a0.y, a1.x, a1.y};
      const float4 d4 = *reinterpret_cast<const float4 *>(&sm.dl[warp][4 * lane]), u4 = *reinterpret_cast<const float4 *>(&sm.uu[warp][4 * lane]);
      const float4 s4 = *reinterpret_cast<const float4 *>(&sm.sg[warp][4 * lane]), y4 = *reinterpret_cast<const float4 *>(&sm.dy[warp][4 * lane]);
      const float d[4] = {d4.x, d4.y, d4.z, d4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
      const float s[4] = {s4.x, s4.y, s4.z, s4.w}, y[4] = {y4.x, y4.y, y4.z, y4.w};
      float du[4], dd[4], sD = 0.f, sb;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        du[j] = fmaf(Dv, y[j], d[j] * gB[j]);
        dd[j] = fmaf(u[j], gB[j], gA[j] * 0.6931471805599453f) * s[j];
        sD = fmaf(y[j], u[j], sD);
      }
      if (n < 4) {                           // the walk runs on past the end, where q may not be zero
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j >= n) dd[j] = 0.f;
      }
      sb = (dd[0] + dd[1]) + (dd[2] + dd[3]);
      st4<T, VEC>(at(a.du, a.du_bs, a.du_ds, i), du, n);
      st4<T, VEC>(at(a.ddelta, a.ddelta_bs, a.ddelta_ds, i), dd, n);
      // one value per half warp, then the sum over its 16 lanes
      float v = (lane < 16 ? sD : sb) + __shfl_xor_sync(0xffffffffu, lane < 16 ? sb : sD, 16);
#pragma unroll
      for (int m = 8; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
      if ((lane & 15) == 0 && i + warp < i_end) {
        float *o = reinterpret_cast<float *>(lane == 0 ? a.dD : a.ddelta_bias);
        if (o) atomicAdd(o + g * cpg + i + warp, v);
      }
    }
    // ---- dA of the warp's 4 states of 4 channels, summed over the lanes: lane (r, k) adds up lanes 4r .. 4r + 3
    // of channel k, then the 8 groups r are folded, each folding leaving a lane half of its 4 states
    {
      const int k = lane & 3, r = lane >> 2;
      const float4 x = *reinterpret_cast<const float4 *>(&sm.da[warp][4 * r][4 * k]), y = *reinterpret_cast<const float4 *>(&sm.da[warp][4 * r + 1][4 * k]);
      const float4 z = *reinterpret_cast<const float4 *>(&sm.da[warp][4 * r + 2][4 * k]), w = *reinterpret_cast<const float4 *>(&sm.da[warp][4 * r + 3][4 * k]);
      const float2 lo = __fadd2_rn(__fadd2_rn(make_float2(x.x, x.y), make_float2(y.x, y.y)), __fadd2_rn(make_float2(z.x, z.y), make_float2(w.x, w.y)));
      const float2 hi = __fadd2_rn(__fadd2_rn(make_float2(x.z, x.w), make_float2(y.z, y.w)), __fadd2_rn(make_float2(z.z, z.w), make_float2(w.z, w.w)));
      const bool u1 = (lane & 16) != 0, u0 = (lane & 8) != 0;
      const float v0 = (u1 ? hi.x : lo.x) + __shfl_xor_sync(0xffffffffu, u1 ? lo.x : hi.x, 16);
      const float v1 = (u1 ? hi.y : lo.y) + __shfl_xor_sync(0xffffffffu, u1 ? lo.y : hi.y, 16);
      float v = (u0 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, u0 ? v0 : v1, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      if ((lane & 4) == 0 && i + k < i_end)
        atomicAdd(reinterpret_cast<float *>(a.dA) + (int64_t)(g * cpg + i + k) * a.dA_ds + (int64_t)(QS * warp + (lane >> 4) * 2 + ((lane >> 3) & 1)) * a.dA_ns, v);
    }
    if (i + BW < i_end) prep(i + BW, buf ^ 1);
    __syncthreads();
  }
  const auto row_out = [&](void *base, int64_t bs, int64_t gs, int64_t ns, int n, float4 v) {
    *reinterpret_cast<float4 *>(own + 4 * lane) = v;
    __syncwarp();
    float *dst = reinterpret_cast<float *>(base) + (int64_t)b * bs + (int64_t)g * gs + (int64_t)n * ns;
#pragma unroll
    for (int k = 0; k < KB; ++k)
      if (tw + lane + 32 * k < L) atomicAdd(dst + tw + lane + 32 * k, own[lane + 32 * k]);
    __syncwarp();
  };
  const auto pairs_out = [&](void *base, int64_t bs, int64_t gs, int64_t ns, int n, const float2 (&v)[KB]) {
    row_out(base, bs, gs, ns, n, make_float4(v[0].x, v[1].x, v[2].x, v[3].x));
    row_out(base, bs, gs, ns, n + 1, make_float4(v[0].y, v[1].y, v[2].y, v[3].y));
  };
  pairs_out(a.dB, a.dB_bs, a.dB_gs, a.dB_ns, QS * warp, dB0);
  pairs_out(a.dB, a.dB_bs, a.dB_gs, a.dB_ns, QS * warp + 2, dB1);
  pairs_out(a.dC, a.dC_bs, a.dC_gs, a.dC_ns, QS * warp, dC0);
  pairs_out(a.dC, a.dC_bs, a.dC_gs, a.dC_ns, QS * warp + 2, dC1);
}

template <typename T> bool quads_aligned(const b200_selscan_bwd_args &a) {
  const b200_selscan_fwd_args &p = a.f;
  const auto ok = [](const void *ptr, int64_t bs, int64_t ds) {
    return !ptr || ((reinterpret_cast<uintptr_t>(ptr) % (4 * sizeof(T))) == 0 && bs % 4 == 0 && ds % 4 == 0);
  };
  return ok(p.delta, p.delta_bs, p.delta_ds) && ok(p.u, p.u_bs, p.u_ds) && ok(a.dout, a.dout_bs, a.dout_ds) &&
         (!p.z || (ok(p.z, p.z_bs, p.z_ds) && ok(p.out, p.out_bs, p.out_ds) && ok(a.dz, a.dz_bs, a.dz_ds))) &&
         ok(p.out_z, p.out_z_bs, p.out_z_ds) && ok(a.du, a.du_bs, a.du_ds) && ok(a.ddelta, a.ddelta_bs, a.ddelta_ds);
}

// a: a window of `total` steps that begins at step t0, as a call of its own (x and stage_h aside)
template <typename T> int launch_bwd(const b200_selscan_bwd_args &a, int t0, int total, void *work, cudaStream_t st) {
  const b200_selscan_fwd_args &f = a.f;
  const int cpg = f.dim / f.n_groups;
  // the carry comes first: it lies in the same place for windows of any length
  const int64_t rows4 = (int64_t)f.batch * f.dim * 4;
  float4 *carry = reinterpret_cast<float4 *>(work), *hs = carry + rows4, *qs = hs + rows4 * seq_blocks(f.seqlen);
  // 1. states and adjoints.  Pieces of the states' walk start where the forward call left a state: every
  // 256 steps is enough parallelism; without stage states only the 2048-step checkpoints of x are there
  SeqPre x{};
  x.hs = hs;
  x.qs = qs;
  x.carry = carry;
  x.t0 = t0;
  x.total = total;
  x.piece = f.stage_h ? kStage : kChunk;
  x.tiles = f.n_groups * ((cpg + FW * QCH - 1) / (FW * QCH));
  x.adj = f.batch * x.tiles;
  const bool al = row16<T>(f.u, f.u_bs, f.u_ds) && row16<T>(f.delta, f.delta_bs, f.delta_ds) && row16<T>(a.dout, a.dout_bs, a.dout_ds) &&
                  row16<T>(f.B, f.B_bs, f.B_ns) && f.B_gs % EPC<T> == 0 && row16<T>(f.C, f.C_bs, f.C_ns) && f.C_gs % EPC<T> == 0 &&
                  (!f.z || row16<T>(f.z, f.z_bs, f.z_ds));
  auto kp = f.z ? (al ? selscan_seq_pre_kernel<T, true, true> : selscan_seq_pre_kernel<T, false, true>)
                : (al ? selscan_seq_pre_kernel<T, true, false> : selscan_seq_pre_kernel<T, false, false>);
  const int smem = PRE_FIX + (al ? FW * 2 * (f.z ? 3 : 2) * QCH * QT * (int)sizeof(T) : 0);
  const int64_t blocks = (int64_t)x.adj * (1 + (f.seqlen + x.piece - 1) / x.piece);
  cudaError_t e = cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return (int)e; }
  kp<<<(unsigned)blocks, FW * 32, smem, st>>>(a, x);
  if (int err = launch_status()) return err;
  // 2. the gradients
  const bool vec = quads_aligned<T>(a);
  auto k = f.z ? (vec ? selscan_seq_bwd_kernel<T, true, true> : selscan_seq_bwd_kernel<T, true, false>)
               : (vec ? selscan_seq_bwd_kernel<T, false, true> : selscan_seq_bwd_kernel<T, false, false>);
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BwdSmem));
  if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return (int)e; }
  // How many thread blocks share a window's channels: the waves of resident blocks that this takes, times the
  // batches of 4 channels that each block then has and about two more for its own start and end
  const int64_t windows = (int64_t)f.batch * f.n_groups * ((f.seqlen + BT - 1) / BT);
  const int64_t slots = (int64_t)BCTA * sm_count_current();
  const int nb = (cpg + BW - 1) / BW;
  int per = nb;
  int64_t best = INT64_MAX;
  for (int split = 1; split <= nb && split <= 64; ++split) {
    const int n = (nb + split - 1) / split;
    const int64_t cost = ((windows * ((nb + n - 1) / n) + slots - 1) / slots) * (n + 2);
    if (cost < best) { best = cost; per = n; }
  }
  const dim3 grid((unsigned)windows, (unsigned)((nb + per - 1) / per));
  k<<<grid, BW * 32, sizeof(BwdSmem), st>>>(a, hs, qs, per);
  return launch_status();
}

// the workspace of one channel of one batch row over `steps` steps: carry, hs, qs
int64_t channel_bytes(int steps) { return 2 * (int64_t)seq_blocks(steps) * QN * 4 + QN * 4; }

// One launch's share of the call: batch rows, channels (whole groups, or part of one) and steps from these on.
struct Slice {
  int b0, rows, c0, chans, t0, steps;
};
// How many channels of a row a workspace of `room` channels takes at a time: whole groups; or less than one group, then
// whole thread blocks or whole warps of the walks where there is room for one.
int slice_channels(const b200_selscan_fwd_args &f, int64_t room) {
  const int cpg = f.dim / f.n_groups;
  if (room >= cpg) return (int)(room / cpg < f.n_groups ? room / cpg : f.n_groups) * cpg;
  const int n = (int)room;
  return n >= FW * QCH ? n / (FW * QCH) * (FW * QCH) : n >= QCH ? n / QCH * QCH : n;
}

int run_slice(const b200_selscan_bwd_args &a, const Slice &w, void *work, cudaStream_t st) {
  const int es = act_size(a.f.dtype), total = a.f.seqlen;
  const int cpg = a.f.dim / a.f.n_groups, g0 = w.c0 / cpg;
  b200_selscan_bwd_args s = a;
  b200_selscan_fwd_args &f = s.f;
  f.batch = w.rows;
  f.dim = w.chans;
  f.seqlen = w.steps;
  f.n_groups = w.chans > cpg ? w.chans / cpg : 1;
  const int64_t n_chunks = (total + kChunk - 1) / kChunk, row0 = (int64_t)w.b0 * a.f.dim + w.c0;
  const auto at = [](const void *p, int64_t bytes) { return p ? (void *)(const_cast<char *>(reinterpret_cast<const char *>(p)) + bytes) : nullptr; };
  const auto act = [&](const void *p, int64_t bs, int64_t ds) { return at(p, (w.b0 * bs + w.c0 * ds + w.t0) * es); };
  f.u = act(f.u, f.u_bs, f.u_ds);
  f.delta = act(f.delta, f.delta_bs, f.delta_ds);
  f.z = act(f.z, f.z_bs, f.z_ds);
  f.out = act(f.out, f.out_bs, f.out_ds);
  f.out_z = act(f.out_z, f.out_z_bs, f.out_z_ds);
  f.B = at(f.B, (w.b0 * f.B_bs + g0 * f.B_gs + w.t0) * es);
  f.C = at(f.C, (w.b0 * f.C_bs + g0 * f.C_gs + w.t0) * es);
  f.A = at(f.A, w.c0 * f.A_ds * 4);
  f.D = at(f.D, (int64_t)w.c0 * 4);
  f.delta_bias = at(f.delta_bias, (int64_t)w.c0 * 4);
  f.x = at(f.x, row0 * n_chunks * 2 * QN * 4);
  if (f.stage_h) f.stage_h = at(f.stage_h, row0 * ((total + f.stage_len - 1) / f.stage_len) * QN * 4);
  s.dout = act(s.dout, s.dout_bs, s.dout_ds);
  s.du = act(s.du, s.du_bs, s.du_ds);
  s.ddelta = act(s.ddelta, s.ddelta_bs, s.ddelta_ds);
  s.dz = act(s.dz, s.dz_bs, s.dz_ds);
  s.dA = at(s.dA, w.c0 * s.dA_ds * 4);
  s.dB = at(s.dB, (w.b0 * s.dB_bs + g0 * s.dB_gs + w.t0) * 4);
  s.dC = at(s.dC, (w.b0 * s.dC_bs + g0 * s.dC_gs + w.t0) * 4);
  s.dD = at(s.dD, (int64_t)w.c0 * 4);
  s.ddelta_bias = at(s.ddelta_bias, (int64_t)w.c0 * 4);
  s.h_in = at(s.h_in, row0 * QN * 4);
  s.q_in = at(s.q_in, row0 * QN * 4);
  if (f.dtype == B200_F32) return launch_bwd<float>(s, w.t0, total, work, st);
  if (f.dtype == B200_BF16) return launch_bwd<__nv_bfloat16>(s, w.t0, total, work, st);
  return launch_bwd<__half>(s, w.t0, total, work, st);
}

// How a call is cut for a workspace of so many bytes: into batch rows while one fits; one row into windows of the
// sequence, from the last to the first, which keeps all its channels in flight (the adjoint is one serial walk however
// it is cut); and only where not even the shortest window of all channels fits into channels as well.
struct Cut {
  int rows, chans, steps;        // rows < 1: not even one channel fits
};
Cut cut_of(const b200_selscan_fwd_args &f, int64_t bytes) {
  const int64_t row = channel_bytes(f.seqlen) * f.dim;
  if (bytes >= row) return {(int)(bytes / row < f.batch ? bytes / row : f.batch), f.dim, f.seqlen};
  const int window = f.seqlen < kChunk ? f.seqlen : kChunk;      // windows begin where a checkpoint is
  if (bytes >= channel_bytes(window) * f.dim) {
    int64_t n = bytes / (channel_bytes(window) * f.dim);
    while (channel_bytes((int)(n + 1) * window) * f.dim <= bytes) ++n;      // one carry for all of them
    return {1, f.dim, (int)n * window};
  }
  const int64_t room = bytes / channel_bytes(window);
  return {room < 1 ? 0 : 1, room < 1 ? 0 : slice_channels(f, room), window};
}

}  // namespace

// Transient device memory of the backward call: the states and adjoints of a slice, 32 bytes per channel and step.
// A slice holds at most 2 GiB of them.
int64_t selscan_seq_bwd_bytes(const b200_selscan_fwd_args &f) {
  const Cut c = cut_of(f, (int64_t)2 << 30);
  return channel_bytes(c.steps) * c.chans * c.rows;
}

bool selscan_seq_bwd_supported(const b200_selscan_bwd_args &a) {
  if (!selscan_seq_supported(a.f)) return false;
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.h_in) | reinterpret_cast<uintptr_t>(a.q_in);
  for (const int64_t ds : {a.f.u_ds, a.f.delta_ds, a.f.z_ds, a.f.out_ds, a.f.out_z_ds, a.dout_ds, a.du_ds, a.ddelta_ds, a.dz_ds})
    if (ds * 4 != (int32_t)(ds * 4)) return false;          // row pitches in bytes are 32-bit numbers in the kernel
  const int64_t cpg = a.f.dim / a.f.n_groups;
  const int64_t gx = (int64_t)a.f.batch * a.f.n_groups * ((a.f.seqlen + BT - 1) / BT);
  const int64_t pre = (int64_t)a.f.batch * a.f.n_groups * ((cpg + FW * QCH - 1) / (FW * QCH)) * (1 + (a.f.seqlen + kStage - 1) / kStage);
  return (al & 15) == 0 && gx < (int64_t)1 << 31 && pre < (int64_t)1 << 31;
}

int selscan_seq_bwd(const b200_selscan_bwd_args &a, void *work, int64_t work_bytes, cudaStream_t st) {
  const int dim = a.f.dim, cpg = dim / a.f.n_groups, L = a.f.seqlen;
  const Cut cut = cut_of(a.f, work_bytes);
  B200_REQUIRE(cut.rows >= 1, B200_ERR_SHAPE, "selscan_bwd: the workspace is too small for one channel and %d steps", cut.steps);
  for (int b = 0; b < a.f.batch; b += cut.rows)
    for (int c = 0, n; c < dim; c += n) {
      n = cut.chans < dim - c ? cut.chans : dim - c;
      if (cut.chans < cpg && n > cpg - c % cpg) n = cpg - c % cpg;      // not past the end of a group
      const int rows = cut.rows < a.f.batch - b ? cut.rows : a.f.batch - b;
      for (int t = (L - 1) / cut.steps * cut.steps; t >= 0; t -= cut.steps)
        if (int e = run_slice(a, {b, rows, c, n, t, cut.steps < L - t ? cut.steps : L - t}, work, st)) return e;
    }
  return 0;
}

}  // namespace b200
