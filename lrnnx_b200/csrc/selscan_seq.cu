// State-parallel selective scan, forward: real A, "mamba" discretization, variable B and C,
// dstate 16, any length, any channel count, any alignment.
//
// With 16 states per channel the scan is bound by the SFU (one ex2 per (t, n, channel): 16 lanes
// per clock per SM) and by instruction issue, not by HBM.  A scan across lanes costs more issue
// slots than the recurrence itself, so there is none: a lane owns 4 states of one channel and
// walks the time axis, a warp is 8 channels x 4 lanes, and a thread block of 4 warps shares the
// B | C tile of a stage of 32 steps.
//   * per step and lane: three 128-bit shared loads (B, C, {delta, delta, delta u, delta u}: the
//     pairs come out as operands of the packed fp32 instructions), 2 + 2 packed products, 4 ex2,
//     2 packed FMAs for the state, 2 for the output, one store of the lane's share of y;
//   * per stage a lane turns into one timestep: it loads its step's element of each of the warp's
//     8 rows (coalesced over the lanes, no alignment needed), one stage ahead in registers, applies
//     bias and softplus once per (channel, step), and after the stage adds up the four shares of y,
//     applies the D skip and the z gate and stores;
//   * the state at the end of every stage_len steps is an optional output (stage_h) for the backward.
// Measured, batch 8 x 1536 channels x 2048 steps, bf16, gated: 220 us (a kernel that scans across the lanes of a warp:
// 302 us; the SFU's floor: 110 us with softplus and gate).  1536 warps are 2.6 per scheduler: the rest is latency
// (IPC 1.8 of 4, SFU 56 %, shared-memory pipe 61 %).  64 x 4096 x 512: 1.00 ms (1.52 ms).  Any length: a 4 x 776 x 1531
// float32 call takes 90 us where the one-warp-per-row kernel that used to serve odd lengths took 1.1 ms.
// Few rows: a step takes a thread block 60 ns however idle the GPU is, so a call whose blocks do not fill it is scanned in
// segments, in two passes: states alone from zero for all segments but the last, then each segment from the state that
// the ones before it lead to (the fold is a short loop at a block's start).  Nothing is corrected afterwards, and 16-bit
// outputs are rounded once.  1 x 64 x 8192: 547 -> 25 us; 1 x 1536 x 512 bf16: 37 -> 18 us (a kernel that scans across lanes: 20).
// The two passes cost 1.5 times one, so calls that fill the GPU are not cut like this.
// Groups of at most 16 channels run in thread blocks of two warps: half of four would only help with the B | C tile.
// Results match csrc/selective_scan/selective_scan.cuh:73-382 of lrnnx for this shape class.
#include "selscan_seq.cuh"

namespace b200 {
namespace {
using namespace seq;

constexpr int TB = 4;             // steps per block of the recurrence

// Segments of the sequence that are scanned side by side in two passes: the first leaves the state that a segment reaches
// from zero and the sum of its step sizes, the second starts every segment from the state that the ones before it lead to.
struct SeqSeg {
  float4 *h;            // (segments, batch * dim, 4); null: a segment is a scan of its own, from a zero state
  float *d;             // (segments, batch * dim)
  int len;              // steps per segment
};

// ALN: every row starts on a 16-byte boundary.  Z: gated.  FW: warps per thread block.  SUM: the first pass of two.
template <typename T, bool ALN, bool Z, int FW, bool SUM>
__global__ void __launch_bounds__(FW * 32, 12 / FW) selscan_seq_fwd_kernel(const b200_selscan_fwd_args p, const SeqSeg seg) {
  constexpr int RAW = QCH * QT * (int)sizeof(T);                 // 8 rows of a stage
  __shared__ __align__(16) float bc_all[2][QT * QROW];           // B | C of a stage, float32, [t][n]
  __shared__ __align__(16) float dd_all[FW][QT * DROW];          // {delta, delta u} per (t, channel)
  __shared__ __align__(16) float ys_all[SUM ? 1 : FW][QT * QROW];       // partial outputs [t][channel][lane share]
  extern __shared__ __align__(16) unsigned char raw_all[];       // ALN: [warp][2 stages][u, delta, (z)] rows as they are
  constexpr int NRAW = Z ? 3 : 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *raw = raw_all + (ALN ? warp * 2 * NRAW * RAW : 0);
  const int c = lane & 7, q = lane >> 3;                         // recurrence: channel, quarter of the states
  const int cpg = p.dim / p.n_groups;
  const int tpg = (cpg + FW * QCH - 1) / (FW * QCH);
  const int bg = blockIdx.x / tpg;
  const int b = bg / p.n_groups, g = bg % p.n_groups;
  const int cin = ((blockIdx.x % tpg) * FW + warp) * QCH;        // first channel of this warp within the group
  const int nch = min(cpg - cin, QCH);                           // <= 0: the warp only helps with the B | C tile
  const int d0 = g * cpg + cin;
  const int n_chunks = (p.seqlen + kChunk - 1) / kChunk;
  const int t_begin = (int)blockIdx.y * seg.len;                 // blockIdx.y = segment of the sequence
  if (t_begin >= p.seqlen) return;
  const int L = min(p.seqlen, t_begin + seg.len);
  const int nst = (L - t_begin + QT - 1) / QT;
  const int dl = nch > 0 ? d0 : g * cpg;                         // a valid row for idle warps' pointers

  // ---- operands: 16-byte asynchronous copies into per-warp buffers, or elements into registers
  RowCopy<T> cu, cd, cz;
  T ru[ALN ? 1 : QCH], rd[ALN ? 1 : QCH], rz[ALN ? 1 : QCH];
  const T *Up = nullptr, *Dp = nullptr, *Zp = nullptr;
  if constexpr (ALN) {
    cu.init(p.u, p.u_bs, p.u_ds, b, dl, lane, nch, t_begin);
    cd.init(p.delta, p.delta_bs, p.delta_ds, b, dl, lane, nch, t_begin);
    if (Z) cz.init(p.z, p.z_bs, p.z_ds, b, dl, lane, nch, t_begin);
  } else {
    Up = reinterpret_cast<const T *>(p.u) + (int64_t)b * p.u_bs + (int64_t)dl * p.u_ds + t_begin + lane;
    Dp = reinterpret_cast<const T *>(p.delta) + (int64_t)b * p.delta_bs + (int64_t)dl * p.delta_ds + t_begin + lane;
    if (Z) Zp = reinterpret_cast<const T *>(p.z) + (int64_t)b * p.z_bs + (int64_t)dl * p.z_ds + t_begin + lane;
  }
  // B | C: a thread takes the same QT / FW steps of one of the 32 rows in every stage
  constexpr int BCS = QT / FW;
  const T *BCp = lane < QN
      ? reinterpret_cast<const T *>(p.B) + (int64_t)b * p.B_bs + (int64_t)g * p.B_gs + (int64_t)lane * p.B_ns
      : reinterpret_cast<const T *>(p.C) + (int64_t)b * p.C_bs + (int64_t)g * p.C_gs + (int64_t)(lane - QN) * p.C_ns;
  BCp += t_begin + BCS * warp;
  constexpr int BCC = BCS / EPC<T>;
  uint4 rbc[BCC];
  auto load_stage = [&](int s) {
    const int left = L - (t_begin + s * QT);
#pragma unroll
    for (int k = 0; k < BCC; ++k) {
      rbc[k] = ld_chunk<T>(BCp + k * EPC<T>, SUM && lane >= QN ? 0 : left - BCS * warp - k * EPC<T>, ALN);
    }
    BCp += QT;
    if constexpr (ALN) {
      const int mine = left - (lane % PPR<T>) * EPC<T>;
      cu.fetch(raw + (s & 1) * NRAW * RAW, lane, nch, mine);
      cd.fetch(raw + ((s & 1) * NRAW + 1) * RAW, lane, nch, mine);
      if constexpr (Z) { cz.fetch(raw + ((s & 1) * NRAW + 2) * RAW, lane, nch, mine); cz.p += QT; }
      cu.p += QT;
      cd.p += QT;
      cp_commit();
    } else {
      const bool ok = lane < left;
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        const bool oki = ok && i < nch;
        rd[i] = oki ? Dp[(int64_t)i * p.delta_ds] : from_f<T>(0.f);
        ru[i] = oki ? Up[(int64_t)i * p.u_ds] : from_f<T>(0.f);
        if (Z) rz[i] = oki ? Zp[(int64_t)i * p.z_ds] : from_f<T>(0.f);
      }
      Up += QT;
      Dp += QT;
      if (Z) Zp += QT;
    }
  };
  load_stage(0);

  float *dd = dd_all[warp], *ys = ys_all[SUM ? 0 : warp];
  float2 A2[2];
  {
    const float *A = reinterpret_cast<const float *>(p.A) + (int64_t)(dl + min(c, max(nch - 1, 0))) * p.A_ds;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      A2[j] = make_float2(decay2(A[(int64_t)(QS * q + 2 * j) * p.A_ns]), decay2(A[(int64_t)(QS * q + 2 * j + 1) * p.A_ns]));
  }
  float bias[QCH], Dv[QCH], cs[QCH];
#pragma unroll
  for (int i = 0; i < QCH; ++i) {
    bias[i] = p.delta_bias && i < nch ? reinterpret_cast<const float *>(p.delta_bias)[dl + i] : 0.f;
    Dv[i] = p.D && i < nch ? reinterpret_cast<const float *>(p.D)[dl + i] : 0.f;
    cs[i] = 0.f;                                                 // this lane's steps' share of the sum of delta
  }
  float2 h0 = make_float2(0.f, 0.f), h1 = h0;
  const bool mine = c < nch;
  const int64_t row = (int64_t)b * p.dim + d0 + c, n_rows = (int64_t)p.batch * p.dim;
  float before = 0.f;                                            // sum of delta before the segment
  if (!SUM && seg.h && mine) {
    const float4 *hj = seg.h + row * 4 + q;
    const float *dj = seg.d + row;
#pragma unroll 4
    for (int j = 0; j < (int)blockIdx.y; ++j, hj += n_rows * 4, dj += n_rows) {
      const float4 hv = *hj;
      const float d = *dj;
      h0 = __ffma2_rn(ex2f2(__fmul2_rn(make_float2(d, d), A2[0])), h0, make_float2(hv.x, hv.y));
      h1 = __ffma2_rn(ex2f2(__fmul2_rn(make_float2(d, d), A2[1])), h1, make_float2(hv.z, hv.w));
      before += d;
    }
  }

  for (int s = 0; s < nst; ++s) {
    const int t0 = t_begin + s * QT;
    const bool live = t0 + lane < L;
    float *bc = bc_all[s & 1];
    // ---- preparation: lane = timestep
#pragma unroll
    for (int k = 0; k < BCC; ++k) {
      float v[EPC<T>];
      unpack(rbc[k], v, T());
#pragma unroll
      for (int j = 0; j < EPC<T>; ++j) bc[(BCS * warp + k * EPC<T> + j) * QROW + lane] = v[j];
    }
    T uc[ALN ? 1 : QCH], zc[ALN ? 1 : QCH];
    float dv[QCH];
    T *su = reinterpret_cast<T *>(raw + (s & 1) * NRAW * RAW);
    T *sz = reinterpret_cast<T *>(raw + ((s & 1) * NRAW + 2) * RAW);
    if constexpr (ALN) {
      const T *sd = reinterpret_cast<const T *>(raw + ((s & 1) * NRAW + 1) * RAW);
      cp_wait<0>();
      __syncwarp();
#pragma unroll
      for (int i = 0; i < QCH; ++i) dv[i] = to_f(sd[i * QT + lane]);
    } else {
#pragma unroll
      for (int i = 0; i < QCH; ++i) { dv[i] = to_f(rd[i]); uc[i] = ru[i]; zc[i] = rz[i]; }
    }
    if (s + 1 < nst) load_stage(s + 1);       // ALN: the other buffer was last read before the previous __syncwarp
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
      const float d = live ? dv[i] : 0.f;                          // past the end: a = 1, b = 0
      const float u = to_f(ALN ? su[i * QT + lane] : uc[ALN ? 0 : i]);
      cs[i] += d;
      *reinterpret_cast<float2 *>(dd + lane * DROW + 2 * i) = make_float2(d, d * u);
    }
    __syncthreads();      // the stage's B | C tile is complete; the other buffer's readers are a barrier behind
    // ---- the recurrence: lane = (channel, four states)
    if (nch > 0) {
#pragma unroll
      for (int blk = 0; blk < QT / TB; ++blk) {
        float2 vd[TB];
        float4 vb[TB], vc[TB];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
          const int t = blk * TB + i;
          vd[i] = *reinterpret_cast<const float2 *>(dd + t * DROW + 2 * c);
          vb[i] = *reinterpret_cast<const float4 *>(bc + t * QROW + QS * q);
          if (!SUM) vc[i] = *reinterpret_cast<const float4 *>(bc + t * QROW + QN + QS * q);
        }
        float2 a0[TB], a1[TB];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
          const float2 d2 = make_float2(vd[i].x, vd[i].x);
          a0[i] = ex2f2(__fmul2_rn(d2, A2[0]));
          a1[i] = ex2f2(__fmul2_rn(d2, A2[1]));
        }
#pragma unroll
        for (int i = 0; i < TB; ++i) {
          const float2 u2 = make_float2(vd[i].y, vd[i].y);
          h0 = __ffma2_rn(a0[i], h0, __fmul2_rn(u2, make_float2(vb[i].x, vb[i].y)));
          h1 = __ffma2_rn(a1[i], h1, __fmul2_rn(u2, make_float2(vb[i].z, vb[i].w)));
          if (SUM) continue;
          const float2 y2 = __ffma2_rn(h1, make_float2(vc[i].z, vc[i].w), __fmul2_rn(h0, make_float2(vc[i].x, vc[i].y)));
          ys[(blk * TB + i) * QROW + 4 * c + q] = y2.x + y2.y;
        }
      }
      if (!SUM && p.stage_h && mine && (((t0 + QT) % p.stage_len) == 0 || t0 + QT >= p.seqlen)) {
        const int64_t n_stages = (p.seqlen + p.stage_len - 1) / p.stage_len;
        *reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.stage_h) + (row * n_stages + t0 / p.stage_len) * QN + QS * q) =
            make_float4(h0.x, h0.y, h1.x, h1.y);
      }
    }
    if (SUM ? s == nst - 1 : ((t0 + QT) % kChunk) == 0 || t0 + QT >= p.seqlen) {      // checkpoint, or the segment's summary
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        const float v = warp_sum(cs[i]);
        if (i == c) sum = v;
      }
      if (SUM && mine) {
        seg.h[((int64_t)blockIdx.y * n_rows + row) * 4 + q] = make_float4(h0.x, h0.y, h1.x, h1.y);
        if (q == 0) seg.d[(int64_t)blockIdx.y * n_rows + row] = sum;
      } else if (mine) {
        sum += before;
        float4 *xr = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.x) + (row * n_chunks + t0 / kChunk) * 2 * QN + 2 * QS * q);
        const float2 P0 = ex2f2(__fmul2_rn(make_float2(sum, sum), A2[0])), P1 = ex2f2(__fmul2_rn(make_float2(sum, sum), A2[1]));
        xr[0] = make_float4(P0.x, h0.x, P0.y, h0.y);
        xr[1] = make_float4(P1.x, h1.x, P1.y, h1.y);
      }
    }
    __syncwarp();
    if constexpr (SUM) continue;
    // ---- output: lane = timestep
    float yv[QCH];
#pragma unroll
    for (int i = 0; i < QCH; ++i) {
      const float4 v = *reinterpret_cast<const float4 *>(ys + lane * QROW + 4 * i);
      yv[i] = fmaf(Dv[i], to_f(ALN ? su[i * QT + lane] : uc[ALN ? 0 : i]), (v.x + v.y) + (v.z + v.w));
    }
    if constexpr (ALN) {
      // in place over the rows of u and z, then out in 16-byte pieces
#pragma unroll
      for (int i = 0; i < QCH; ++i) {
        su[i * QT + lane] = from_f<T>(yv[i]);
        if (Z) {
          const float z = to_f(sz[i * QT + lane]);
          sz[i * QT + lane] = from_f<T>(yv[i] * z * sigm(z));
        }
      }
      __syncwarp();
      const int off = (lane % PPR<T>) * EPC<T>, left = L - t0 - off;
#pragma unroll
      for (int k = 0; k < CPL<T>; ++k) {
        const int r = lane / PPR<T> + 4 * k;
        if (r < nch && left > 0) {
          st_chunk<T>(reinterpret_cast<T *>(p.out) + (int64_t)b * p.out_bs + (int64_t)(d0 + r) * p.out_ds + t0 + off,
                      *reinterpret_cast<const uint4 *>(su + (lane + 32 * k) * EPC<T>), left);
          if (Z)
            st_chunk<T>(reinterpret_cast<T *>(p.out_z) + (int64_t)b * p.out_z_bs + (int64_t)(d0 + r) * p.out_z_ds + t0 + off,
                        *reinterpret_cast<const uint4 *>(sz + (lane + 32 * k) * EPC<T>), left);
        }
      }
    } else if (live) {
      T *Op = reinterpret_cast<T *>(p.out) + (int64_t)b * p.out_bs + (int64_t)dl * p.out_ds + t0 + lane;
      T *OZp = Z ? reinterpret_cast<T *>(p.out_z) + (int64_t)b * p.out_z_bs + (int64_t)dl * p.out_z_ds + t0 + lane : nullptr;
#pragma unroll
      for (int i = 0; i < QCH; ++i)
        if (i < nch) {
          Op[(int64_t)i * p.out_ds] = from_f<T>(yv[i]);
          if (Z) {
            const float z = to_f(zc[ALN ? 0 : i]);
            OZp[(int64_t)i * p.out_z_ds] = from_f<T>(yv[i] * z * sigm(z));
          }
        }
    }
    __syncwarp();
  }
}

// Warps per thread block: four share a B | C tile; a group of at most 16 channels has work for two.
int warps_per_block(const b200_selscan_fwd_args &a) { return a.dim / a.n_groups > 2 * QCH ? 4 : 2; }

int64_t fwd_blocks(const b200_selscan_fwd_args &a) {
  const int cpg = a.dim / a.n_groups, per = warps_per_block(a) * QCH;
  return (int64_t)a.batch * a.n_groups * ((cpg + per - 1) / per);
}

template <typename T> bool rows_aligned(const b200_selscan_fwd_args &a) {
  return row16<T>(a.u, a.u_bs, a.u_ds) && row16<T>(a.delta, a.delta_bs, a.delta_ds) && row16<T>(a.B, a.B_bs, a.B_ns) && a.B_gs % EPC<T> == 0 &&
         row16<T>(a.C, a.C_bs, a.C_ns) && a.C_gs % EPC<T> == 0 && row16<T>(a.out, a.out_bs, a.out_ds) &&
         (!a.z || (row16<T>(a.z, a.z_bs, a.z_ds) && row16<T>(a.out_z, a.out_z_bs, a.out_z_ds)));
}

template <typename T, bool ALN, bool Z, int FW, bool SUM>
int launch(const b200_selscan_fwd_args &a, const SeqSeg &seg, int segments, cudaStream_t st) {
  auto k = selscan_seq_fwd_kernel<T, ALN, Z, FW, SUM>;
  const int smem = ALN ? FW * 2 * (Z ? 3 : 2) * QCH * QT * (int)sizeof(T) : 0;      // u, delta, (z) as they are
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return (int)e; }
  k<<<dim3((unsigned)fwd_blocks(a), (unsigned)segments), FW * 32, smem, st>>>(a, seg);
  return launch_status();
}
template <typename T, int FW> int launch_warps(const b200_selscan_fwd_args &a, const SeqSeg &seg, int segments, cudaStream_t st) {
  const bool al = rows_aligned<T>(a);
  if (seg.h)
    if (int e = al ? launch<T, true, false, FW, true>(a, seg, segments - 1, st) : launch<T, false, false, FW, true>(a, seg, segments - 1, st)) return e;
  if (a.z) return al ? launch<T, true, true, FW, false>(a, seg, segments, st) : launch<T, false, true, FW, false>(a, seg, segments, st);
  return al ? launch<T, true, false, FW, false>(a, seg, segments, st) : launch<T, false, false, FW, false>(a, seg, segments, st);
}

template <typename T> int launch_fwd(const b200_selscan_fwd_args &a, cudaStream_t st) {
  b200_selscan_fwd_args p = a;
  const int n = a.l_segments > 1 ? a.l_segments : 1;
  SeqSeg seg{nullptr, nullptr, a.seqlen};
  if (n > 1 && a.seg_work) {
    const int64_t rows = (int64_t)a.batch * a.dim;
    seg = {reinterpret_cast<float4 *>(a.seg_work), reinterpret_cast<float *>(a.seg_work) + (int64_t)n * rows * QN, a.seg_len};
  } else if (n > 1) {
    seg.len = ((a.seqlen + n - 1) / n + kChunk - 1) / kChunk * kChunk;      // whole checkpoint chunks
    p.stage_h = nullptr;                          // segments start from zero: their states are not the sequence's
  }
  return warps_per_block(a) == 4 ? launch_warps<T, 4>(p, seg, n, st) : launch_warps<T, 2>(p, seg, n, st);
}
}  // namespace

bool selscan_seq_supported(const b200_selscan_fwd_args &a) {
  if (a.is_complex || a.method != B200_DISC_MAMBA || !a.var_B || !a.var_C || a.deltaA || a.dstate != QN) return false;
  // 128-bit accesses: the states in x and stage_h
  if ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.stage_h)) & 15) return false;
  return fwd_blocks(a) < (int64_t)1 << 31;
}

int selscan_seq_fwd(const b200_selscan_fwd_args &a, cudaStream_t st) {
  if (a.dtype == B200_F32) return launch_fwd<float>(a, st);
  if (a.dtype == B200_BF16) return launch_fwd<__nv_bfloat16>(a, st);
  return launch_fwd<__half>(a, st);
}

}  // namespace b200
