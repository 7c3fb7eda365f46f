// extern "C" entry points of liblrnnx_b200.so: argument validation and
// dispatch to the kernels.  See include/lrnnx_b200.h for the contract.
#include "common.cuh"
#include "dispatch.h"
#include <cstring>

namespace b200 {

static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

static int check_selscan(const b200_selscan_fwd_args &a) {
  B200_REQUIRE(a.u && a.delta && a.A && a.B && a.C, B200_ERR_NULL, "selscan: u, delta, A, B, C must be non-null");
  B200_REQUIRE(a.batch > 0 && a.dim > 0 && a.seqlen > 0 && a.dstate > 0, B200_ERR_SHAPE,
               "selscan: batch, dim, seqlen, dstate must be positive");
  // same limit as csrc/selective_scan/selective_scan_cpu.cpp:327
  B200_REQUIRE(a.dstate <= kMaxDState, B200_ERR_SHAPE, "selective_scan only supports state dimension <= 256");
  B200_REQUIRE(a.n_groups >= 1 && a.dim % a.n_groups == 0, B200_ERR_SHAPE,
               "selscan: dim (%d) must be a multiple of n_groups (%d)", a.dim, a.n_groups);
  B200_REQUIRE(a.dtype == B200_F32 || a.dtype == B200_F16 || a.dtype == B200_BF16, B200_ERR_DTYPE,
               "selscan: unknown activation dtype %d", a.dtype);
  B200_REQUIRE(a.method >= B200_DISC_ZOH && a.method <= B200_DISC_S7, B200_ERR_DTYPE,
               "Discretization method not supported");
  // csrc/selective_scan/selective_scan_cpu.cpp:299-305
  B200_REQUIRE(!(a.method == B200_DISC_S7 && a.is_complex), B200_ERR_DTYPE,
               "S7 discretization only supports real (float) weights, not complex");
  B200_REQUIRE(!(a.method == B200_DISC_RGLRU && a.is_complex), B200_ERR_DTYPE,
               "RGLRU discretization only supports real (float) weights, not complex");
  return 0;
}

}  // namespace b200

using namespace b200;

extern "C" {

const char *b200_last_error(void) { return g_err; }
int b200_abi_version(void) { return 7; }

// size of an argument block as this library was compiled; lets a binding
// verify its own struct layout before the first call
int b200_sizeof(const char *name) {
  if (!name) return -1;
  if (!strcmp(name, "b200_selscan_fwd_args")) return (int)sizeof(b200_selscan_fwd_args);
  if (!strcmp(name, "b200_selscan_bwd_args")) return (int)sizeof(b200_selscan_bwd_args);
  if (!strcmp(name, "b200_selscan_fixup_args")) return (int)sizeof(b200_selscan_fixup_args);
  if (!strcmp(name, "b200_selscan_adjsum_args")) return (int)sizeof(b200_selscan_adjsum_args);
  if (!strcmp(name, "b200_simpscan_args")) return (int)sizeof(b200_simpscan_args);
  if (!strcmp(name, "b200_ssu_args")) return (int)sizeof(b200_ssu_args);
  if (!strcmp(name, "b200_s4_args")) return (int)sizeof(b200_s4_args);
  if (!strcmp(name, "b200_s5_step_args")) return (int)sizeof(b200_s5_step_args);
  if (!strcmp(name, "b200_conv1d_args")) return (int)sizeof(b200_conv1d_args);
  if (!strcmp(name, "b200_rmsnorm_args")) return (int)sizeof(b200_rmsnorm_args);
  if (!strcmp(name, "b200_cgemm_args")) return (int)sizeof(b200_cgemm_args);
  if (!strcmp(name, "b200_cgemm_planes_args")) return (int)sizeof(b200_cgemm_planes_args);
  if (!strcmp(name, "b200_cgemm_grad_args")) return (int)sizeof(b200_cgemm_grad_args);
  if (!strcmp(name, "b200_xent_args")) return (int)sizeof(b200_xent_args);
  if (!strcmp(name, "b200_skinny_linear_args")) return (int)sizeof(b200_skinny_linear_args);
  return -1;
}

int b200_selscan_fwd(const b200_selscan_fwd_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "selscan_fwd: null argument block");
  if (int e = check_selscan(*args)) return e;
  B200_REQUIRE(args->out && args->x, B200_ERR_NULL, "selscan_fwd: out and x must be non-null");
  B200_REQUIRE(!args->z || args->out_z, B200_ERR_NULL, "selscan_fwd: out_z is required when z is given");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (args->l_segments > 1 && args->seg_work) {
    const int64_t S = args->l_segments, len = args->seg_len;
    B200_REQUIRE(len > 0 && len % 32 == 0 && S * len >= args->seqlen && (S - 1) * len < args->seqlen, B200_ERR_SHAPE,
                 "selscan_fwd: %d segments of %d steps do not make up %d", args->l_segments, args->seg_len, args->seqlen);
    B200_REQUIRE((reinterpret_cast<uintptr_t>(args->seg_work) & 15) == 0, B200_ERR_ALIGN, "selscan_fwd: seg_work must be 16-byte aligned");
  }
  if (selscan_seq_supported(*args)) {
    b200_selscan_fwd_args a = *args;
    if (a.stage_len != kStage) a.stage_h = nullptr;
    return selscan_seq_fwd(a, st);
  }
  B200_REQUIRE(args->l_segments <= 1, B200_ERR_UNSUPPORTED,
               "selscan_fwd: l_segments > 1 is only available on the state-parallel kernels' shape class");
  if (selscan_row1_supported(*args)) return selscan_row1_fwd(*args, st);
  return selscan_fwd_generic(*args, st);
}

int b200_selscan_stage_states(const b200_selscan_fwd_args *args) {
  if (!args || check_selscan(*args) || args->l_segments > 1) return 0;
  b200_selscan_fwd_args a = *args;
  a.stage_h = nullptr;
  return selscan_seq_supported(a) ? kStage : 0;
}

int64_t b200_selscan_bwd_work_bytes(const b200_selscan_bwd_args *args) {
  if (!args || check_selscan(args->f) || !selscan_seq_bwd_supported(*args)) return 0;
  return selscan_seq_bwd_bytes(args->f);
}

int b200_selscan_bwd(const b200_selscan_bwd_args *args, void *stream) {
  B200_REQUIRE(args, B200_ERR_NULL, "selscan_bwd: null argument block");
  if (int e = check_selscan(args->f)) return e;
  const b200_selscan_fwd_args &f = args->f;
  B200_REQUIRE(args->dout && args->du && args->ddelta && args->dA && args->dB && args->dC, B200_ERR_NULL,
               "selscan_bwd: dout, du, ddelta, dA, dB, dC must be non-null");
  // csrc/selective_scan/selective_scan_cpu.cpp:573
  B200_REQUIRE(f.x || f.seqlen <= kChunk, B200_ERR_NULL, "selscan_bwd: x is required when seqlen > 2048");
  // csrc/selective_scan/selective_scan_cpu.cpp:550
  B200_REQUIRE(!f.z || (f.out && args->dz), B200_ERR_NULL, "selscan_bwd: out and dz are required when z is given");
  B200_REQUIRE(!f.deltaA || args->ddeltaA, B200_ERR_NULL, "selscan_bwd: ddeltaA is required when deltaA is given");
  B200_REQUIRE(!f.D || args->dD, B200_ERR_NULL, "selscan_bwd: dD is required when D is given");
  B200_REQUIRE(!f.delta_bias || args->ddelta_bias, B200_ERR_NULL,
               "selscan_bwd: ddelta_bias is required when delta_bias is given");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  B200_REQUIRE(!(args->h_in || args->q_in) || !f.is_complex, B200_ERR_UNSUPPORTED, "selscan_bwd: h_in / q_in need a real A");
  if (!args->h_in && !args->q_in && selscan_row1_supported(f)) return selscan_row1_bwd(*args, st);
  if (!selscan_seq_bwd_supported(*args)) return selscan_bwd_generic(*args, st);
  b200_selscan_bwd_args a = *args;
  // the forward's stage states start from zero: with a state entering the sequence they are not its states
  if (a.f.stage_len != kStage || a.h_in) a.f.stage_h = nullptr;
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a.work) & 31) == 0, B200_ERR_ALIGN, "selscan_bwd: work must be 32-byte aligned");
  if (a.work) return selscan_seq_bwd(a, a.work, a.work_bytes, st);
  void *work = nullptr;
  const int64_t bytes = selscan_seq_bwd_bytes(f);
  if (cudaMallocAsync(&work, (size_t)bytes, st) != cudaSuccess) {
    cudaGetLastError();                       // no room for the workspace: the coverage kernel needs none
    return selscan_bwd_generic(*args, st);
  }
  const int e = selscan_seq_bwd(a, work, bytes, st);
  cudaFreeAsync(work, st);
  return e;
}

}  // extern "C"
