// Internal (C++) entry points behind the extern "C" layer in api.cu.
#pragma once
#include <cuda_runtime.h>
#include "../../include/lrnnx_b200.h"

namespace b200 {

constexpr int kStage = 256;       // the state-parallel backward starts its walks every so many steps
// Spacings of stage_h that it can start them from: whole 32-step stages, of which one ends where each walk begins.
// States of any other spacing are neither written nor read.
inline bool stage_usable(int stage_len) { return stage_len > 0 && stage_len % 32 == 0 && kStage % stage_len == 0; }

// coverage kernels: every variant (selscan_generic.cu)
int selscan_fwd_generic(const b200_selscan_fwd_args &a, cudaStream_t st);
int selscan_bwd_generic(const b200_selscan_bwd_args &a, cudaStream_t st);

// state-parallel kernels (selscan_seq.cu, selscan_seq_bwd.cu)
bool selscan_seq_supported(const b200_selscan_fwd_args &a);
int selscan_seq_stage_len(const b200_selscan_fwd_args &a);
int selscan_seq_fwd(const b200_selscan_fwd_args &a, cudaStream_t st);
bool selscan_seq_bwd_supported(const b200_selscan_bwd_args &a);
int64_t selscan_seq_bwd_bytes(const b200_selscan_fwd_args &f);
int selscan_seq_bwd(const b200_selscan_bwd_args &a, void *work, int64_t work_bytes, cudaStream_t st);

// one state per channel, constant B and C: RG-LRU and S7 (selscan_row1.cu)
bool selscan_row1_supported(const b200_selscan_fwd_args &a);
int selscan_row1_fwd(const b200_selscan_fwd_args &a, cudaStream_t st);
int selscan_row1_bwd(const b200_selscan_bwd_args &a, cudaStream_t st);

// status word of the tensor-core projection kernel (cgemm_tc.cu)
int cgemm_status_read();

// status word of the decode-step pipeline (ssu.cu): non-zero after an expired bounded wait
int ssu_status_read();

}  // namespace b200
