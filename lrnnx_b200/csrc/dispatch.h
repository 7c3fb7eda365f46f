// Internal (C++) entry points behind the extern "C" layer in api.cu.
#pragma once
#include <cuda_runtime.h>
#include "../../include/lrnnx_b200.h"

namespace b200 {

// Spacing of the states that the state-parallel forward leaves for the backward, which starts its own walk from them:
// pieces of 256 steps fill the GPU wherever the rows alone do not, and closer states would only cost memory (every 32
// steps they are as large as a 16-bit activation).  States of any other spacing are neither written nor read.
constexpr int kStage = 256;

// coverage kernels: every variant (selscan_generic.cu)
int selscan_fwd_generic(const b200_selscan_fwd_args &a, cudaStream_t st);
int selscan_bwd_generic(const b200_selscan_bwd_args &a, cudaStream_t st);

// state-parallel kernels (selscan_seq.cu, selscan_seq_bwd.cu)
bool selscan_seq_supported(const b200_selscan_fwd_args &a);
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
