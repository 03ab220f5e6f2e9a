// Host-side interface of routed_gemm.cu: the rows forms of the bf16 GEMM for problems that know their occupied rows.  The launch
// functions of grouped_gemm.cuh check problem and sizes and come here.
#pragma once

#include "grouped_gemm.cuh"

namespace mok {

int launch_routed_gemm(const GemmProblem& pb, const void* A0, const void* A1, int K, const void* B0, const void* B1, void* D, int N,
                       bool b_is_kn, cudaStream_t stream, const RowScatter* scatter);
int launch_routed_gate_up(const GemmProblem& pb, const void* A, int K, const void* Wg, const void* Wu, void* gate, void* up, void* hidden,
                          int N, bool has_limit, float limit, cudaStream_t stream);
int launch_routed_down_dgrad(const GemmProblem& pb, const void* A, int K, const void* B, const void* gate, const void* up, void* d_hidden,
                             void* d_gate, void* d_up, float* row_partial, int N, bool has_limit, float limit, cudaStream_t stream);

}  // namespace mok
