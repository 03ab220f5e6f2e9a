// Host-side interface of the tcgen05 grouped GEMM (grouped_gemm.cu), used by the fused-layer entry points.
#pragma once

#include "mok_common.cuh"

namespace mok {

// A grouped-GEMM problem over schedule rows.  Rows are grouped by expert: expert e owns the contiguous,
// 256-aligned row range [cum[e], cum[e+1]) given by `tokens_per_expert`; only rows inside the window
// [row_begin, min(row_end, *num_tokens)) are touched, and activation buffers are indexed by (row - row_begin)
// (the macrobatch ring).  A dense problem (one expert, `dense_rows` rows) has tokens_per_expert == nullptr.
struct GemmProblem {
    const int32_t* tokens_per_expert = nullptr;
    const int32_t* num_tokens = nullptr;
    int num_experts = 1;
    int dense_rows = 0;
    int row_begin = 0, row_end = 0;
    int buffer_rows = 0;   // rows of the activation buffers (macrobatch size, or T for a dense problem)
    // optional: rows of each expert that can be non-zero (the rest of its 256-aligned range is zero padding).  The K loop of
    // a weight gradient ends at this count rounded up to the K step; the rows forms of the bf16 GEMM then put the tokens on
    // the N side of the MMA and leave the padding out (routed_gemm.cu)
    const int32_t* occupied_rows = nullptr;
    uint32_t* status = nullptr;
};

// Output rows of a rows form that are stored into the token owners' slot buffers: row r goes to
// ptr[peer_rank[r]][peer_token[r], :] (local or peer memory; padding rows nowhere), and with row_scalar its fp32 value
// row_scalar[r - row_begin] to scalar_ptr[peer_rank[r]][peer_token[r]].  One GEMM epilogue then does what a plain store
// and a combine pass over the stored rows would do.
struct RowScatter {
    uint64_t ptr[MOK_MAX_EP] = {};
    uint64_t scalar_ptr[MOK_MAX_EP] = {};
    const int32_t* peer_rank = nullptr;    // [schedule rows]; nullptr = not scattered
    const int32_t* peer_token = nullptr;
    const float* row_scalar = nullptr;
    int ep = 0, routes_per_rank = 0;
};

// D_s[row, :] = A[row, :K] * B_s[e]^T for s < n_sets (two sets share A: gate and up projections).
// With `scatter` (one set only) D0 is nullptr and the rows go to their slots.
// b_is_kn = false: B_s is [E, N, K];  true: B_s is [E, K, N].
int launch_rows_gemm(const GemmProblem& pb, const void* A, int K, const void* B0, const void* B1, void* D0, void* D1,
                     int N, bool b_is_kn, cudaStream_t stream, const RowScatter* scatter = nullptr);

// Forward gate and up projections with the SwiGLU in the epilogue: gate = A * Wg[e]^T, up = A * Wu[e]^T (both stored as
// bf16 [rows, N]) and hidden = silu(gate) * up computed from the stored (rounded) values, optionally clamped.
int launch_gate_up_fused(const GemmProblem& pb, const void* A, int K, const void* Wg, const void* Wu, void* gate, void* up,
                         void* hidden, int N, bool has_limit, float limit, cudaStream_t stream);

// Input gradient of the down projection with the SwiGLU backward in the epilogue: d_hidden = A * B[e] (B stored [E, K, N])
// rounded to bf16 and stored, d_gate / d_up from it and the saved gate / up [rows, N].
// row_partial (or nullptr): [rows, N / 128] sums of d_hidden * hidden for the router-weight gradient (launch_router_grad).
// Needs pb.occupied_rows.
int launch_down_dgrad_fused(const GemmProblem& pb, const void* A, int K, const void* B, const void* gate, const void* up, void* d_hidden,
                            void* d_gate, void* d_up, float* row_partial, int N, bool has_limit, float limit, cudaStream_t stream);

// D[row, :] = A0[row, :K] * B0[e] + A1[row, :K] * B1[e] with B_s stored [E, K, N] (gate+up input gradient).
int launch_rows_gemm_dual(const GemmProblem& pb, const void* A0, const void* A1, int K, const void* B0, const void* B1,
                          void* D, int N, cudaStream_t stream, const RowScatter* scatter = nullptr);

// D[e] [M, N] (+)= A[rows_e, M]^T * B[rows_e, N]; accumulates when expert e's rows began before row_begin.
// out_f32: D is fp32 and is overwritten (single-window problems only).
int launch_wgrad_gemm(const GemmProblem& pb, const void* A, int M, const void* B, int N, void* D, cudaStream_t stream,
                      bool out_f32 = false);

// fp32 D[row, :] = A[row, :K] * (B_hi[e] + B_lo[e])^T with B_* stored [E, N, K]; B_lo may be nullptr.  Two bf16 terms
// carry an fp32 weight matrix to about 16 mantissa bits, which the router logits need (fp32 accumulation throughout).
int launch_rows_gemm_f32(const GemmProblem& pb, const void* A, int K, const void* B_hi, const void* B_lo, float* D, int N,
                         cudaStream_t stream);

}  // namespace mok
