// Grouped bf16 GEMM over routed rows with the tokens on the N side of the MMA: D^T[features, tokens] = W[e] * A^T.
//
// The schedule pads every expert to 256 rows.  With the rows on the M side (grouped_gemm.cu) an MMA costs the same however
// many of its 256 rows carry a token; M = 256 is what a CTA pair needs to run at full rate.  The N side may be any multiple
// of 32, so here a tile is 256 output features x up to 256 tokens, and N, the bytes staged and the time of the MMA follow the
// rows that are occupied, rounded up to 64 (the K step of the weight-gradient GEMMs, which read the results).
// Everything else is as there: a cluster of two CTAs per tile, TMA into a 6-stage ring of 64-wide K steps, tcgen05.mma
// cta_group::2 issued by the leader, two 256-column accumulators, a persistent walk over the same tile list and the same sums
// in the same order (the results are bitwise equal).  Tensor memory lanes are features and columns are tokens, so the
// epilogue turns blocks of 32 tokens x 32 features around in shared memory before it stores them.
//
// At 32 rows per expert (128 experts, hidden 2048, intermediate 768) gate / up takes 171 us instead of 187 us and the down
// projection 79 instead of 85 us; both then read the weights at 4.7 to 5.1 TB/s.  With full tiles the transposition in the
// epilogue costs a little more than it saves; row_trim_enabled() in layer.cu says where the line lies.
// Needs GemmProblem::occupied_rows; dense problems and callers without it use grouped_gemm.cu.
#include "gemm_tiles.cuh"
#include "routed_gemm.cuh"
#include "swiglu_math.cuh"

namespace mok {
namespace {

using namespace tiles;

constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int W_TILE_BYTES = BM_CTA * BK * 2;        // 16 KB: 128 features
constexpr int T_TILE_BYTES = BN_CTA * BK * 2;        // 16 KB: up to 128 tokens
constexpr int STAGE_BYTES = W_TILE_BYTES + T_TILE_BYTES;
constexpr int CHUNK_BYTES = 64 * BK * 2;             // one 64(MN) x 64(K) block of an MN-major operand: 8 KB
constexpr int kTokenStep = 64;                       // granularity of N
constexpr int kTokenBox = 32;                        // rows of a token copy of a partial tile: N / 2 per CTA is a multiple of it
constexpr int kHalf = 64;                            // gate / up form: gate rows, then up rows, of a CTA's weight tile

constexpr int EPI_STORE = 0, EPI_GATE_UP = 1, EPI_SWIGLU_BWD = 2;

// Eight epilogue warps in two groups of four: a group covers the CTA's 128 tensor-memory lanes and takes every other block
// of 32 tokens.  It stages the block as 32 rows of 128 features (bf16; 272 bytes a row: free of bank conflicts both ways) and
// stores rows of 256 bytes, so that a store instruction touches 4 lines.  One group of four warps that turned 32 x 32 blocks
// around by itself took longer than the MMAs of a tile with K = 768 (down projection of 147k rows 706 instead of 520 us).
constexpr int kThreads = 64 + 256;
constexpr int kRowPitchBytes = 2 * BM_CTA + 16;
constexpr int kBlockBytes = 32 * kRowPitchBytes;

struct SharedLayout {
    static constexpr int kFull = STAGES * STAGE_BYTES;            // STAGES x 8 B (leader's are used)
    static constexpr int kEmpty = kFull + 8 * STAGES;             // STAGES x 8 B
    static constexpr int kTmemFull = kEmpty + 8 * STAGES;         // 2 x 8 B
    static constexpr int kTmemEmpty = kTmemFull + 16;             // 2 x 8 B (leader's are used)
    static constexpr int kTmemPtr = kTmemEmpty + 16;              // 4 B
    static constexpr int kAbort = kTmemPtr + 4;                   // 4 B
    static constexpr int kEpilogue = kFull + 256;                 // staging
    static constexpr int kCum = kEpilogue + 2 * kBlockBytes;      // (E + 1) x 4 B, then E x 4 B occupied rows
};

// Occupied rows of a tile, rounded up to kTokenStep; 0 for a tile that holds padding only.
__device__ __forceinline__ int tile_tokens(const int* cum, const int* occupied, const Tile& tile) {
    const int left = occupied[tile.expert] - (tile.row0 - cum[tile.expert]);
    return min(max((left + kTokenStep - 1) / kTokenStep * kTokenStep, 0), BN);
}

// The four epilogue warps of a group meet; true when all of them came with `ok`.  Every warp gets here equally often whatever
// happened to its (bounded) waits, so the barrier always completes.
__device__ __forceinline__ bool group_sync(int group, bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.and.pred p, %2, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(all)
        : "r"(static_cast<uint32_t>(ok)), "r"(group + 1)
        : "memory");
    return all != 0;
}
__device__ __forceinline__ void group_sync(int group) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(group + 1) : "memory"); }

template <bool CLAMP>
__device__ __forceinline__ uint4 swiglu_vec(const uint4& g, const uint4& u, float limit) {
    return make_uint4(swiglu_pair<CLAMP>(g.x, u.x, limit), swiglu_pair<CLAMP>(g.y, u.y, limit), swiglu_pair<CLAMP>(g.z, u.z, limit),
                      swiglu_pair<CLAMP>(g.w, u.w, limit));
}

template <bool CLAMP>
__device__ __forceinline__ float swiglu_bwd_vec(const uint4& g, const uint4& u, const uint4& dh, float limit, uint4& dg, uint4& du) {
    float sum = swiglu_bwd_pair<CLAMP>(g.x, u.x, dh.x, limit, dg.x, du.x);
    sum += swiglu_bwd_pair<CLAMP>(g.y, u.y, dh.y, limit, dg.y, du.y);
    sum += swiglu_bwd_pair<CLAMP>(g.z, u.z, dh.z, limit, dg.z, du.z);
    sum += swiglu_bwd_pair<CLAMP>(g.w, u.w, dh.w, limit, dg.w, du.w);
    return sum;
}

// One operand set: weights, and the tokens in boxes for a full tile (128 rows) and for a partial one.
struct RoutedMaps {
    CUtensorMap w, full, part;
};

// W_MN: the weights are stored [E, K, N] (input gradients), otherwise [E, N, K].
template <bool W_MN, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
routed_gemm_kernel(const __grid_constant__ RoutedMaps m0, const __grid_constant__ RoutedMaps m1, const KernelParams p) {
    static_assert(EPI == EPI_STORE || W_MN == (EPI == EPI_SWIGLU_BWD),
                  "gate / up is a forward form, the SwiGLU backward an input gradient");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_full = smem_base + SharedLayout::kFull;
    const uint32_t bar_empty = smem_base + SharedLayout::kEmpty;
    const uint32_t bar_tmem_full = smem_base + SharedLayout::kTmemFull;
    const uint32_t bar_tmem_empty = smem_base + SharedLayout::kTmemEmpty;
    volatile uint32_t* tmem_ptr_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + SharedLayout::kTmemPtr);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + SharedLayout::kAbort);
    int* cum = reinterpret_cast<int*>(smem_gen + SharedLayout::kCum);
    int* occupied = cum + p.num_experts + 1;

    // nothing to do for a row window behind the schedule's last row: leave before anything is set up (both CTAs alike)
    if (min(p.row_end, *p.num_tokens) <= p.row_begin) return;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int cta_rank = static_cast<int>(cluster_cta_rank());   // 0 = leader of the pair
    const int pair = blockIdx.x >> 1;
    const int num_pairs = gridDim.x >> 1;

    // ---- set-up ---------------------------------------------------------------------------------------
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full + 8 * s, 1);      // leader: one arrive.expect_tx covering both CTAs' bytes
            mbar_init(bar_empty + 8 * s, 1);     // one commit per use, delivered to both CTAs
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar_tmem_full + 8 * s, 1);
            mbar_init(bar_tmem_empty + 8 * s, 16);   // leader: eight epilogue warps of each CTA
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&m0.w); tma_prefetch_desc(&m0.full); tma_prefetch_desc(&m0.part);
        if (p.k_sets > 1 || EPI == EPI_GATE_UP) tma_prefetch_desc(&m1.w);
        if (p.k_sets > 1) { tma_prefetch_desc(&m1.full); tma_prefetch_desc(&m1.part); }
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_ptr_slot)), TMEM_COLS);
        tmem_relinquish_pair();
    }
    if (warp == 2) expert_row_prefix(p, cum, lane);   // cum[0..E]: first schedule row of every expert
    if (warp == 3)
        for (int e = lane; e < p.num_experts; e += 32) occupied[e] = p.occupied_rows[e];
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();     // both CTAs' barriers exist before either one signals the other
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr_slot;

    const int lo = p.row_begin;
    const int hi = min(p.row_end, *p.num_tokens);
    const int num_tiles = total_tiles<MODE_ROWS>(p, lo, hi);

    if (warp == 0) {
        // ---- TMA producer (both CTAs) -----------------------------------------------------------------
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = pair; t < num_tiles && ok; t += num_pairs) {
            Tile tile;
            decode_tile<MODE_ROWS, BK>(p, cum, lo, hi, t, tile);
            const int n = tile_tokens(cum, occupied, tile);
            if (n == 0) continue;
            const int row = tile.row0 - p.row_begin + cta_rank * (n / 2);
            for (int kb = 0; kb < tile.k_blocks; ++kb) {
                ok = mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_flag, p.status);
                if (!ok) break;
                if (lane == 0) {
                    const uint32_t full_local = bar_full + 8 * stage;
                    const uint32_t full = full_local & kPairLeaderMask;   // the leader's barrier collects all bytes
                    const uint32_t w_dst = smem_base + stage * STAGE_BYTES;
                    const uint32_t t_dst = w_dst + W_TILE_BYTES;
                    if (cta_rank == 0) mbar_expect_tx(full_local, 2 * W_TILE_BYTES + n * BK * 2);
                    const int kset = kb >= p.k_blocks ? 1 : 0;
                    const int kk = (kb - kset * p.k_blocks) * BK;
                    const RoutedMaps& maps = kset ? m1 : m0;
                    if (EPI == EPI_GATE_UP) {   // 64 gate and the same 64 up features per CTA
                        const int f = tile.n0 / 2 + cta_rank * kHalf;
                        tma_load_4d_pair(w_dst, &m0.w, full, kk, f, tile.expert, 0);
                        tma_load_4d_pair(w_dst + kHalf * BK * 2, &m1.w, full, kk, f, tile.expert, 0);
                    } else if (W_MN) {
#pragma unroll
                        for (int c = 0; c < BM_CTA / 64; ++c)
                            tma_load_4d_pair(w_dst + c * CHUNK_BYTES, &maps.w, full, tile.n0 + cta_rank * BM_CTA + c * 64, kk, tile.expert, 0);
                    } else {
                        tma_load_4d_pair(w_dst, &maps.w, full, kk, tile.n0 + cta_rank * BM_CTA, tile.expert, 0);
                    }
                    if (n == BN) {
                        tma_load_4d_pair(t_dst, &maps.full, full, kk, row, 0, 0);
                    } else {
                        for (int i = 0; i < n / 2; i += kTokenBox) tma_load_4d_pair(t_dst + i * BK * 2, &maps.part, full, kk, row + i, 0, 0);
                    }
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer (leader CTA only) ----------------------------------------------------------------
        if (cta_rank == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int iter = 0;
            bool ok = true;
            constexpr uint32_t kWStep = W_MN ? 128u : 2u;   // descriptor steps per 16-wide K slice, as in grouped_gemm.cu
            for (int t = pair; t < num_tiles && ok; t += num_pairs) {
                Tile tile;
                decode_tile<MODE_ROWS, BK>(p, cum, lo, hi, t, tile);
                const int n = tile_tokens(cum, occupied, tile);
                if (n == 0) continue;
                const uint32_t idesc = umma_idesc_bf16(BM, n, W_MN, false);
                const int acc = iter & 1;
                const uint32_t acc_phase = (iter >> 1) & 1u;
                ok = mbar_wait(bar_tmem_empty + 8 * acc, acc_phase ^ 1u, abort_flag, p.status);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * BN;
                for (int kb = 0; kb < tile.k_blocks; ++kb) {
                    ok = mbar_wait(bar_full + 8 * stage, phase, abort_flag, p.status);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (lane == 0) {
                        const uint32_t w_addr = smem_base + stage * STAGE_BYTES;
                        const uint64_t w_desc = W_MN ? umma_smem_desc(w_addr, CHUNK_BYTES, 1024) : umma_smem_desc(w_addr, 16, 1024);
                        const uint64_t t_desc = umma_smem_desc(w_addr + W_TILE_BYTES, 16, 1024);
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            umma_bf16_pair(d_tmem, w_desc + k * kWStep, t_desc + k * 2u, idesc, (kb | k) != 0 ? 1u : 0u);
                        umma_commit_pair(bar_empty + 8 * stage);                            // frees the stage in both CTAs
                        if (kb == tile.k_blocks - 1) umma_commit_pair(bar_tmem_full + 8 * acc);   // accumulators complete
                    }
                    __syncwarp();
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
                ++iter;
            }
        }
    } else {
        // ---- epilogue (both CTAs, each for its own 128 features) -------------------------------------------
        const int quarter = warp & 3;                 // tensor-memory lanes [32*quarter, 32*quarter + 32)
        const int group = (warp - 2) >> 2;
        uint8_t* block = smem_gen + SharedLayout::kEpilogue + group * kBlockBytes;
        // reading back: 8 features of a row; store and SwiGLU backward 16 lanes a row, gate / up 8 lanes a row of each half
        constexpr int kVecs = EPI == EPI_GATE_UP ? 8 : 16;
        constexpr int kRowsPerWarp = 32 / kVecs;      // rows of one instruction
        constexpr int kTurns = 8 / kRowsPerWarp;      // a warp takes 8 of the 32 rows
        const int seg = lane % kVecs;
        const int sub = quarter * kRowsPerWarp + lane / kVecs;   // row of turn 0; later turns 4 * kRowsPerWarp further on
        int iter = 0;
        bool ok = true;
        for (int t = pair; t < num_tiles && ok; t += num_pairs) {
            Tile tile;
            decode_tile<MODE_ROWS, BK>(p, cum, lo, hi, t, tile);
            const int n = tile_tokens(cum, occupied, tile);
            const int row0 = tile.row0 - p.row_begin;
            const bool scattered = EPI == EPI_STORE && p.scatter.peer_rank != nullptr;
            const int f0 = EPI == EPI_GATE_UP ? tile.n0 / 2 + cta_rank * kHalf : tile.n0 + cta_rank * BM_CTA;   // first feature of the CTA
            const long long first = static_cast<long long>(row0) * p.ldd + f0 + seg * 8;
            if (n > 0) {
                const int acc = iter & 1;
                const uint32_t acc_phase = (iter >> 1) & 1u;
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN;
                bf16* slot = nullptr;                 // lane kRowsPerWarp * i + j: slot of the row that turn i stores in lanes j * kVecs ...
                uint4 gate[kTurns], up[kTurns];
                auto find_slot = [&](int c) {
                    const int r = c + (lane % 8) / kRowsPerWarp * (4 * kRowsPerWarp) + quarter * kRowsPerWarp + lane % kRowsPerWarp;
                    // CTA 0 of the first column tile delivers the row scalars and reports bad entries
                    slot = scatter_slot(p.scatter, tile.row0 + r, p.row_begin, p.ldd, tile.n0 == 0 && cta_rank == 0 && lane < 8, p.status);
                };
                if (scattered) find_slot(group * 32);   // while the tile is still being accumulated
                if (EPI == EPI_SWIGLU_BWD) {
#pragma unroll
                    for (int i = 0; i < kTurns; ++i) {
                        const long long off = first + static_cast<long long>(group * 32 + i * 4 * kRowsPerWarp + sub) * p.ldd;
                        gate[i] = __ldg(reinterpret_cast<const uint4*>(p.gate + off));
                        up[i] = __ldg(reinterpret_cast<const uint4*>(p.up + off));
                    }
                }
                ok = group_sync(group, mbar_wait(bar_tmem_full + 8 * acc, acc_phase, abort_flag, p.status));
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll 1
                for (int c = group * 32; c < n; c += 64) {   // n is a multiple of 64: both groups have the same number of blocks
                    const bool more = c + 64 < n;
                    const unsigned long long slots = reinterpret_cast<unsigned long long>(slot);
                    if (scattered && more) find_slot(c + 64);   // used a whole turn later
                    {
                        uint32_t v[32];
                        tmem_ld_32x32(taddr + c, v);
                        tmem_ld_wait();
                        if (!more) {                  // everything is in registers: the next tile but one may accumulate here
                            tc_fence_before_sync();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_leader(bar_tmem_empty + 8 * acc);
                        }
                        uint8_t* mine = block + (quarter * 32 + lane) * 2;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            *reinterpret_cast<bf16*>(mine + i * kRowPitchBytes) = __float2bfloat16_rn(__uint_as_float(v[i]));
                    }
                    group_sync(group);
#pragma unroll
                    for (int i = 0; i < kTurns; ++i) {
                        const int r = i * 4 * kRowsPerWarp + sub;
                        const long long off = first + static_cast<long long>(c + r) * p.ldd;
                        const uint4 w = *reinterpret_cast<const uint4*>(block + r * kRowPitchBytes + seg * 16);
                        if (EPI == EPI_GATE_UP) {     // a row: 64 gate features, then the same 64 up features
                            const uint4 u = *reinterpret_cast<const uint4*>(block + r * kRowPitchBytes + 2 * kHalf + seg * 16);
                            const uint4 h = p.clamp ? swiglu_vec<true>(w, u, p.limit) : swiglu_vec<false>(w, u, 0.f);
                            *reinterpret_cast<uint4*>(p.D0 + off) = w;
                            *reinterpret_cast<uint4*>(p.D1 + off) = u;
                            *reinterpret_cast<uint4*>(p.D2 + off) = h;
                        } else if (EPI == EPI_SWIGLU_BWD) {
                            const uint4 g = gate[i], u = up[i];
                            if (more) {
                                gate[i] = __ldg(reinterpret_cast<const uint4*>(p.gate + off + 64 * p.ldd));
                                up[i] = __ldg(reinterpret_cast<const uint4*>(p.up + off + 64 * p.ldd));
                            }
                            uint4 dg, du;
                            float sum = p.clamp ? swiglu_bwd_vec<true>(g, u, w, p.limit, dg, du) : swiglu_bwd_vec<false>(g, u, w, 0.f, dg, du);
                            *reinterpret_cast<uint4*>(p.D0 + off) = w;
                            *reinterpret_cast<uint4*>(p.D1 + off) = dg;
                            *reinterpret_cast<uint4*>(p.D2 + off) = du;
#pragma unroll
                            for (int s = 1; s < kVecs; s <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
                            if (seg == 0 && p.row_partial != nullptr)
                                p.row_partial[static_cast<long long>(row0 + c + r) * (p.n_blocks * (BM / BM_CTA)) + f0 / BM_CTA] = sum;
                        } else if (scattered) {
                            bf16* dst = reinterpret_cast<bf16*>(__shfl_sync(0xffffffffu, slots, i * kRowsPerWarp + lane / kVecs));
                            if (dst != nullptr) *reinterpret_cast<uint4*>(dst + f0 + seg * 8) = w;
                        } else {
                            *reinterpret_cast<uint4*>(p.D0 + off) = w;
                        }
                    }
                    group_sync(group);                // the block may be overwritten
                }
                ++iter;
            }
            // the padding rows behind: zeros, which is what zero inputs accumulate to
            if (!scattered) {
                const uint4 zero = make_uint4(0, 0, 0, 0);
                for (int r = n + group * 4 * kRowsPerWarp + sub; r < BN; r += 8 * kRowsPerWarp) {
                    const long long off = first + static_cast<long long>(r) * p.ldd;
                    *reinterpret_cast<uint4*>(p.D0 + off) = zero;
                    if (EPI != EPI_STORE) {
                        *reinterpret_cast<uint4*>(p.D1 + off) = zero;
                        *reinterpret_cast<uint4*>(p.D2 + off) = zero;
                    }
                    if (EPI == EPI_SWIGLU_BWD && p.row_partial != nullptr && seg == 0)
                        p.row_partial[static_cast<long long>(row0 + r) * (p.n_blocks * (BM / BM_CTA)) + f0 / BM_CTA] = 0.0f;
                }
            }
        }
    }

    // ---- teardown -------------------------------------------------------------------------------------
    if (*abort_flag) {   // give copies that are still in flight time to land before shared memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();   // the peer's shared memory and barriers stay valid until both CTAs are done
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

template <bool W_MN, int EPI>
int launch(const RoutedMaps& m0, const RoutedMaps& m1, const KernelParams& kp, int max_tiles, cudaStream_t stream) {
    static int resident_pairs[16] = {0};
    const size_t smem = 1024 + SharedLayout::kCum + 4 * (2 * static_cast<size_t>(kp.num_experts) + 2);
    return launch_pairs<kThreads>(routed_gemm_kernel<W_MN, EPI>, "routed_gemm_kernel", resident_pairs, smem, max_tiles, stream, m0, m1, kp);
}

int fill_maps(RoutedMaps* m, const GemmProblem& pb, const void* A, const void* W, int N, int K, bool kn, int weight_rows) {
    MOK_TRY(make_map(&m->full, A, K, pb.buffer_rows, 1, BK, BN_CTA));
    MOK_TRY(make_map(&m->part, A, K, pb.buffer_rows, 1, BK, kTokenBox));
    return kn ? make_map(&m->w, W, N, K, pb.num_experts, 64, BK) : make_map(&m->w, W, K, N, pb.num_experts, BK, weight_rows);
}

KernelParams rows_params(const GemmProblem& pb, int N, int K, int k_sets) {
    KernelParams kp = base_params(pb);
    kp.n_blocks = N / BM;
    kp.k_blocks = K / BK;
    kp.k_sets = k_sets;
    kp.ldd = N;
    kp.m_group = rows_group(2LL * k_sets * N * K);
    return kp;
}

int tiles_of(const GemmProblem& pb, const KernelParams& kp) { return ((pb.row_end - pb.row_begin) / BN) * kp.n_blocks; }

}  // namespace

int launch_routed_gemm(const GemmProblem& pb, const void* A0, const void* A1, int K, const void* B0, const void* B1, void* D, int N,
                       bool b_is_kn, cudaStream_t stream, const RowScatter* scatter) {
    RoutedMaps m0, m1;
    MOK_TRY(fill_maps(&m0, pb, A0, B0, N, K, b_is_kn, BM_CTA));
    MOK_TRY(fill_maps(&m1, pb, A1 ? A1 : A0, B1 ? B1 : B0, N, K, b_is_kn, BM_CTA));
    KernelParams kp = rows_params(pb, N, K, A1 ? 2 : 1);
    MOK_TRY(set_output(kp, D, scatter));
    return b_is_kn ? launch<true, EPI_STORE>(m0, m1, kp, tiles_of(pb, kp), stream)
                   : launch<false, EPI_STORE>(m0, m1, kp, tiles_of(pb, kp), stream);
}

int launch_routed_gate_up(const GemmProblem& pb, const void* A, int K, const void* Wg, const void* Wu, void* gate, void* up, void* hidden,
                          int N, bool has_limit, float limit, cudaStream_t stream) {
    RoutedMaps m0, m1;
    MOK_TRY(fill_maps(&m0, pb, A, Wg, N, K, false, kHalf));
    MOK_TRY(fill_maps(&m1, pb, A, Wu, N, K, false, kHalf));
    KernelParams kp = rows_params(pb, 2 * N, K, 1);   // one tile per 128 gate and the same 128 up features
    kp.ldd = N;
    kp.D0 = static_cast<bf16*>(gate);
    kp.D1 = static_cast<bf16*>(up);
    kp.D2 = static_cast<bf16*>(hidden);
    kp.clamp = has_limit ? 1 : 0;
    kp.limit = limit;
    return launch<false, EPI_GATE_UP>(m0, m1, kp, tiles_of(pb, kp), stream);
}

int launch_routed_down_dgrad(const GemmProblem& pb, const void* A, int K, const void* B, const void* gate, const void* up, void* d_hidden,
                             void* d_gate, void* d_up, float* row_partial, int N, bool has_limit, float limit, cudaStream_t stream) {
    RoutedMaps m0;
    MOK_TRY(fill_maps(&m0, pb, A, B, N, K, true, BM_CTA));
    KernelParams kp = rows_params(pb, N, K, 1);
    kp.D0 = static_cast<bf16*>(d_hidden);
    kp.D1 = static_cast<bf16*>(d_gate);
    kp.D2 = static_cast<bf16*>(d_up);
    kp.gate = static_cast<const bf16*>(gate);
    kp.up = static_cast<const bf16*>(up);
    kp.row_partial = row_partial;
    kp.clamp = has_limit ? 1 : 0;
    kp.limit = limit;
    return launch<true, EPI_SWIGLU_BWD>(m0, m0, kp, tiles_of(pb, kp), stream);
}

}  // namespace mok
