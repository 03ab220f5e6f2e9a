// MXFP8 quantizer: bf16 -> e4m3 elements with one e8m0 scale per 32 elements along the row, for a matrix and /
// or its transpose.  HBM-bound: every 128 x 128 tile is staged in shared memory once and both layouts are
// produced from it (2 B read, up to 2 x 1.03 B written per element).
//
// Arithmetic (bit-exact with the reference device code, csrc/mxfp8.cuh:45-72): scale = max(amax * fp32(1/448),
// 1e-12) rounded UP to a power of two (cvt.rp.satfinite.ue8m0x2), elements multiplied by the exact reciprocal
// 2^(127-e) and converted with cvt.rn.satfinite.e4m3x2.  Scale bytes are stored in the tensor-core scale-factor
// layout: tile [rows/128][cols/128] of 512 bytes, byte (r % 32) * 16 + (r / 32) * 4 + kblock (csrc/mxfp8.cuh:181-184).
//
// The same kernel serves the stand-alone op (whole matrices) and the fused layer (a window of schedule rows of an
// activation buffer, limited on the device by the padded token count; the transposed output then is a column range
// of a wider [cols, buffer_rows] matrix).
#include "mxfp8.cuh"
#include "swiglu_math.cuh"

namespace mok {
namespace {

constexpr int kTile = 128;
constexpr int kRowPitch = kTile * 2 + 16;   // bytes; the 16-byte pad keeps row-wise 16 B reads conflict free
constexpr int kOutPitch = kTile + 16;       // bytes per staged e4m3 output row; staged over the bf16 tile it came from
constexpr int kTileBytes = kTile * kRowPitch;

// 128 rows x 128 bytes from the staging tile to global memory, eight lanes per row: every store instruction of a
// warp writes four complete 128-byte lines (a thread writing its own row would touch 32 lines with 16 bytes each).
template <int THREADS>
__device__ __forceinline__ void store_staged_rows(const uint8_t* otile, uint8_t* out, long long ld, int tid) {
#pragma unroll
    for (int i = tid; i < kTile * 8; i += THREADS) {
        const int r = i >> 3, seg = i & 7;
        *reinterpret_cast<uint4*>(out + static_cast<long long>(r) * ld + seg * 16) =
            *reinterpret_cast<const uint4*>(otile + r * kOutPitch + seg * 16);
    }
}

// One 512-byte scale tile from shared memory: single scale bytes stored to global memory would be a quarter of all store
// requests of a tile.
constexpr int kScaleTile = 512;
__device__ __forceinline__ void store_scale_tile(const uint8_t* staged, uint8_t* out, int tid) {
    if (tid < kScaleTile / 16) reinterpret_cast<uint4*>(out)[tid] = reinterpret_cast<const uint4*>(staged)[tid];
}

// Transposed layout of a staged bf16 tile: column of the tile = row of the transpose, four blocks of 32 down the column.
// `out` is the transposed tile's first byte (rows `ld` apart), `scale_tile` its 512-byte scale tile.  THREADS threads (128 or
// 256) with tid 0.. take one tile; every thread of the block calls, and the tile must be complete (a barrier before the call
// is the caller's).  A thread takes two adjacent columns (one 32-bit shared-memory word per row, conflict free across the
// warp) and one or two of the four row blocks.  The e4m3 rows and the scale bytes are staged over the tile itself, which
// nobody reads any more by then, and leave as full lines.
template <int THREADS>
__device__ __forceinline__ void quantize_tile_transposed(uint8_t* tile, int tid, uint8_t* out, long long ld, uint8_t* scale_tile) {
    constexpr int kBlocks = 256 / THREADS;
    const int pair = tid & 63, first = (tid >> 6) * kBlocks;
    const int col_a = 2 * pair, col_b = col_a + 1;
    uint32_t sa[kBlocks], sb[kBlocks];
    uint32_t qa[kBlocks][8], qb[kBlocks][8];
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) {
        const uint8_t* column = tile + (first + k) * 32 * kRowPitch + pair * 4;
        uint32_t w[32], m = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) w[i] = *reinterpret_cast<const uint32_t*>(column + i * kRowPitch);
#pragma unroll
        for (int i = 0; i < 32; ++i) m = bf16x2_absmax(m, w[i]);
        const float2 amax = unpack_bf16x2(m);
        sa[k] = mxfp8_scale_byte(amax.x);
        sb[k] = mxfp8_scale_byte(amax.y);
        const float inv_a = mxfp8_inverse_scale(sa[k]), inv_b = mxfp8_inverse_scale(sb[k]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 v0 = unpack_bf16x2(w[4 * i]), v1 = unpack_bf16x2(w[4 * i + 1]), v2 = unpack_bf16x2(w[4 * i + 2]),
                         v3 = unpack_bf16x2(w[4 * i + 3]);
            qa[k][i] = mxfp8_convert4(v0.x * inv_a, v1.x * inv_a, v2.x * inv_a, v3.x * inv_a);
            qb[k][i] = mxfp8_convert4(v0.y * inv_b, v1.y * inv_b, v2.y * inv_b, v3.y * inv_b);
        }
    }
    __syncthreads();
    uint8_t* staged_scales = tile + kTile * kOutPitch;
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) {
        uint4* dst_a = reinterpret_cast<uint4*>(tile + col_a * kOutPitch + (first + k) * 32);
        uint4* dst_b = reinterpret_cast<uint4*>(tile + col_b * kOutPitch + (first + k) * 32);
        dst_a[0] = make_uint4(qa[k][0], qa[k][1], qa[k][2], qa[k][3]);
        dst_a[1] = make_uint4(qa[k][4], qa[k][5], qa[k][6], qa[k][7]);
        dst_b[0] = make_uint4(qb[k][0], qb[k][1], qb[k][2], qb[k][3]);
        dst_b[1] = make_uint4(qb[k][4], qb[k][5], qb[k][6], qb[k][7]);
        staged_scales[(col_a & 31) * 16 + (col_a >> 5) * 4 + first + k] = static_cast<uint8_t>(sa[k]);
        staged_scales[(col_b & 31) * 16 + (col_b >> 5) * 4 + first + k] = static_cast<uint8_t>(sb[k]);
    }
    __syncthreads();
    store_staged_rows<THREADS>(tile, out, ld, tid);
    store_scale_tile(staged_scales, scale_tile, tid);
}

struct QuantArgs {
    const bf16* x;             // row 0 of the span / matrix 0
    long long x_ld;            // elements between rows
    long long x_mat_stride;    // elements between matrices (blockIdx.z)
    uint8_t* q;                // normal output, same shape as x
    long long q_mat_stride;
    uint8_t* sc;               // scale tile (row tile 0, col tile 0)
    long long sc_row_tile_stride, sc_mat_stride;   // bytes
    uint8_t* qt;               // transposed output: element (c, r) at qt[c * qt_ld + r]
    long long qt_ld, qt_mat_stride;
    uint8_t* sct;              // scale tile (col tile 0, row tile 0) of the transposed output
    long long sct_row_tile_stride, sct_mat_stride;
    const int* num_tokens;     // optional device row limit (schedule rows)
    int row_begin, row_end;    // schedule rows covered by the span (row_end also bounds a dense matrix)
};

__device__ __forceinline__ void copy_async_16(void* dst, const void* src, bool valid) {   // zeros when not valid
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Bound by HBM.  A block walks `tiles_per_block` column tiles of one row tile; the next tile is on its way into the second
// buffer while one is being quantized.  One tile per block and plain loads left the block waiting for its own loads two
// thirds of the time, whatever the order of the tiles: 37k gathered rows of 7168 359 us (242 us with the leaner arithmetic
// and 6 instead of 4 resident blocks), now 197 us (5.5 TB/s); weights 32 x 2048 x 7168 in both layouts 395 -> 340 us.
// 16 lanes per row and eight consecutive columns per lane, eight rows per thread: a block of 32 along the row is four adjacent
// lanes, so the normal layout is quantized from registers (mxfp8_quantize_quarter) and stored as full 128-byte lines.
// GATHER: the tile's rows are schedule rows whose tokens are read where they lie (`x` = all tokens of this rank), and
// with weights scaled on the way, instead of from a buffer that a dispatch pass has filled.
constexpr int kQuantThreads = 256;
constexpr int kQuantBlocksPerSm = 3;
template <bool GATHER>
__global__ void __launch_bounds__(kQuantThreads, kQuantBlocksPerSm) quantize_kernel(const QuantArgs a, const LocalRows g, int tiles_per_block) {
    extern __shared__ __align__(16) uint8_t quant_tiles[];       // two bf16 input tiles, padded rows
    __shared__ __align__(16) uint8_t row_scales[kScaleTile];
    __shared__ int tokens[GATHER ? kTile : 1];
    __shared__ float scales[GATHER ? kTile : 1];
    const int tid = threadIdx.x, v = tid & 15, rq = tid >> 4;
    const int tc0 = blockIdx.x * tiles_per_block, tr = blockIdx.y, e = blockIdx.z;
    if (GATHER && tc0 == 0 && tr == 0 && tid == 0 && *a.num_tokens > g.rows.covered_rows && g.rows.status != nullptr)
        atomicOr(g.rows.status, (uint32_t)MOK_STATUS_BAD_SCHEDULE_ENTRY);
    const int limit = a.num_tokens != nullptr ? min(a.row_end, *a.num_tokens) : a.row_end;
    if (a.row_begin + tr * kTile >= limit) return;

    const bf16* src = a.x + static_cast<long long>(tc0) * kTile + v * 8;
    if (GATHER) {
        if (tid < kTile) {
            const int row = a.row_begin + tr * kTile + tid;
            const int peer = g.rows.peer_rank[row], route = g.rows.peer_token[row];
            const bool valid = peer == 0 && route >= 0 && route < g.num_routes;
            if (peer >= 0 && !valid && tc0 == 0 && g.rows.status != nullptr)
                atomicOr(g.rows.status, (uint32_t)MOK_STATUS_BAD_SCHEDULE_ENTRY);
            const float w = valid && g.weights != nullptr ? g.weights[route] : 0.0f;
            tokens[tid] = valid ? route / g.topk : -1;
            scales[tid] = w;
            if (tc0 == 0 && g.weights != nullptr) g.row_weight[tr * kTile + tid] = w;
        }
        __syncthreads();
    } else {
        src += e * a.x_mat_stride + static_cast<long long>(tr) * kTile * a.x_ld;
    }
    const int tiles = min(tiles_per_block, static_cast<int>(a.x_ld / kTile) - tc0);
    auto fetch = [&](int t) {
        uint8_t* dst = quant_tiles + (t & 1) * kTileBytes + v * 16;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = rq + 16 * j;
            const int token = GATHER ? tokens[r] : r;            // padding row: zeros, as a dispatch writes them
            copy_async_16(dst + r * kRowPitch, src + t * kTile + max(token, 0) * a.x_ld, token >= 0);
        }
        copy_async_commit();
    };
    fetch(0);
    for (int t = 0; t < tiles; ++t) {
        if (t + 1 < tiles) {
            fetch(t + 1);
            copy_async_wait<1>();
        } else {
            copy_async_wait<0>();
        }
        const int tc = tc0 + t;
        uint8_t* tile = quant_tiles + (t & 1) * kTileBytes;
        uint8_t* q = a.q + e * a.q_mat_stride + static_cast<long long>(tr) * kTile * a.x_ld + static_cast<long long>(tc) * kTile + v * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) {                            // the rows that this thread has fetched itself
            const int r = rq + 16 * j;
            uint4* mine = reinterpret_cast<uint4*>(tile + r * kRowPitch + v * 16);
            uint4 val = *mine;
            if (GATHER && g.weights != nullptr && tokens[r] >= 0) {
                val = scale_vec(val, scales[r]);
                *mine = val;
            }
            if (a.q != nullptr) {
                uint2 bytes;
                uint32_t sb;
                mxfp8_quantize_quarter(val, bytes, sb);
                *reinterpret_cast<uint2*>(q + r * a.x_ld) = bytes;
                if ((v & 3) == 0) row_scales[(r & 31) * 16 + (r >> 5) * 4 + (v >> 2)] = static_cast<uint8_t>(sb);
            }
        }
        __syncthreads();
        if (a.q != nullptr)
            store_scale_tile(row_scales, a.sc + e * a.sc_mat_stride + tr * a.sc_row_tile_stride + static_cast<long long>(tc) * kScaleTile, tid);
        if (a.qt != nullptr)
            quantize_tile_transposed<kQuantThreads>(
                tile, tid,
                a.qt + e * a.qt_mat_stride + static_cast<long long>(tc) * kTile * a.qt_ld + static_cast<long long>(tr) * kTile,
                a.qt_ld, a.sct + e * a.sct_mat_stride + tc * a.sct_row_tile_stride + static_cast<long long>(tr) * kScaleTile);
        if (t + 1 < tiles) __syncthreads();                      // the tile and the scale bytes may be overwritten
    }
}

// ---- fused activation steps ---------------------------------------------------------------------------------------
// Both kernels walk a 128 x 128 tile with 16 lanes per row and eight consecutive columns per lane, sixteen rows per
// thread in the forward (128 threads) and eight in the backward (256): a block of 32 along the row is four adjacent lanes, so
// the normal layout is quantized straight from registers (mxfp8_quantize_quarter) and stored as full 128-byte lines; the values
// that also need the transposed layout go through a shared-memory tile.
struct FusedFwdArgs {
    const bf16 *gate, *up;
    uint8_t *gate_q, *gate_sc, *up_q, *up_sc, *hidden_q, *hidden_sc, *hidden_qt, *hidden_sct;
    long long sc_row_tile_stride, qt_ld, sct_row_tile_stride;
    const int* num_tokens;
    int row_begin, row_end, cols;
    float limit;
};

template <bool CLAMP>
__global__ void __launch_bounds__(128) swiglu_quantize_fwd_kernel(const FusedFwdArgs a) {
    __shared__ __align__(16) uint8_t tile[kTileBytes];
    const int tid = threadIdx.x, v = tid & 15, rq = tid >> 4;
    const int tc = blockIdx.x, tr = blockIdx.y;
    const int limit_row = min(a.row_end, *a.num_tokens);
    if (a.row_begin + tr * kTile >= limit_row) return;
    const long long sc_off = tr * a.sc_row_tile_stride + static_cast<long long>(tc) * 512;
#pragma unroll 4
    for (int j = 0; j < 16; ++j) {
        const int r = rq + 8 * j;
        const long long off = (static_cast<long long>(tr) * kTile + r) * a.cols + tc * kTile + v * 8;
        const uint4 g = *reinterpret_cast<const uint4*>(a.gate + off);
        const uint4 u = *reinterpret_cast<const uint4*>(a.up + off);
        uint4 h;
        h.x = swiglu_pair<CLAMP>(g.x, u.x, a.limit);
        h.y = swiglu_pair<CLAMP>(g.y, u.y, a.limit);
        h.z = swiglu_pair<CLAMP>(g.z, u.z, a.limit);
        h.w = swiglu_pair<CLAMP>(g.w, u.w, a.limit);
        const int sidx = (r & 31) * 16 + (r >> 5) * 4 + (v >> 2);
        uint2 q;
        uint32_t sb;
        mxfp8_quantize_quarter(g, q, sb);
        *reinterpret_cast<uint2*>(a.gate_q + off) = q;
        if ((v & 3) == 0) a.gate_sc[sc_off + sidx] = static_cast<uint8_t>(sb);
        mxfp8_quantize_quarter(u, q, sb);
        *reinterpret_cast<uint2*>(a.up_q + off) = q;
        if ((v & 3) == 0) a.up_sc[sc_off + sidx] = static_cast<uint8_t>(sb);
        mxfp8_quantize_quarter(h, q, sb);
        *reinterpret_cast<uint2*>(a.hidden_q + off) = q;
        if ((v & 3) == 0) a.hidden_sc[sc_off + sidx] = static_cast<uint8_t>(sb);
        *reinterpret_cast<uint4*>(tile + r * kRowPitch + v * 16) = h;
    }
    __syncthreads();
    quantize_tile_transposed<128>(tile, tid, a.hidden_qt + static_cast<long long>(tc) * kTile * a.qt_ld + static_cast<long long>(tr) * kTile,
                             a.qt_ld, a.hidden_sct + tc * a.sct_row_tile_stride + static_cast<long long>(tr) * 512);
}

struct FusedBwdArgs {
    const uint8_t *gate_q, *gate_sc, *up_q, *up_sc;
    const bf16* d_hidden;
    uint8_t *dg_q, *dg_sc, *du_q, *du_sc, *dg_qt, *dg_sct, *du_qt, *du_sct;
    long long sc_row_tile_stride, qt_ld, sct_row_tile_stride;
    float* row_partial;
    const int* num_tokens;
    int row_begin, row_end, cols;
    float limit;
};

// 256 threads, 8 rows each; d_gate and d_up have a tile of their own, and half of the block transposes each.  135k rows of
// 2048: 997 us with one tile (d_up waited in 64 registers, 16 warps per SM, loads in the order of use), 720 us like this.
template <bool CLAMP>
__global__ void __launch_bounds__(256, 3) swiglu_quantize_bwd_kernel(const FusedBwdArgs a) {
    extern __shared__ __align__(16) uint8_t bwd_tiles[];
    __shared__ __align__(16) uint8_t row_scales[2][kScaleTile];
    const int tid = threadIdx.x, v = tid & 15, rq = tid >> 4;
    const int tc = blockIdx.x, tr = blockIdx.y;
    const int limit_row = min(a.row_end, *a.num_tokens);
    if (a.row_begin + tr * kTile >= limit_row) return;
    const long long sc_off = tr * a.sc_row_tile_stride + static_cast<long long>(tc) * 512;
    const int tiles = a.cols / kTile;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        uint2 gq[4], uq[4];   // four rows in flight before the first of them is used
        uint4 dh[4];
        uint32_t gs[4], us[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = rq + 16 * (4 * part + j);
            const long long off = (static_cast<long long>(tr) * kTile + r) * a.cols + tc * kTile + v * 8;
            const int sidx = (r & 31) * 16 + (r >> 5) * 4 + (v >> 2);
            gq[j] = __ldg(reinterpret_cast<const uint2*>(a.gate_q + off));
            uq[j] = __ldg(reinterpret_cast<const uint2*>(a.up_q + off));
            dh[j] = __ldg(reinterpret_cast<const uint4*>(a.d_hidden + off));
            gs[j] = __ldg(a.gate_sc + sc_off + sidx);
            us[j] = __ldg(a.up_sc + sc_off + sidx);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = rq + 16 * (4 * part + j);
            const long long row = static_cast<long long>(tr) * kTile + r;
            const long long off = row * a.cols + tc * kTile + v * 8;
            const int sidx = (r & 31) * 16 + (r >> 5) * 4 + (v >> 2);
            const uint4 g = mxfp8_dequantize8(gq[j], gs[j]);
            const uint4 u = mxfp8_dequantize8(uq[j], us[j]);
            uint4 dg, du;
            float acc = swiglu_bwd_pair<CLAMP>(g.x, u.x, dh[j].x, a.limit, dg.x, du.x);
            acc += swiglu_bwd_pair<CLAMP>(g.y, u.y, dh[j].y, a.limit, dg.y, du.y);
            acc += swiglu_bwd_pair<CLAMP>(g.z, u.z, dh[j].z, a.limit, dg.z, du.z);
            acc += swiglu_bwd_pair<CLAMP>(g.w, u.w, dh[j].w, a.limit, dg.w, du.w);
#pragma unroll
            for (int off_l = 1; off_l < 16; off_l <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off_l);   // the row's 16 lanes
            if (v == 0) a.row_partial[row * tiles + tc] = acc;
            uint2 q;
            uint32_t sb;
            mxfp8_quantize_quarter(dg, q, sb);
            *reinterpret_cast<uint2*>(a.dg_q + off) = q;
            if ((v & 3) == 0) row_scales[0][sidx] = static_cast<uint8_t>(sb);
            mxfp8_quantize_quarter(du, q, sb);
            *reinterpret_cast<uint2*>(a.du_q + off) = q;
            if ((v & 3) == 0) row_scales[1][sidx] = static_cast<uint8_t>(sb);
            *reinterpret_cast<uint4*>(bwd_tiles + r * kRowPitch + v * 16) = dg;
            *reinterpret_cast<uint4*>(bwd_tiles + kTileBytes + r * kRowPitch + v * 16) = du;
        }
    }
    __syncthreads();
    const long long t_off = static_cast<long long>(tc) * kTile * a.qt_ld + static_cast<long long>(tr) * kTile;
    const long long ts_off = tc * a.sct_row_tile_stride + static_cast<long long>(tr) * 512;
    const bool up = tid >= 128;
    store_scale_tile(row_scales[up], (up ? a.du_sc : a.dg_sc) + sc_off, tid & 127);
    quantize_tile_transposed<128>(bwd_tiles + (up ? kTileBytes : 0), tid & 127, (up ? a.du_qt : a.dg_qt) + t_off, a.qt_ld,
                             (up ? a.du_sct : a.dg_sct) + ts_off);
}

__global__ void __launch_bounds__(256) router_grad_kernel(const float* __restrict__ row_partial, int tiles,
                                                           const float* __restrict__ row_weight, float* __restrict__ row_grad,
                                                           const int* __restrict__ num_tokens, int row_begin, int row_end) {
    const int rows = min(row_end, *num_tokens) - row_begin;
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
        float acc = 0.0f;
        for (int t = 0; t < tiles; ++t) acc += row_partial[static_cast<long long>(row) * tiles + t];
        const float w = row_weight[row];
        row_grad[row] = w > 0.0f ? acc / w : 0.0f;
    }
}

// bf16[r, c] = e4m3[r, c] * 2^(scale(r, c / 32) - 127); exact (3 mantissa bits fit bf16).  One thread per 16 elements.
__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ sc,
                                                          long long sc_row_tile_stride, bf16* __restrict__ out, int cols,
                                                          const int* __restrict__ num_tokens, int row_begin, int row_end) {
    const int limit = num_tokens != nullptr ? min(row_end, *num_tokens) : row_end;
    const long long rows = limit - row_begin;
    const int vec_per_row = cols / 16;
    const long long n = rows * vec_per_row;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const long long r = i / vec_per_row;
        const int c = static_cast<int>(i - r * vec_per_row) * 16;
        const uint4 v = *reinterpret_cast<const uint4*>(q + r * cols + c);
        const int rr = static_cast<int>(r & 127);
        const uint8_t sbyte = sc[(r >> 7) * sc_row_tile_stride + static_cast<long long>(c >> 7) * 512 + (rr & 31) * 16 + (rr >> 5) * 4 +
                                 ((c & 127) >> 5)];
        const float scale = __uint_as_float(static_cast<uint32_t>(sbyte) << 23);
        const uint32_t words[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[8];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(words[w] >> (16 * h)), __NV_E4M3);
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
                o[w * 2 + h] = pack_bf16x2(f.x * scale, f.y * scale);
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(out + r * cols + c);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

template <bool GATHER>
int launch_quantize(const QuantArgs& a, const LocalRows& g, const dim3& tiles, cudaStream_t stream) {
    static bool done[16] = {false};
    int dev = 0;
    MOK_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 16) return MOK_ERR_UNSUPPORTED;
    if (!done[dev]) {
        MOK_CUDA_CHECK(cudaFuncSetAttribute(quantize_kernel<GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kTileBytes));
        done[dev] = true;
    }
    // as many tiles per block as leave every resident block at least two turns, up to 8
    const long long total = static_cast<long long>(tiles.x) * tiles.y * tiles.z;
    long long per_block = total / (2LL * kQuantBlocksPerSm * sm_count());
    per_block = per_block < 1 ? 1 : per_block > 8 ? 8 : per_block;
    const dim3 grid((tiles.x + per_block - 1) / per_block, tiles.y, tiles.z);
    quantize_kernel<GATHER><<<grid, kQuantThreads, 2 * kTileBytes, stream>>>(a, g, static_cast<int>(per_block));
    MOK_LAUNCH_CHECK("mxfp8_quantize_kernel");
    return MOK_OK;
}

}  // namespace

int launch_quantize_rows(const void* x, int cols, const int32_t* num_tokens, int row_begin, int row_end, void* q, void* sc,
                         long long sc_row_tile_stride, void* qt, long long qt_ld, void* sct, long long sct_row_tile_stride,
                         cudaStream_t stream, const LocalRows* gather) {
    if (x == nullptr || cols <= 0 || cols % 128 != 0 || row_end <= row_begin || (row_end - row_begin) % 128 != 0)
        return MOK_ERR_INVALID_ARGUMENT;
    if ((q == nullptr) != (sc == nullptr) || (qt == nullptr) != (sct == nullptr) || (q == nullptr && qt == nullptr))
        return MOK_ERR_INVALID_ARGUMENT;
    if (gather != nullptr && ((reinterpret_cast<uintptr_t>(x) & 15u) != 0 || num_tokens == nullptr || !gather->rows.peer_rank ||
                              !gather->rows.peer_token || gather->topk < 1 || (gather->weights != nullptr && !gather->row_weight)))
        return MOK_ERR_INVALID_ARGUMENT;
    QuantArgs a{};
    a.x = static_cast<const bf16*>(x);
    a.x_ld = cols;
    a.q = static_cast<uint8_t*>(q);
    a.sc = static_cast<uint8_t*>(sc);
    a.sc_row_tile_stride = sc_row_tile_stride;
    a.qt = static_cast<uint8_t*>(qt);
    a.qt_ld = qt_ld;
    a.sct = static_cast<uint8_t*>(sct);
    a.sct_row_tile_stride = sct_row_tile_stride;
    a.num_tokens = num_tokens;
    a.row_begin = row_begin;
    a.row_end = row_end;
    const int row_tiles = (row_end - row_begin) / 128;
    if (row_tiles > 65535) return MOK_ERR_TOO_LARGE;
    dim3 grid(cols / 128, row_tiles, 1);
    return gather != nullptr ? launch_quantize<true>(a, *gather, grid, stream) : launch_quantize<false>(a, LocalRows{}, grid, stream);
}

int launch_dequantize_rows(const void* q, const void* sc, long long sc_row_tile_stride, void* out, int cols,
                           const int32_t* num_tokens, int row_begin, int row_end, cudaStream_t stream) {
    if (q == nullptr || sc == nullptr || out == nullptr || cols <= 0 || cols % 128 != 0 || row_end <= row_begin)
        return MOK_ERR_INVALID_ARGUMENT;
    const long long items = static_cast<long long>(row_end - row_begin) * (cols / 16);
    long long blocks = (items + 255) / 256;
    const long long cap = static_cast<long long>(sm_count()) * 16;
    if (blocks > cap) blocks = cap;
    dequantize_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(static_cast<const uint8_t*>(q), static_cast<const uint8_t*>(sc),
                                                                    sc_row_tile_stride, static_cast<bf16*>(out), cols, num_tokens,
                                                                    row_begin, row_end);
    MOK_LAUNCH_CHECK("mxfp8_dequantize_kernel");
    return MOK_OK;
}

namespace {

// `smem`: dynamic shared memory, whose limit is raised once per device and kernel instantiation.
template <typename Kernel, typename Args>
int launch_tile_kernel(Kernel kernel, const char* name, bool (&done)[16], const Args& args, int cols, int rows, int threads, int smem,
                       cudaStream_t stream) {
    if (rows / 128 > 65535) return MOK_ERR_TOO_LARGE;
    int dev = 0;
    MOK_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 16) return MOK_ERR_UNSUPPORTED;
    if (smem > 0 && !done[dev]) {
        MOK_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        done[dev] = true;
    }
    dim3 grid(cols / 128, rows / 128, 1);
    kernel<<<grid, threads, smem, stream>>>(args);
    MOK_LAUNCH_CHECK(name);
    return MOK_OK;
}

}  // namespace

int launch_swiglu_quantize_fwd(const void* gate, const void* up, int cols, const int32_t* num_tokens, int row_begin, int row_end,
                               void* gate_q, void* gate_sc, void* up_q, void* up_sc, void* hidden_q, void* hidden_sc,
                               long long sc_row_tile_stride, void* hidden_qt, long long qt_ld, void* hidden_sct,
                               long long sct_row_tile_stride, bool has_limit, float limit, cudaStream_t stream) {
    if (!gate || !up || !num_tokens || !gate_q || !gate_sc || !up_q || !up_sc || !hidden_q || !hidden_sc || !hidden_qt || !hidden_sct)
        return MOK_ERR_INVALID_ARGUMENT;
    if (cols <= 0 || cols % 128 != 0 || row_end <= row_begin || (row_end - row_begin) % 128 != 0) return MOK_ERR_INVALID_ARGUMENT;
    FusedFwdArgs a{};
    a.gate = static_cast<const bf16*>(gate);
    a.up = static_cast<const bf16*>(up);
    a.gate_q = static_cast<uint8_t*>(gate_q);
    a.gate_sc = static_cast<uint8_t*>(gate_sc);
    a.up_q = static_cast<uint8_t*>(up_q);
    a.up_sc = static_cast<uint8_t*>(up_sc);
    a.hidden_q = static_cast<uint8_t*>(hidden_q);
    a.hidden_sc = static_cast<uint8_t*>(hidden_sc);
    a.hidden_qt = static_cast<uint8_t*>(hidden_qt);
    a.hidden_sct = static_cast<uint8_t*>(hidden_sct);
    a.sc_row_tile_stride = sc_row_tile_stride;
    a.qt_ld = qt_ld;
    a.sct_row_tile_stride = sct_row_tile_stride;
    a.num_tokens = num_tokens;
    a.row_begin = row_begin;
    a.row_end = row_end;
    a.cols = cols;
    a.limit = limit;
    static bool done_clamp[16] = {false}, done_plain[16] = {false};
    if (has_limit)
        return launch_tile_kernel(swiglu_quantize_fwd_kernel<true>, "swiglu_quantize_fwd_kernel", done_clamp, a, cols,
                                  row_end - row_begin, 128, 0, stream);
    return launch_tile_kernel(swiglu_quantize_fwd_kernel<false>, "swiglu_quantize_fwd_kernel", done_plain, a, cols,
                              row_end - row_begin, 128, 0, stream);
}

int launch_swiglu_quantize_bwd(const void* gate_q, const void* gate_sc, const void* up_q, const void* up_sc, const void* d_hidden,
                               int cols, const int32_t* num_tokens, int row_begin, int row_end, void* d_gate_q, void* d_gate_sc,
                               void* d_up_q, void* d_up_sc, long long sc_row_tile_stride, void* d_gate_qt, void* d_gate_sct,
                               void* d_up_qt, void* d_up_sct, long long qt_ld, long long sct_row_tile_stride, float* row_partial,
                               bool has_limit, float limit, cudaStream_t stream) {
    if (!gate_q || !gate_sc || !up_q || !up_sc || !d_hidden || !num_tokens || !d_gate_q || !d_gate_sc || !d_up_q || !d_up_sc ||
        !d_gate_qt || !d_gate_sct || !d_up_qt || !d_up_sct || !row_partial)
        return MOK_ERR_INVALID_ARGUMENT;
    if (cols <= 0 || cols % 128 != 0 || row_end <= row_begin || (row_end - row_begin) % 128 != 0) return MOK_ERR_INVALID_ARGUMENT;
    FusedBwdArgs a{};
    a.gate_q = static_cast<const uint8_t*>(gate_q);
    a.gate_sc = static_cast<const uint8_t*>(gate_sc);
    a.up_q = static_cast<const uint8_t*>(up_q);
    a.up_sc = static_cast<const uint8_t*>(up_sc);
    a.d_hidden = static_cast<const bf16*>(d_hidden);
    a.dg_q = static_cast<uint8_t*>(d_gate_q);
    a.dg_sc = static_cast<uint8_t*>(d_gate_sc);
    a.du_q = static_cast<uint8_t*>(d_up_q);
    a.du_sc = static_cast<uint8_t*>(d_up_sc);
    a.dg_qt = static_cast<uint8_t*>(d_gate_qt);
    a.dg_sct = static_cast<uint8_t*>(d_gate_sct);
    a.du_qt = static_cast<uint8_t*>(d_up_qt);
    a.du_sct = static_cast<uint8_t*>(d_up_sct);
    a.sc_row_tile_stride = sc_row_tile_stride;
    a.qt_ld = qt_ld;
    a.sct_row_tile_stride = sct_row_tile_stride;
    a.row_partial = row_partial;
    a.num_tokens = num_tokens;
    a.row_begin = row_begin;
    a.row_end = row_end;
    a.cols = cols;
    a.limit = limit;
    static bool done_clamp[16] = {false}, done_plain[16] = {false};
    if (has_limit)
        return launch_tile_kernel(swiglu_quantize_bwd_kernel<true>, "swiglu_quantize_bwd_kernel", done_clamp, a, cols,
                                  row_end - row_begin, 256, 2 * kTileBytes, stream);
    return launch_tile_kernel(swiglu_quantize_bwd_kernel<false>, "swiglu_quantize_bwd_kernel", done_plain, a, cols,
                              row_end - row_begin, 256, 2 * kTileBytes, stream);
}

int launch_router_grad(const float* row_partial, int tiles, const float* row_weight, float* row_grad, const int32_t* num_tokens,
                       int row_begin, int row_end, cudaStream_t stream) {
    if (!row_partial || !row_weight || !row_grad || !num_tokens || tiles <= 0 || row_end <= row_begin) return MOK_ERR_INVALID_ARGUMENT;
    long long blocks = (static_cast<long long>(row_end - row_begin) + 255) / 256;
    const long long cap = static_cast<long long>(sm_count()) * 8;
    if (blocks > cap) blocks = cap;
    router_grad_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(row_partial, tiles, row_weight, row_grad, num_tokens, row_begin,
                                                                     row_end);
    MOK_LAUNCH_CHECK("router_grad_kernel");
    return MOK_OK;
}

}  // namespace mok

extern "C" int mok_mxfp8_quantize(const void* x_bf16, int num_matrices, int rows, int cols, void* x_fp8, void* x_sc,
                                  void* x_fp8_t, void* x_sc_t, mok_stream_t stream) {
    using namespace mok;
    if (x_bf16 == nullptr || num_matrices <= 0 || rows <= 0 || cols <= 0 || rows % 128 != 0 || cols % 128 != 0)
        return MOK_ERR_INVALID_ARGUMENT;
    if ((x_fp8 == nullptr) != (x_sc == nullptr) || (x_fp8_t == nullptr) != (x_sc_t == nullptr)) return MOK_ERR_INVALID_ARGUMENT;
    if (x_fp8 == nullptr && x_fp8_t == nullptr) return MOK_ERR_INVALID_ARGUMENT;
    if (num_matrices > 65535 || rows / 128 > 65535) return MOK_ERR_TOO_LARGE;
    const long long elems = static_cast<long long>(rows) * cols;
    QuantArgs a{};
    a.x = static_cast<const bf16*>(x_bf16);
    a.x_ld = cols;
    a.x_mat_stride = elems;
    a.q = static_cast<uint8_t*>(x_fp8);
    a.q_mat_stride = elems;
    a.sc = static_cast<uint8_t*>(x_sc);
    a.sc_row_tile_stride = static_cast<long long>(cols / 128) * 512;
    a.sc_mat_stride = static_cast<long long>(rows / 128) * a.sc_row_tile_stride;
    a.qt = static_cast<uint8_t*>(x_fp8_t);
    a.qt_ld = rows;
    a.qt_mat_stride = elems;
    a.sct = static_cast<uint8_t*>(x_sc_t);
    a.sct_row_tile_stride = static_cast<long long>(rows / 128) * 512;
    a.sct_mat_stride = static_cast<long long>(cols / 128) * a.sct_row_tile_stride;
    a.num_tokens = nullptr;
    a.row_begin = 0;
    a.row_end = rows;
    dim3 grid(cols / 128, rows / 128, num_matrices);
    return launch_quantize<false>(a, LocalRows{}, grid, reinterpret_cast<cudaStream_t>(stream));
}
