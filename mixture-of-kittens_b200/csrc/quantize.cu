// MXFP8 codec kernels: bf16 -> E4M3 with one E8M0 scale per 32 elements, along rows
// ("normal") and/or along columns ("transposed": the quantisation of x^T), scales laid out
// in the 32 x 16-byte tiles that tcgen05 block-scaled MMA consumes.
//   quantize_kernel         plain quantiser            (reference: csrc/mxfp8.cuh:188-278)
//   (SwiGLU forward + quantise is the epilogue of the MXFP8 gate/up GEMM, gemm_mxfp8.cu)
//   swiglu_bwd_quant_kernel de-quantise saved gate/up, SwiGLU backward, router-gradient partials,
//                           quantise d_gate / d_up      (reference: swiglu.cuh:209-566)
// One 128 x 128 tile per CTA.  A thread quantises 16 columns of a row straight from the registers it
// loaded them into (the block maximum is shared with the neighbouring lane) and stages them in shared
// memory as packed bf16 pairs; the column-wise pass (a thread owns 32 rows of two adjacent columns)
// reads them back.  Both are free of bank conflicts, and every global access covers whole lines.  The kernels
// are bound by HBM, but only if the per-element instruction count stays small: everything works on
// bf16 pairs (packed abs/max for the block maximum, one conversion instruction per two outputs)
// and global memory is touched 32 bytes per thread per instruction.
#include <cuda_fp8.h>

#include "common.cuh"
#include "mxfp8_codec.cuh"

namespace mokb {
namespace {

constexpr int TILE = 128;
constexpr int TILE_WORDS = TILE * TILE / 2;

// Where word c (a pair of columns) of row r lies in a staged tile: 64 words per row in 16-byte units, the unit number
// XORed so that both passes are free of bank conflicts.  A row is written by eight lanes, 32 bytes each: flipping the
// lowest bit in the upper half of the row spreads a quarter-warp's 16-byte stores over all banks.  A warp reads eight
// words of each of four rows that lie 32 apart: the row's block number, shifted by one, puts those on different banks.
__device__ __forceinline__ int tile_unit(int r, int u) { return r * 16 + (u ^ (u >> 3) ^ ((r >> 5) << 1)); }
__device__ __forceinline__ void stage_16_columns(uint32_t* tile, int r, int seg, const uint32_t (&w)[8]) {
    uint4* t = reinterpret_cast<uint4*>(tile);
    t[tile_unit(r, 2 * seg)] = make_uint4(w[0], w[1], w[2], w[3]);
    t[tile_unit(r, 2 * seg + 1)] = make_uint4(w[4], w[5], w[6], w[7]);
}

// Row-wise quantisation from registers: lanes 2j and 2j+1 hold one 32-value block (16 consecutive values each).
// Eight lanes store 128 contiguous bytes of a row.
__device__ __forceinline__ void quantize_16_columns(const uint32_t (&w)[8], uint8_t* q_dst, uint8_t* sc_dst) {
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = absmax2(m, w[i]);
    float amax = fmaxf(bf16_lo(m), bf16_hi(m));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    float inv;
    const uint32_t byte = scale_byte(amax, &inv);
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        o[i] = e4m3x4(bf16_lo(w[2 * i]) * inv, bf16_hi(w[2 * i]) * inv, bf16_lo(w[2 * i + 1]) * inv, bf16_hi(w[2 * i + 1]) * inv);
    *reinterpret_cast<uint4*>(q_dst) = make_uint4(o[0], o[1], o[2], o[3]);
    if ((threadIdx.x & 1) == 0) *sc_dst = static_cast<uint8_t>(byte);
}

// Column-wise quantisation of a staged tile into qt [cols, rows] (+ scales), 256 threads: a thread owns 32 rows of a pair
// of adjacent columns.  The four row blocks of a column sit in neighbouring lanes, so that a store instruction writes
// whole 128-byte lines of eight columns instead of 32 bytes of 32 of them.
__device__ __forceinline__ void quantize_tile_cols(const uint32_t* tile, uint8_t* qt, uint8_t* sct, int64_t col_base,
                                                   int64_t r0, int64_t c0, int64_t rows) {
    const int kb = threadIdx.x & 3, cp = threadIdx.x >> 2;
    uint32_t w[32];
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        w[i] = tile[tile_unit(kb * 32 + i, cp >> 2) * 4 + (cp & 3)];
        m = absmax2(m, w[i]);
    }
    float inv_a, inv_b;
    const uint32_t byte_a = scale_byte(bf16_lo(m), &inv_a);
    const uint32_t byte_b = scale_byte(bf16_hi(m), &inv_b);
    uint32_t out[8];
    const int64_t col = col_base + c0 + 2 * cp;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        out[i] = e4m3x4(bf16_lo(w[4 * i]) * inv_a, bf16_lo(w[4 * i + 1]) * inv_a, bf16_lo(w[4 * i + 2]) * inv_a, bf16_lo(w[4 * i + 3]) * inv_a);
    st_global_32B(qt + col * rows + r0 + kb * 32, out);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        out[i] = e4m3x4(bf16_hi(w[4 * i]) * inv_b, bf16_hi(w[4 * i + 1]) * inv_b, bf16_hi(w[4 * i + 2]) * inv_b, bf16_hi(w[4 * i + 3]) * inv_b);
    st_global_32B(qt + (col + 1) * rows + r0 + kb * 32, out);
    sct[scale_offset(col, (r0 >> 5) + kb, rows >> 7)] = static_cast<uint8_t>(byte_a);
    sct[scale_offset(col + 1, (r0 >> 5) + kb, rows >> 7)] = static_cast<uint8_t>(byte_b);
}

// Rows [begin, min(end, *num_rows)); the grid's y index counts 128-row tiles from `begin`.  Row numbers are those of the
// caller's row space (the schedule's, for the layer): a buffer that holds only rows [first, first + M) of it is passed
// with its pointers moved back by `first` rows, so begin/end may exceed the buffer's own row count M.
struct RowWindow {
    const int32_t* num_rows;
    int begin, end;
};
__device__ __forceinline__ bool tile_in_window(const RowWindow& w, int64_t* r0) {
    *r0 = static_cast<int64_t>(blockIdx.y) * TILE + w.begin;
    const int live = w.num_rows ? min(max(*w.num_rows, 0), w.end) : w.end;
    return *r0 < live;
}

// 256 threads per block; the blocks of the launch walk the 128 x 128 tiles (column tiles fastest).
// 32 x 2048 x 7168 both ways: 341 us (5.6 TB/s), row-wise alone 229 (6.2).  The SM's default split between L1 and shared memory is
// part of that: with the GEMMs' split (all shared memory, as the pulls that run beside them have it) 458 and 322 us.
__global__ void __launch_bounds__(256) quantize_kernel(const __nv_bfloat16* __restrict__ x, int64_t E, int64_t M, int64_t N,
                                                       uint8_t* __restrict__ q, uint8_t* __restrict__ sc,
                                                       uint8_t* __restrict__ qt, uint8_t* __restrict__ sct) {
    __shared__ __align__(16) uint32_t tile[TILE_WORDS];
    const int64_t row_tiles = M / TILE;
    const int64_t col_tiles = N / TILE;
    const int64_t ntiles = E * row_tiles * col_tiles;
    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int64_t e = t / (row_tiles * col_tiles);
        const int64_t rem = t - e * row_tiles * col_tiles;
        const int64_t rt = rem / col_tiles;
        const int64_t c0 = (rem - rt * col_tiles) * TILE;
        const int64_t r0 = rt * TILE;
        const int seg = threadIdx.x & 7, rr = threadIdx.x >> 3;      // 16 columns of rows rr, rr + 32, ..
        const __nv_bfloat16* src = x + (e * M + r0 + rr) * N + c0 + seg * 16;
        uint32_t val[4][8];
#pragma unroll
        for (int k = 0; k < 4; ++k) ld_global_32B(src + 32 * k * N, val[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t row = e * M + r0 + rr + 32 * k;
            if (qt) stage_16_columns(tile, rr + 32 * k, seg, val[k]);
            if (q) quantize_16_columns(val[k], q + row * N + c0 + seg * 16, sc + scale_offset(row, (c0 >> 5) + (seg >> 1), N >> 7));
        }
        __syncthreads();
        if (qt) quantize_tile_cols(tile, qt, sct, e * N, r0, c0, M);
        __syncthreads();          // the tile is free for the next load
    }
}

// Column-wise ("transposed") quantisation of one matrix only, for callers that ask for nothing else: qt [N, M] + scales from
// x [M, N].  No shared memory and at most 64 registers.  A lane owns a pair of adjacent columns over a block of 32 rows: its 32
// loads are independent, and a warp's load of one row is one 128-byte line.  Same arithmetic as quantize_tile_cols.
constexpr int CTILE_COLS = 64;
__global__ void __maxnreg__(64) quantize_cols_kernel(const __nv_bfloat16* __restrict__ x, int64_t M, int64_t N,
                                                     uint8_t* __restrict__ qt, uint8_t* __restrict__ sct) {
    const int64_t col_tiles = N / CTILE_COLS;
    const int64_t ntiles = M / TILE * col_tiles;
    const int cp = threadIdx.x & 31, kb = threadIdx.x >> 5;      // a pair of adjacent columns, a block of 32 rows
    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int64_t rt = t / col_tiles;
        const int64_t c0 = (t - rt * col_tiles) * CTILE_COLS;
        const int64_t r0 = rt * TILE + kb * 32;
        const int64_t col = c0 + 2 * cp;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(x + r0 * N + col);
        const int64_t pitch = N / 2;                             // 32-bit words per row
        // pass 1: the block maximum of both columns, eight independent loads at a time; pass 2 reads the rows again
        // (cache hits) four at a time.  Keeping the 32 values (and the 32 row addresses) in registers across the
        // conversion would take about 170 registers; this way the kernel stays within 64.
        uint32_t m = 0u;
        const uint32_t* p1 = src;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = __ldg(p1 + i * pitch);
#pragma unroll
            for (int i = 0; i < 8; ++i) m = absmax2(m, w[i]);
            p1 += 8 * pitch;
        }
        float inv_a, inv_b;
        const uint32_t byte_a = scale_byte(bf16_lo(m), &inv_a);
        const uint32_t byte_b = scale_byte(bf16_hi(m), &inv_b);
        uint32_t out_a[8], out_b[8];
        const uint32_t* p2 = src;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)       // (volatile: must stay a second load, not a reuse of pass 1's registers)
                asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(w[j]) : "l"(p2 + j * pitch));
            p2 += 4 * pitch;
            out_a[i] = e4m3x4(bf16_lo(w[0]) * inv_a, bf16_lo(w[1]) * inv_a, bf16_lo(w[2]) * inv_a, bf16_lo(w[3]) * inv_a);
            out_b[i] = e4m3x4(bf16_hi(w[0]) * inv_b, bf16_hi(w[1]) * inv_b, bf16_hi(w[2]) * inv_b, bf16_hi(w[3]) * inv_b);
        }
        st_global_32B(qt + col * M + r0, out_a);
        st_global_32B(qt + (col + 1) * M + r0, out_b);
        sct[scale_offset(col, r0 >> 5, M >> 7)] = static_cast<uint8_t>(byte_a);
        sct[scale_offset(col + 1, r0 >> 5, M >> 7)] = static_cast<uint8_t>(byte_b);
    }
}

struct Clamp {
    int on;
    float limit;
};


// two E4M3 bytes (the low 16 bits of v) -> two floats
__device__ __forceinline__ float2 e4m3x2_to_float2(uint32_t v) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(v & 0xffffu), __NV_E4M3);
    return __half22float2(*reinterpret_cast<const __half2*>(&h));
}

// Saved gate/up (E4M3 + scales), d_hidden bf16 -> d_gate, d_up, their row-wise and column-wise quantisations,
// and the per-(row, 128-column block) router-gradient partial sum(d_hidden * silu(g) * u) / w.
// grid (I/128, window rows/128), 256 threads: eight threads per row, 16 columns each, rows 32 apart in four trips; the next
// trip's operands are in flight while this one's are worked on.  Every global access of a warp covers whole 128-byte
// lines of four rows.  d_gate / d_up are quantised row-wise from registers and staged (two tiles) for the column-wise pass.
// The row gradient is summed in the order of the columns, so the lanes of a row hand the sum on, 32 registers of factors each:
// two blocks per SM (three would spill: 1094 us).  135 k rows of 2048: 752 us (3.0 TB/s), bound by instructions, of which the
// IEEE quotients take 110 us and the order of the sum 30; 1188 us with a row per thread and 32 columns.
__global__ void __launch_bounds__(256, 2) swiglu_bwd_quant_kernel(
    const uint8_t* __restrict__ gate_q, const uint8_t* __restrict__ gate_sc, const uint8_t* __restrict__ up_q,
    const uint8_t* __restrict__ up_sc, const __nv_bfloat16* __restrict__ d_hidden, int64_t rows_cap, int64_t I,
    RowWindow win, Clamp c, const float* __restrict__ row_scale,
    uint8_t* dg_q, uint8_t* dg_sc, uint8_t* dg_qt, uint8_t* dg_sct,
    uint8_t* du_q, uint8_t* du_sc, uint8_t* du_qt, uint8_t* du_sct, float* __restrict__ partials) {
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t *tdg = sm, *tdu = sm + TILE_WORDS;
    const int64_t c0 = static_cast<int64_t>(blockIdx.x) * TILE;
    int64_t r0;
    if (!tile_in_window(win, &r0)) return;
    const int seg = threadIdx.x & 7, rr = threadIdx.x >> 3;
    const int64_t col = c0 + seg * 16;
    const size_t sc_off = scale_offset(r0 + rr, col >> 5, I >> 7);      // of row rr + 32 k: 4 k bytes further on
    struct Operands {
        uint4 g, u;
        uint32_t dh[8];
        uint32_t gs, us;
        float w;
    };
    auto fetch = [&](int k) {
        Operands o;
        const int64_t row = r0 + rr + 32 * k;
        o.g = *reinterpret_cast<const uint4*>(gate_q + row * I + col);
        o.u = *reinterpret_cast<const uint4*>(up_q + row * I + col);
        ld_global_32B(d_hidden + row * I + col, o.dh);
        o.gs = gate_sc[sc_off + 4 * k];
        o.us = up_sc[sc_off + 4 * k];
        o.w = row_scale ? row_scale[row] : 1.0f;
        return o;
    };
    Operands next = fetch(0);
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        const Operands o = next;
        if (k < 3) next = fetch(k + 1);
        const int64_t row = r0 + rr + 32 * k;
        const float gs = __uint_as_float(o.gs << 23), us = __uint_as_float(o.us << 23);
        const float inv_w = o.w > 0.0f ? 1.0f / o.w : 0.0f;
        const uint32_t gv[4] = {o.g.x, o.g.y, o.g.z, o.g.w}, uv[4] = {o.u.x, o.u.y, o.u.z, o.u.w};
        uint32_t wg[8], wu[8];
        float rg_a[16], rg_b[16];          // factors of the row gradient's terms
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 gq = e4m3x2_to_float2(gv[i >> 1] >> ((i & 1) * 16));
            const float2 uq = e4m3x2_to_float2(uv[i >> 1] >> ((i & 1) * 16));
            const float gg[2] = {gq.x * gs, gq.y * gs}, uu[2] = {uq.x * us, uq.y * us};
            const float dhv[2] = {bf16_lo(o.dh[i]), bf16_hi(o.dh[i])};
            float dg[2], du[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float g = gg[j], u = uu[j];
                bool g_ok = true, u_ok = true;
                if (c.on) {
                    g_ok = g <= c.limit;
                    u_ok = (u >= -c.limit) && (u <= c.limit);
                    g = fminf(g, c.limit);
                    u = fminf(fmaxf(u, -c.limit), c.limit);
                }
                const float sig = 1.0f / (1.0f + __expf(-g));      // (IEEE: __fdividef is zero for gates between -88.7 and -87.3)
                const float silu = g * sig;
                const float dsilu = (1.0f - silu) * sig + silu;
                dg[j] = g_ok ? dsilu * u * dhv[j] : 0.0f;
                du[j] = u_ok ? silu * dhv[j] : 0.0f;
                rg_a[2 * i + j] = dhv[j] * inv_w;
                rg_b[2 * i + j] = silu * u;
            }
            wg[i] = pack2(dg[0], dg[1]);
            wu[i] = pack2(du[0], du[1]);
        }
        stage_16_columns(tdg, rr + 32 * k, seg, wg);
        stage_16_columns(tdu, rr + 32 * k, seg, wu);
        quantize_16_columns(wg, dg_q + row * I + col, dg_sc + sc_off + 4 * k);
        quantize_16_columns(wu, du_q + row * I + col, du_sc + sc_off + 4 * k);
        if (partials) {      // the 64 columns of a half row in ascending order, handed from lane to lane; then the two halves
            float run = 0.0f;
#pragma unroll
            for (int s = 0; s < 4; ++s) {      // (after step s the first s + 1 lanes of a half row hold their final sums)
                const float left = __shfl_up_sync(0xffffffffu, run, 1);
                run = (seg & 3) ? left : 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) run = fmaf(rg_a[i], rg_b[i], run);
            }
            const float upper = __shfl_down_sync(0xffffffffu, run, 4);
            if (seg == 3) partials[row * (I >> 7) + blockIdx.x] = run + upper;
        }
    }
    __syncthreads();
    quantize_tile_cols(tdg, dg_qt, dg_sct, 0, r0, c0, rows_cap);
    quantize_tile_cols(tdu, du_qt, du_sct, 0, r0, c0, rows_cap);
}

// row_grad[row] = sum over the column blocks of partials[row, :], in block order (fixed, reproducible)
__global__ void row_sum_kernel(const float* __restrict__ partials, int nblk, RowWindow win, float* __restrict__ out) {
    const int rows = win.num_rows ? min(max(*win.num_rows, 0), win.end) : win.end;
    for (int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x + win.begin; row < rows;
         row += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        float s = 0.0f;
        for (int b = 0; b < nblk; ++b) s += partials[row * nblk + b];
        out[row] = s;
    }
}

}  // namespace

namespace {
bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }
int check_window(const char* who, int row_begin, int* row_end, int64_t rows) {
    if (*row_end <= 0) *row_end = static_cast<int>(rows);
    MOKB_REQUIRE(row_begin >= 0 && row_begin % 128 == 0 && *row_end % 128 == 0 && row_begin <= *row_end && *row_end - row_begin <= rows,
                 "%s: bad row window [%d, %d) for %lld rows", who, row_begin, *row_end, static_cast<long long>(rows));
    return MOKB_OK;
}
}  // namespace

int swiglu_bwd_quant_impl(const void* gate_q, const void* gate_sc, const void* up_q, const void* up_sc, const void* d_hidden,
                          int64_t rows_cap, int64_t I, const int32_t* num_rows, int row_begin, int row_end, int has_limit, float limit,
                          const float* row_scale, void* dg_q, void* dg_sc, void* dg_qt, void* dg_sct,
                          void* du_q, void* du_sc, void* du_qt, void* du_sct, float* partials, float* row_grad,
                          cudaStream_t stream) {
    TraceScope trace(stream, "swiglu_bwd_quant", row_begin);
    MOKB_REQUIRE(gate_q && gate_sc && up_q && up_sc && d_hidden && dg_q && dg_sc && dg_qt && dg_sct && du_q && du_sc && du_qt && du_sct,
                 "swiglu_bwd_quant: null pointer");
    MOKB_REQUIRE((partials == nullptr) == (row_grad == nullptr), "swiglu_bwd_quant: partials and row_grad go together");
    MOKB_REQUIRE(rows_cap > 0 && rows_cap % 128 == 0 && I > 0 && I % 128 == 0 && rows_cap / 128 <= 65535, "swiglu_bwd_quant: bad sizes");
    MOKB_REQUIRE(aligned32(gate_q) && aligned32(up_q) && aligned32(d_hidden) && aligned32(dg_q) && aligned32(dg_qt) && aligned32(du_q) &&
                 aligned32(du_qt), "swiglu_bwd_quant: tensors must be 32-byte aligned");
    MOKB_TRY(check_window("swiglu_bwd_quant", row_begin, &row_end, rows_cap));
    if (row_begin == row_end) return MOKB_OK;
    const size_t smem = 2 * TILE_WORDS * sizeof(uint32_t);
    MOKB_CUDA(cudaFuncSetAttribute(swiglu_bwd_quant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const RowWindow win{num_rows, row_begin, row_end};
    const dim3 grid(static_cast<unsigned>(I / 128), static_cast<unsigned>((row_end - row_begin) / 128));
    share_sms_with_gemm<swiglu_bwd_quant_kernel>();
    swiglu_bwd_quant_kernel<<<grid, 256, smem, stream>>>(
        static_cast<const uint8_t*>(gate_q), static_cast<const uint8_t*>(gate_sc), static_cast<const uint8_t*>(up_q),
        static_cast<const uint8_t*>(up_sc), static_cast<const __nv_bfloat16*>(d_hidden), rows_cap, I, win, Clamp{has_limit, limit},
        row_scale, static_cast<uint8_t*>(dg_q), static_cast<uint8_t*>(dg_sc), static_cast<uint8_t*>(dg_qt), static_cast<uint8_t*>(dg_sct),
        static_cast<uint8_t*>(du_q), static_cast<uint8_t*>(du_sc), static_cast<uint8_t*>(du_qt), static_cast<uint8_t*>(du_sct), partials);
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    if (row_grad) {
        const int blocks = min(sm_count() * 4, (row_end - row_begin + 255) / 256);
        row_sum_kernel<<<blocks, 256, 0, stream>>>(partials, static_cast<int>(I / 128), win, row_grad);
        MOKB_CUDA(cudaGetLastError());
        note_launch();
    }
    return MOKB_OK;
}

}  // namespace mokb

using namespace mokb;

extern "C" int mokb_mxfp8_quantize(const void* x_bf16, int64_t E, int64_t M, int64_t N,
                                   void* x_fp8, void* x_sc, void* x_fp8_t, void* x_sc_t, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    TraceScope trace(stream, "quantize");
    MOKB_REQUIRE(x_bf16 != nullptr, "mxfp8_quantize: null input");
    MOKB_REQUIRE(E > 0 && M > 0 && N > 0 && M % 128 == 0 && N % 128 == 0, "mxfp8_quantize: M and N must be positive multiples of 128");
    MOKB_REQUIRE((x_fp8 == nullptr) == (x_sc == nullptr) && (x_fp8_t == nullptr) == (x_sc_t == nullptr),
                 "mxfp8_quantize: data and scale outputs go together");
    MOKB_REQUIRE(x_fp8 || x_fp8_t, "mxfp8_quantize: at least one quantised layout must be requested");
    MOKB_REQUIRE(aligned32(x_bf16) && aligned32(x_fp8) && aligned32(x_fp8_t), "mxfp8_quantize: tensors must be 32-byte aligned");
    if (x_fp8 == nullptr && E == 1) {
        const int64_t ct = (M / 128) * (N / CTILE_COLS);
        const unsigned blocks = static_cast<unsigned>(ct < 8ll * sm_count() ? ct : 8ll * sm_count());
        quantize_cols_kernel<<<blocks, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x_bf16), M, N, static_cast<uint8_t*>(x_fp8_t),
                                                         static_cast<uint8_t*>(x_sc_t));
    } else {
        const int64_t tiles = E * (M / 128) * (N / 128);
        const unsigned blocks = static_cast<unsigned>(tiles < 16ll * sm_count() ? tiles : 16ll * sm_count());
        quantize_kernel<<<blocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x_bf16), E, M, N, static_cast<uint8_t*>(x_fp8),
                                                    static_cast<uint8_t*>(x_sc), static_cast<uint8_t*>(x_fp8_t), static_cast<uint8_t*>(x_sc_t));
    }
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}
