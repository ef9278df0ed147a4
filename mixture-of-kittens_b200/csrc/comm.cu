// Cross-GPU pieces of the layer, all over plain peer-to-peer loads and stores
// through NVLink/NVSwitch unicast addresses (no NCCL, no multicast object):
//   * route all-gather   (reference: csrc/utils.cuh:191-249, NVLS multicast store)
//   * device barrier     (reference: csrc/utils.cuh:251-299, multimem.red)
//   * dispatch = row pull from the token's home rank
//                        (reference: csrc/megakernel/dispatch_combine.cuh:1-150)
//   * combine  = row push into the home rank's [T*K, H] buffer
//                        (reference: dispatch_combine.cuh:152-266)
// With ep_size == 1 the same kernels run against the local pointers.
#include "common.cuh"
#include "mxfp8_codec.cuh"

namespace mokb {
namespace {

__device__ __forceinline__ void st_v4(void* p, uint4 v) {
    asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// W 32-bit words per access: 4 (16 bytes) or 8 (32 bytes: one full sector, half the instructions)
template <int W>
struct Words {
    uint32_t w[W];
};
template <int W>
__device__ __forceinline__ Words<W> ld_words(const void* p) {
    Words<W> v;
    if (W == 8) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]),
                     "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    } else {
        asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "l"(p));
    }
    return v;
}
template <int W>
__device__ __forceinline__ void st_words(void* p, const Words<W>& v) {
    if (W == 8) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]),
                     "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7]) : "memory");
    } else {
        asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]) : "memory");
    }
}

__global__ void all_gather_kernel(const uint4* __restrict__ src, PeerPtrs peers, int R, int rank, int64_t nvec) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec; i += stride) {
        const uint4 v = src[i];
        for (int r = 0; r < R; ++r) st_v4(static_cast<uint4*>(peers.p[r]) + rank * nvec + i, v);
    }
}

// One CTA.  Thread r adds 1 to rank r's barrier word (release, system scope);
// thread 0 then waits until the local word reaches the new target.
__global__ void barrier_kernel(PeerPtrs peers, int R, int rank, int32_t* target, int32_t* status,
                               unsigned long long timeout_ns) {
    __shared__ int new_target;
    if (threadIdx.x == 0) {
        new_target = *target + R;
        *target = new_target;
    }
    __syncthreads();
    if (threadIdx.x < R) {
        __threadfence_system();
        asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(peers.p[threadIdx.x]) : "memory");
    }
    if (threadIdx.x == 0) {
        const int32_t* mine = static_cast<const int32_t*>(peers.p[rank]);
        unsigned long long t0;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (uint32_t i = 0;; ++i) {
            int32_t v;
            asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(mine) : "memory");
            if (v - new_target >= 0) break;
            if ((i & 63) == 63) {
                unsigned long long t1;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
                if (t1 - t0 > timeout_ns) {
                    atomicCAS(status, MOKB_ST_OK, MOKB_ST_BARRIER_TIMEOUT);
                    break;
                }
                __nanosleep(100);
            }
        }
        __threadfence_system();
    }
}

// Row-wise MXFP8 form of the rows a dispatch pulls (QUANT variants): E4M3 bytes [rows, H] and packed scales.
struct RowQuant {
    uint8_t* q;
    uint8_t* sc;
    int col_tiles;          // H / 128
};

// A launch that feeds a running GEMM: its warps take pieces of the row window from `ticket` (zero at launch) in order, so
// that the rows arrive in order however many of the blocks are resident at a time, and count what they have finished in
// window_ready[window].  One launch serves all windows (there used to be one per window: at 256 rows a window the sixteen
// launches cost four times as much as the copies).
struct PullOrder {
    int32_t* ticket;             // null: a fixed share of the rows per warp, nothing counted
    int32_t* window_ready;
    int window_rows;             // a multiple of 256
};
__device__ __forceinline__ int take_ticket(int32_t* ticket) {
    int v = 0;
    if ((threadIdx.x & 31) == 0) v = atomicAdd(ticket, 1);
    return __shfl_sync(0xffffffffu, v, 0);
}
// the whole warp's stores so far are counted as `n` arrivals (a GEMM acquires the counter before it reads the rows)
__device__ __forceinline__ void count_arrivals(int32_t* counter, int n) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        red_release_gpu_add(counter, n);
    }
}

// One warp per schedule row, 16- or 32-byte accesses, four loads in flight per lane.  QUANT (32-byte accesses only; for callers of
// mokb_dispatch_rows_window that want the bf16 rows as well -- the MXFP8 layer pulls with pull_quant_kernel):
// the row is also quantised along its columns from the registers it passes through -- a lane holds 16 consecutive
// values, two neighbouring lanes one 32-value block (the reference quantises the tile it has just pulled,
// csrc/megakernel/dispatch_combine.cuh:88-114; the values are those of quantize_kernel, byte for byte).
template <bool SCALE, int W, bool QUANT>
__global__ void __maxnreg__(64) dispatch_kernel(PeerPtrs src, PeerPtrs scale_src, const int32_t* __restrict__ peer_rank,
                                const int32_t* __restrict__ peer_token_idx, const int32_t* __restrict__ num_rows,
                                int max_rows, int row_begin, int row_end, int R, int row_divisor, int vec_per_row,
                                Words<W>* __restrict__ dst, float* __restrict__ row_scale_out, int32_t* done_counter, RowQuant rq,
                                IndexGuard guard, PullOrder order) {
    int rows = num_rows ? *num_rows : max_rows;
    rows = rows < 0 ? 0 : (rows > max_rows ? 0 : rows);
    rows = min(rows, row_end);
    const int lane = threadIdx.x & 31;
    const int warps_per_block = blockDim.x >> 5;
    const int warp = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
    const int nwarps = gridDim.x * warps_per_block;
    // The indices (and the remote scale) of a warp's next row are fetched while it moves the current one: three
    // dependent round trips (indices, scale over NVLink, data over NVLink) would otherwise sit in front of every row.
    // Rows go in pieces of 1 << piece: one row at a fixed stride, or, by ticket, as many as leave every warp a few pieces
    // (a piece costs its warp a fence: about a microsecond, against 1.5 us for a row of 7168).
    int piece = 0;
    if (order.ticket) {
        const int share = (rows - row_begin) / nwarps;
        piece = share >= 32 ? 3 : share >= 8 ? 2 : share >= 2 ? 1 : 0;
    }
    int cur = order.ticket ? take_ticket(order.ticket) : warp;
    int nxt = order.ticket ? take_ticket(order.ticket) : warp + nwarps;
    int row = row_begin + (cur << piece);
    int pr_next = -1, tok_next = 0;
    float w_next = 1.f;
    auto fetch_indices = [&](int r) {
        pr_next = -1;
        if (r < rows) {
            pr_next = peer_rank[r];
            tok_next = peer_token_idx[r];
            if (pr_next >= 0 && pr_next < R && !index_ok(guard, tok_next, kBadIndexPull, r)) pr_next = -1;
            if (SCALE && pr_next >= 0 && pr_next < R) w_next = static_cast<const float*>(scale_src.p[pr_next])[tok_next];
        }
    };
    fetch_indices(row);
    int done = -1;               // the piece whose last row has been stored but not yet counted
    for (int next_row; row < rows; row = next_row) {
        if (done >= 0) {
            count_arrivals(order.window_ready + (done << piece) / order.window_rows, 1 << piece);
            done = -1;
        }
        const int pr = pr_next;
        const int tok = tok_next;
        const float w = SCALE ? w_next : 1.f;
        next_row = row + 1;
        if ((next_row - row_begin) >> piece != cur) {
            if (order.ticket) done = cur;
            cur = nxt;
            nxt = order.ticket ? take_ticket(order.ticket) : nxt + nwarps;
            next_row = row_begin + (cur << piece);
        }
        fetch_indices(next_row);
        Words<W>* out = dst + static_cast<size_t>(row) * vec_per_row;
        if (pr < 0 || pr >= R) {      // padding row (or a rank outside the pointer list: treated as padding, never dereferenced)
            Words<W> zero;
#pragma unroll
            for (int k = 0; k < W; ++k) zero.w[k] = 0u;
            for (int v = lane; v < vec_per_row; v += 32) st_words<W>(out + v, zero);
            if (SCALE && lane == 0 && row_scale_out) row_scale_out[row] = 0.f;
            if (QUANT) {          // a zero row: zero bytes and the scale of an all-zero block
                float inv;
                const uint8_t zb = static_cast<uint8_t>(scale_byte(0.f, &inv));
                for (int v = lane; v < vec_per_row; v += 32) {
                    asm volatile("st.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(rq.q + static_cast<size_t>(row) * vec_per_row * 16 + v * 16), "r"(0u) : "memory");
                    if ((v & 1) == 0) rq.sc[scale_offset(row, v >> 1, rq.col_tiles)] = zb;
                }
            }
            continue;
        }
        const Words<W>* in = static_cast<const Words<W>*>(src.p[pr]) + static_cast<size_t>(tok / row_divisor) * vec_per_row;
        if (SCALE && lane == 0 && row_scale_out) row_scale_out[row] = w;
        // (every lane makes the same number of trips: the quantising variant shuffles between lanes inside)
        for (int vb = 0; vb < vec_per_row; vb += 128) {
            const int v0 = vb + lane;
            Words<W> r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v0 + 32 * u < vec_per_row) r[u] = ld_words<W>(in + v0 + 32 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool live = v0 + 32 * u < vec_per_row;
                if (live) {
                    if (SCALE) {
#pragma unroll
                        for (int k = 0; k < W; ++k) {
                            const float2 f = unpack_bf16(r[u].w[k]);
                            r[u].w[k] = pack_bf16(f.x * w, f.y * w);
                        }
                    }
                    st_words<W>(out + v0 + 32 * u, r[u]);
                }
                if (QUANT) {      // lanes 2j and 2j+1 hold one 32-value block (W = 8: 16 values per lane); whole warp
                    uint32_t m = 0u;
                    if (live) {
#pragma unroll
                        for (int k = 0; k < W; ++k) m = absmax2(m, r[u].w[k]);
                    }
                    float amax = fmaxf(bf16_lo(m), bf16_hi(m));
                    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                    if (live) {
                        float inv;
                        const uint32_t byte = scale_byte(amax, &inv);
                        const int v = v0 + 32 * u;
                        uint32_t o[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = e4m3x4(bf16_lo(r[u].w[2 * k]) * inv, bf16_hi(r[u].w[2 * k]) * inv,
                                          bf16_lo(r[u].w[2 * k + 1]) * inv, bf16_hi(r[u].w[2 * k + 1]) * inv);
                        asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(rq.q + static_cast<size_t>(row) * vec_per_row * 16 + v * 16),
                                     "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                        if ((lane & 1) == 0) rq.sc[scale_offset(row, v >> 1, rq.col_tiles)] = static_cast<uint8_t>(byte);
                    }
                }
            }
        }
    }
    if (done >= 0) count_arrivals(order.window_ready + (done << piece) / order.window_rows, 1 << piece);
    if (done_counter) {      // this block's rows of the window have landed: one arrival for whoever consumes them
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            red_release_gpu_add(done_counter, 1);
        }
    }
}

// Row pull with both MXFP8 forms of the rows -- along columns (q, sc: what the row-tiled GEMMs read) and along tokens
// (qt, sct: what the weight gradients read) -- from the one read of each value: the bf16 rows are not stored.  (A pull
// that stored them and a second pass that read them twice for the token-wise form moved 8 bytes per value instead of 4.)
// A warp works on 32 rows x 32 columns at a time: a half-warp holds 16 rows, a lane two adjacent columns of them, so the
// token-wise block maximum is local but for one shuffle, and the column-wise maxima of 16 rows over 16 lanes take eight
// shuffles of packed pairs (half of the values change lanes at each step).  Few warps fit beside a GEMM, so everything that
// takes a round trip to memory is asked for ahead: the next 32 columns while these are worked on, the next unit's ticket,
// indices and first columns before this one is counted.  At most 128 registers and no shared memory: one block of 128
// threads fits beside any of the GEMMs.  The values are those of quantize_kernel, byte for byte.
// 135168 rows of 7168, alone: 1.25 ms on the whole chip (3.0 TB/s; pull 0.88 + second pass 0.85 before), 3.0 ms with one block per
// SM, bound by the latency of a warp's chain of instructions (32 x 64 columns without the loads ahead: 3.6 ms).
struct TokenQuant {
    uint8_t *q, *sc, *qt, *sct;
    int64_t t_rows;              // token columns of qt
};
constexpr int kQuantRows = 32, kQuantCols = 256;

// 32 rows (lane i knows row i's address) x 32 columns: v[i] = columns col, col + 1 of row i of the half-warp's 16.  The loads
// are unconditional: a load under a predicate is waited for where it stands (all of them cost a round trip each).
__device__ __forceinline__ void pull_columns(uint32_t (&v)[16], const uint32_t* row_ptr, int col) {
    const int base = threadIdx.x & 16;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(row_ptr), base | i));
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(v[i]) : "l"(p + (col >> 1)));
    }
}

template <bool SCALE>
__device__ __forceinline__ void quantize_columns(uint32_t (&v)[16], uint32_t live, float w, int r0, int col, int hidden, const TokenQuant& tq) {
    const int lane = threadIdx.x & 31, base = lane & 16;
    if (live != 0xffffffffu) {        // padding rows: whatever was loaded in their place
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (live >> (base | i)) & 1u ? v[i] : 0u;
    }
    if (SCALE) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float f = __shfl_sync(0xffffffffu, w, base | i);
            v[i] = pack2(bf16_lo(v[i]) * f, bf16_hi(v[i]) * f);
        }
    }
    {      // along tokens: this lane's 16 rows and those of the lane 16 away are one block of each of its two columns
        uint32_t m = 0u;
#pragma unroll
        for (int i = 0; i < 16; ++i) m = absmax2(m, v[i]);
        m = absmax2(m, __shfl_xor_sync(0xffffffffu, m, 16));
        float inv_a, inv_b;
        const uint32_t byte_a = scale_byte(bf16_lo(m), &inv_a);
        const uint32_t byte_b = scale_byte(bf16_hi(m), &inv_b);
        uint8_t* dst = tq.qt + col * tq.t_rows + r0 + base;
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            o[i] = e4m3x4(bf16_lo(v[4 * i]) * inv_a, bf16_lo(v[4 * i + 1]) * inv_a, bf16_lo(v[4 * i + 2]) * inv_a, bf16_lo(v[4 * i + 3]) * inv_a);
        *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            o[i] = e4m3x4(bf16_hi(v[4 * i]) * inv_b, bf16_hi(v[4 * i + 1]) * inv_b, bf16_hi(v[4 * i + 2]) * inv_b, bf16_hi(v[4 * i + 3]) * inv_b);
        *reinterpret_cast<uint4*>(dst + tq.t_rows) = make_uint4(o[0], o[1], o[2], o[3]);
        // the half-warps write the scale of one of the two columns each
        tq.sct[scale_offset(col + (base >> 4), r0 >> 5, tq.t_rows >> 7)] = static_cast<uint8_t>(base ? byte_b : byte_a);
    }
    // along columns: the 16 lanes of a half-warp hold one block of each of its rows
    uint32_t p[8];       // p[i]: this lane's maxima of rows i (low half) and i + 8 (high half)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t lo = __byte_perm(v[i], v[i + 8], 0x5410), hi = __byte_perm(v[i], v[i + 8], 0x7632);
        p[i] = absmax2(lo & 0x7fff7fffu, hi);
    }
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const uint32_t give = upper ? p[i] : p[i + half], keep = upper ? p[i + half] : p[i];
            p[i] = absmax2(keep, __shfl_xor_sync(0xffffffffu, give, half));
        }
    }
    p[0] = absmax2(p[0], __shfl_xor_sync(0xffffffffu, p[0], 8));
    // lane l now has the block maxima of rows l % 8 and l % 8 + 8 of its half-warp; it works out one of the two scales
    const bool second = (lane & 8) != 0;
    float inv;
    const uint32_t byte = scale_byte(second ? bf16_hi(p[0]) : bf16_lo(p[0]), &inv);
    tq.sc[scale_offset(r0 + base + (lane & 15), col >> 5, hidden >> 7)] = static_cast<uint8_t>(byte);
    uint8_t* dst = tq.q + static_cast<int64_t>(r0 + base) * hidden + col;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float f = __shfl_sync(0xffffffffu, inv, base | i);
        uint16_t pair;
        asm volatile("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(pair) : "f"(bf16_lo(v[i]) * f), "f"(bf16_hi(v[i]) * f));
        *reinterpret_cast<uint16_t*>(dst + static_cast<int64_t>(i) * hidden) = pair;
    }
}

template <bool SCALE>
__global__ void __maxnreg__(128) pull_quant_kernel(const __grid_constant__ PeerPtrs src, const __grid_constant__ PeerPtrs scale_src, const int32_t* __restrict__ peer_rank,
                                                   const int32_t* __restrict__ peer_token_idx, const int32_t* __restrict__ num_rows,
                                                   int max_rows, int row_begin, int row_end, int R, int row_divisor, int hidden,
                                                   float* __restrict__ row_scale_out, TokenQuant tq, IndexGuard guard, PullOrder order) {
    int rows = num_rows ? *num_rows : max_rows;
    rows = rows < 0 ? 0 : (rows > max_rows ? 0 : rows);
    rows = min(rows, row_end);
    const int lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    // a unit: 32 rows x 256, 512 or 1024 columns, as many as leave every warp a few units (counting one costs a fence)
    const int groups = rows > row_begin ? (rows - row_begin + kQuantRows - 1) / kQuantRows : 0;
    const int share = static_cast<int>(static_cast<int64_t>(groups) * (hidden / kQuantCols) / nwarps);
    const int unit_cols = kQuantCols << (share >= 32 ? 2 : share >= 16 ? 1 : 0);
    const int col_units = (hidden + unit_cols - 1) / unit_cols;
    const int units = groups * col_units;
    // row r0 + lane of a unit: its rank and route, then (a second round trip) its address and scale
    int pr = -1, tok = 0;
    auto look_up = [&](int unit) {
        const int row = row_begin + unit / col_units * kQuantRows + lane;
        pr = -1;
        if (unit < units && row < rows) {
            pr = peer_rank[row];
            tok = peer_token_idx[row];
        }
    };
    struct Rows {
        const uint32_t* ptr;         // of this lane's row; of a scheduled row of the unit if it is padding
        uint32_t live;               // which of the 32 rows are scheduled (none: nothing is loaded)
        float w;
    };
    auto resolve = [&](int unit) {
        Rows out;
        out.ptr = nullptr;
        out.w = 0.f;
        if (pr >= 0 && pr < R && index_ok(guard, tok, kBadIndexPull, row_begin + unit / col_units * kQuantRows + lane)) {
            out.ptr = static_cast<const uint32_t*>(src.p[pr]) + static_cast<size_t>(tok / row_divisor) * (hidden / 2);
            if (SCALE) out.w = static_cast<const float*>(scale_src.p[pr])[tok];
        }
        out.live = __ballot_sync(0xffffffffu, out.ptr != nullptr);
        const unsigned long long any = __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(out.ptr), __ffs(out.live | 0x80000000u) - 1);
        if (out.ptr == nullptr) out.ptr = reinterpret_cast<const uint32_t*>(any);
        return out;
    };
    auto next_unit = [&](int u) { return order.ticket ? take_ticket(order.ticket) : u + nwarps; };
    int unit = order.ticket ? take_ticket(order.ticket) : static_cast<int>(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    if (unit >= units) return;
    look_up(unit);
    Rows cur = resolve(unit);
    uint32_t va[16], vb[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) va[i] = vb[i] = 0u;
    const int lane_col = 2 * (lane & 15);
    if (cur.live) pull_columns(va, cur.ptr, unit % col_units * unit_cols + lane_col);
    while (unit < units) {
        const int g = unit / col_units;
        const int c0 = (unit - g * col_units) * unit_cols, c1 = min(c0 + unit_cols, hidden);
        const int r0 = row_begin + g * kQuantRows;
        if (SCALE && c0 == 0 && row_scale_out && r0 + lane < rows) row_scale_out[r0 + lane] = cur.w;
        int next = 0;
        Rows nxt = {nullptr, 0u, 0.f};
#pragma unroll 1
        for (int c = c0; c < c1; c += 64) {            // (at least four trips: the columns are a multiple of 256)
            if (cur.live) pull_columns(vb, cur.ptr, c + 32 + lane_col);
            if (c == c0) next = next_unit(unit);
            if (c == c0 + 64) look_up(next);
            if (c + 64 == c1) nxt = resolve(next);
            quantize_columns<SCALE>(va, cur.live, cur.w, r0, c + lane_col, hidden, tq);
            if (c + 64 < c1) {
                if (cur.live) pull_columns(va, cur.ptr, c + 64 + lane_col);
            } else if (nxt.live) {
                pull_columns(va, nxt.ptr, next % col_units * unit_cols + lane_col);
            }
            quantize_columns<SCALE>(vb, cur.live, cur.w, r0, c + 32 + lane_col, hidden, tq);
        }
        if (order.ticket) count_arrivals(order.window_ready + g * kQuantRows / order.window_rows, (c1 - c0) / kQuantCols);
        unit = next;
        cur = nxt;
    }
}

template <int W>
__global__ void combine_kernel(const Words<W>* __restrict__ src, PeerPtrs dst, PeerPtrs val_dst,
                               const int32_t* __restrict__ peer_rank, const int32_t* __restrict__ peer_token_idx,
                               const int32_t* __restrict__ num_rows, int max_rows, int row_begin, int row_end, int R,
                               int vec_per_row, const float* __restrict__ row_values, const int32_t* wait_counter,
                               int arrivals_per_row_block, int32_t* status, int index_limit) {
    int rows = num_rows ? *num_rows : max_rows;
    rows = rows < 0 ? 0 : (rows > max_rows ? 0 : rows);
    rows = min(rows, row_end);
    if (wait_counter) {
        // the rows come from a GEMM that is still running: wait (bounded) until every tile of this window is stored
        __shared__ int go;
        if (threadIdx.x == 0) {
            const int expected = ((rows - row_begin) / 256) * arrivals_per_row_block;
            go = expected <= 0 || flag_wait(wait_counter, expected, nullptr, status, kWaitWindowDone, row_begin / 256);
        }
        __syncthreads();
        if (!go) return;
    }
    const int lane = threadIdx.x & 31;
    const int warps_per_block = blockDim.x >> 5;
    const int warp = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
    const int nwarps = gridDim.x * warps_per_block;
    for (int row = row_begin + warp; row < rows; row += nwarps) {
        const int pr = peer_rank[row];
        if (pr < 0 || pr >= R) continue;
        const int tok = peer_token_idx[row];
        if (!index_ok(IndexGuard{index_limit, status}, tok, kBadIndexPush, row)) continue;
        const Words<W>* in = src + static_cast<size_t>(row) * vec_per_row;
        Words<W>* out = static_cast<Words<W>*>(dst.p[pr]) + static_cast<size_t>(tok) * vec_per_row;
        for (int v0 = lane; v0 < vec_per_row; v0 += 128) {
            Words<W> r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v0 + 32 * u < vec_per_row) r[u] = ld_words<W>(in + v0 + 32 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v0 + 32 * u < vec_per_row) st_words<W>(out + v0 + 32 * u, r[u]);
        }
        if (row_values && lane == 0) static_cast<float*>(val_dst.p[pr])[tok] = row_values[row];
    }
}

// 32-byte accesses need 32-byte aligned rows everywhere: the local buffer and every peer's
bool rows_aligned32(const void* local, const PeerPtrs& peers, int R, int64_t hidden) {
    if (hidden % 16 != 0 || (reinterpret_cast<uintptr_t>(local) & 31) != 0) return false;
    for (int r = 0; r < R; ++r)
        if ((reinterpret_cast<uintptr_t>(peers.p[r]) & 31) != 0) return false;
    return true;
}

int fill_peers(PeerPtrs* out, const uint64_t* host, int R, const char* what) {
    MOKB_REQUIRE(host != nullptr, "%s: null pointer list", what);
    for (int r = 0; r < kPeerMax; ++r) out->p[r] = nullptr;
    for (int r = 0; r < R; ++r) {
        MOKB_REQUIRE(host[r] != 0 && (host[r] & 15) == 0, "%s[%d] = 0x%llx is null or not 16-byte aligned", what, r,
                     (unsigned long long)host[r]);
        out->p[r] = reinterpret_cast<void*>(static_cast<uintptr_t>(host[r]));
    }
    return MOKB_OK;
}

unsigned long long g_barrier_timeout_ns = 10ull * 1000 * 1000 * 1000;

}  // namespace
}  // namespace mokb

using namespace mokb;

extern "C" int mokb_set_barrier_timeout_ms(int ms) {
    MOKB_REQUIRE(ms > 0, "barrier timeout must be positive");
    g_barrier_timeout_ns = static_cast<unsigned long long>(ms) * 1000ull * 1000ull;
    return MOKB_OK;
}

extern "C" int mokb_all_gather_top_experts(const int32_t* top_experts, const uint64_t* gather_buffer_ptrs_host,
                                           int ep_size, int rank, int64_t numel, void* stream) {
    TraceScope trace(static_cast<cudaStream_t>(stream), "all_gather_top_experts");
    MOKB_REQUIRE(top_experts != nullptr, "all_gather_top_experts: null input");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP && rank >= 0 && rank < ep_size, "all_gather_top_experts: bad ep_size/rank");
    MOKB_REQUIRE(numel > 0 && numel % 4 == 0, "all_gather_top_experts: numel must be a positive multiple of 4");
    MOKB_REQUIRE((reinterpret_cast<uintptr_t>(top_experts) & 15) == 0, "all_gather_top_experts: input not 16-byte aligned");
    PeerPtrs peers;
    MOKB_TRY(fill_peers(&peers, gather_buffer_ptrs_host, ep_size, "gather_buffer_ptrs"));
    const int64_t nvec = numel / 4;
    const int threads = 256;
    int64_t blocks = (nvec + threads - 1) / threads;
    if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
    all_gather_kernel<<<static_cast<unsigned>(blocks), threads, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const uint4*>(top_experts), peers, ep_size, rank, nvec);
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}

extern "C" int mokb_barrier_all(const uint64_t* barrier_ptrs_host, int ep_size, int rank, int32_t* target,
                                int32_t* status, void* stream) {
    TraceScope trace(static_cast<cudaStream_t>(stream), "barrier_all");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP && rank >= 0 && rank < ep_size, "barrier_all: bad ep_size/rank");
    MOKB_REQUIRE(target && status, "barrier_all: null pointer");
    PeerPtrs peers;
    MOKB_REQUIRE(barrier_ptrs_host != nullptr, "barrier_all: null pointer list");
    for (int r = 0; r < kPeerMax; ++r) peers.p[r] = nullptr;
    for (int r = 0; r < ep_size; ++r) {
        MOKB_REQUIRE(barrier_ptrs_host[r] != 0 && (barrier_ptrs_host[r] & 3) == 0, "barrier_all: bad pointer for rank %d", r);
        peers.p[r] = reinterpret_cast<void*>(static_cast<uintptr_t>(barrier_ptrs_host[r]));
    }
    barrier_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(peers, ep_size, rank, target, status, g_barrier_timeout_ns);
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}

namespace mokb {

int comm_default_blocks() { return sm_count() * 16; }

int dispatch_rows_impl(const uint64_t* src_ptrs_host, int ep_size, const int32_t* peer_rank,
                       const int32_t* peer_token_idx, const int32_t* num_rows, int max_rows, int row_begin, int row_end,
                       int row_divisor, int64_t hidden, void* dst, const uint64_t* row_scale_ptrs_host,
                       float* row_scale_out, int blocks, cudaStream_t s, int32_t* done_counter, void* q_out, void* q_sc_out,
                       int64_t index_limit, int32_t* status, int32_t* ticket, int window_rows) {
    TraceScope trace(s, row_scale_ptrs_host ? "dispatch_scaled" : "dispatch", row_begin);
    MOKB_REQUIRE((q_out == nullptr) == (q_sc_out == nullptr), "dispatch_rows: the quantised rows and their scales go together");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP, "dispatch_rows: bad ep_size");
    MOKB_REQUIRE(peer_rank && peer_token_idx && dst, "dispatch_rows: null pointer");
    MOKB_REQUIRE(max_rows >= 0 && row_divisor >= 1 && hidden > 0 && hidden % 8 == 0, "dispatch_rows: bad sizes");
    MOKB_REQUIRE(row_begin >= 0 && row_begin <= row_end, "dispatch_rows: bad row window");
    MOKB_REQUIRE(index_limit >= 0 && index_limit <= INT32_MAX && (index_limit == 0 || status != nullptr),
                 "dispatch_rows: index_limit needs a status word and must fit 31 bits");
    const IndexGuard guard{static_cast<int>(index_limit), status};
    MOKB_REQUIRE((reinterpret_cast<uintptr_t>(dst) & 15) == 0, "dispatch_rows: dst not 16-byte aligned");
    PeerPtrs src, scale;
    MOKB_TRY(fill_peers(&src, src_ptrs_host, ep_size, "src_ptrs"));
    for (int r = 0; r < kPeerMax; ++r) scale.p[r] = nullptr;
    if (max_rows == 0 || row_begin >= max_rows) return MOKB_OK;
    // 128 threads: one warp per SM quarter, so that a block finds room beside a GEMM CTA whatever that kernel's warp count
    const int threads = 128;
    if (blocks <= 0) blocks = comm_default_blocks();
    const bool wide = rows_aligned32(dst, src, ep_size, hidden);
    const int vec = static_cast<int>(hidden / (wide ? 16 : 8));
    for (int r = 0; r < ep_size && row_scale_ptrs_host; ++r) {
        MOKB_REQUIRE(row_scale_ptrs_host[r] != 0, "dispatch_rows: null scale pointer for rank %d", r);
        scale.p[r] = reinterpret_cast<void*>(static_cast<uintptr_t>(row_scale_ptrs_host[r]));
    }
    const RowQuant rq{static_cast<uint8_t*>(q_out), static_cast<uint8_t*>(q_sc_out), static_cast<int>(hidden / 128)};
    if (q_out) {
        MOKB_REQUIRE(wide && hidden % 128 == 0 && (reinterpret_cast<uintptr_t>(q_out) & 15) == 0,
                     "dispatch_rows: quantised output needs 32-byte aligned rows, hidden %% 128 == 0 and a 16-byte aligned buffer");
    }
#define MOKB_DISPATCH(SC, WW, QQ)                                                                                              \
    do {                                                                                                                       \
        share_sms_with_gemm<dispatch_kernel<SC, WW, QQ>>();                                                                    \
        dispatch_kernel<SC, WW, QQ><<<blocks, threads, 0, s>>>(src, scale, peer_rank, peer_token_idx, num_rows, max_rows,      \
            row_begin, row_end, ep_size, row_divisor, vec, static_cast<Words<WW>*>(dst), SC ? row_scale_out : nullptr,         \
            ticket ? nullptr : done_counter, rq, guard, PullOrder{ticket, done_counter, window_rows});                                                                                          \
    } while (0)
    if (row_scale_ptrs_host) {
        if (q_out) MOKB_DISPATCH(true, 8, true);
        else if (wide) MOKB_DISPATCH(true, 8, false);
        else MOKB_DISPATCH(true, 4, false);
    } else {
        if (q_out) MOKB_DISPATCH(false, 8, true);
        else if (wide) MOKB_DISPATCH(false, 8, false);
        else MOKB_DISPATCH(false, 4, false);
    }
#undef MOKB_DISPATCH
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}

// Arrivals that pull_quant_rows_impl counts per 256 rows (dispatch_rows_impl by ticket: 256).
int pull_quant_arrivals(int64_t hidden) { return static_cast<int>(256 / kQuantRows * (hidden / kQuantCols)); }

// Rows [row_begin, row_end) from their home ranks into both MXFP8 forms (q / sc, qt / sct addressed by schedule row;
// qt has t_rows token columns).  ticket / window_ready / window_rows: see PullOrder.
int pull_quant_rows_impl(const uint64_t* src_ptrs_host, int ep_size, const int32_t* peer_rank, const int32_t* peer_token_idx,
                         const int32_t* num_rows, int max_rows, int row_begin, int row_end, int row_divisor, int64_t hidden,
                         const uint64_t* row_scale_ptrs_host, float* row_scale_out, void* q, void* sc, void* qt, void* sct, int64_t t_rows,
                         int blocks, cudaStream_t s, int32_t* ticket, int32_t* window_ready, int window_rows, int64_t index_limit,
                         int32_t* status) {
    TraceScope trace(s, row_scale_ptrs_host ? "dispatch_quant_scaled" : "dispatch_quant", row_begin);
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP && peer_rank && peer_token_idx && q && sc && qt && sct, "pull_quant_rows: null pointer");
    MOKB_REQUIRE(hidden > 0 && hidden % kQuantCols == 0 && row_divisor >= 1 && row_begin >= 0 && row_begin <= row_end && row_begin % 128 == 0 && t_rows % 128 == 0,
                 "pull_quant_rows: bad sizes");
    // a warp stores 32 rows and 32 token columns at a time, also where the device's row count ends inside of them
    MOKB_REQUIRE(max_rows >= 0 && max_rows % 128 == 0 && row_end % 128 == 0, "pull_quant_rows: max_rows and row_end must be multiples of 128");
    MOKB_REQUIRE((row_end < max_rows ? row_end : max_rows) - row_begin <= t_rows, "pull_quant_rows: %d rows do not fit the %lld token columns",
                 (row_end < max_rows ? row_end : max_rows) - row_begin, static_cast<long long>(t_rows));
    MOKB_REQUIRE((reinterpret_cast<uintptr_t>(q) & 1) == 0 && (reinterpret_cast<uintptr_t>(qt) & 31) == 0, "pull_quant_rows: outputs not aligned");
    MOKB_REQUIRE(ticket == nullptr || (window_ready && window_rows > 0 && window_rows % 256 == 0), "pull_quant_rows: a ticket needs windows");
    MOKB_REQUIRE(index_limit >= 0 && index_limit <= INT32_MAX && (index_limit == 0 || status != nullptr), "pull_quant_rows: bad index limit");
    PeerPtrs src, scale;
    MOKB_TRY(fill_peers(&src, src_ptrs_host, ep_size, "src_ptrs"));
    for (int r = 0; r < kPeerMax; ++r) scale.p[r] = nullptr;
    for (int r = 0; r < ep_size && row_scale_ptrs_host; ++r) {
        MOKB_REQUIRE(row_scale_ptrs_host[r] != 0, "pull_quant_rows: null scale pointer for rank %d", r);
        scale.p[r] = reinterpret_cast<void*>(static_cast<uintptr_t>(row_scale_ptrs_host[r]));
    }
    if (max_rows == 0 || row_begin >= max_rows) return MOKB_OK;
    if (blocks <= 0) blocks = comm_default_blocks();
    const TokenQuant tq{static_cast<uint8_t*>(q), static_cast<uint8_t*>(sc), static_cast<uint8_t*>(qt), static_cast<uint8_t*>(sct), t_rows};
    const IndexGuard guard{static_cast<int>(index_limit), status};
    const PullOrder order{ticket, window_ready, window_rows};
    auto kernel = row_scale_ptrs_host ? pull_quant_kernel<true> : pull_quant_kernel<false>;
    if (row_scale_ptrs_host) share_sms_with_gemm<pull_quant_kernel<true>>();
    else share_sms_with_gemm<pull_quant_kernel<false>>();
    kernel<<<blocks, 128, 0, s>>>(src, scale, peer_rank, peer_token_idx, num_rows, max_rows, row_begin, row_end, ep_size, row_divisor,
                                  static_cast<int>(hidden), row_scale_out, tq, guard, order);
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}

int combine_rows_impl(const void* src, const uint64_t* dst_ptrs_host, int ep_size, const int32_t* peer_rank,
                      const int32_t* peer_token_idx, const int32_t* num_rows, int max_rows, int row_begin, int row_end,
                      int64_t hidden, const float* row_values, const uint64_t* value_ptrs_host, int blocks, cudaStream_t s,
                      const int32_t* wait_counter, int arrivals_per_row_block, int32_t* status, int64_t index_limit) {
    TraceScope trace(s, "combine", row_begin);
    MOKB_REQUIRE(index_limit >= 0 && index_limit <= INT32_MAX && (index_limit == 0 || status != nullptr),
                 "combine_rows: index_limit needs a status word and must fit 31 bits");
    MOKB_REQUIRE(wait_counter == nullptr || (arrivals_per_row_block > 0 && status != nullptr && row_begin % 256 == 0),
                 "combine_rows: a wait counter needs arrivals_per_row_block, a status word and a window that starts on a 256-row block");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP, "combine_rows: bad ep_size");
    MOKB_REQUIRE(src && peer_rank && peer_token_idx, "combine_rows: null pointer");
    MOKB_REQUIRE(max_rows >= 0 && hidden > 0 && hidden % 8 == 0, "combine_rows: bad sizes");
    MOKB_REQUIRE(row_begin >= 0 && row_begin <= row_end, "combine_rows: bad row window");
    MOKB_REQUIRE((row_values == nullptr) == (value_ptrs_host == nullptr), "combine_rows: row_values and value_ptrs go together");
    PeerPtrs dst, val;
    MOKB_TRY(fill_peers(&dst, dst_ptrs_host, ep_size, "dst_ptrs"));
    for (int r = 0; r < kPeerMax; ++r) val.p[r] = nullptr;
    if (value_ptrs_host)
        for (int r = 0; r < ep_size; ++r) {
            MOKB_REQUIRE(value_ptrs_host[r] != 0, "combine_rows: null value pointer for rank %d", r);
            val.p[r] = reinterpret_cast<void*>(static_cast<uintptr_t>(value_ptrs_host[r]));
        }
    if (max_rows == 0 || row_begin >= max_rows) return MOKB_OK;
    if (blocks <= 0) blocks = comm_default_blocks();
    share_sms_with_gemm<combine_kernel<8>>();
    share_sms_with_gemm<combine_kernel<4>>();
    if (rows_aligned32(src, dst, ep_size, hidden))
        combine_kernel<8><<<blocks, 128, 0, s>>>(static_cast<const Words<8>*>(src), dst, val, peer_rank, peer_token_idx, num_rows, max_rows,
                                                 row_begin, row_end, ep_size, static_cast<int>(hidden / 16), row_values, wait_counter,
                                                 arrivals_per_row_block, status, static_cast<int>(index_limit));
    else
        combine_kernel<4><<<blocks, 128, 0, s>>>(static_cast<const Words<4>*>(src), dst, val, peer_rank, peer_token_idx, num_rows, max_rows,
                                                 row_begin, row_end, ep_size, static_cast<int>(hidden / 8), row_values, wait_counter,
                                                 arrivals_per_row_block, status, static_cast<int>(index_limit));
    MOKB_CUDA(cudaGetLastError());
    note_launch();
    return MOKB_OK;
}

}  // namespace mokb

extern "C" int mokb_dispatch_rows(const uint64_t* src_ptrs_host, int ep_size, const int32_t* peer_rank,
                                  const int32_t* peer_token_idx, const int32_t* num_rows, int max_rows,
                                  int row_divisor, int64_t hidden, void* dst,
                                  const uint64_t* row_scale_ptrs_host, float* row_scale_out, void* stream) {
    return dispatch_rows_impl(src_ptrs_host, ep_size, peer_rank, peer_token_idx, num_rows, max_rows, 0, max_rows, row_divisor,
                              hidden, dst, row_scale_ptrs_host, row_scale_out, 0, static_cast<cudaStream_t>(stream), nullptr, nullptr, nullptr);
}

extern "C" int mokb_comm_default_blocks(void) { return comm_default_blocks(); }

extern "C" int mokb_dispatch_rows_window(const uint64_t* src_ptrs_host, int ep_size, const int32_t* peer_rank,
                                         const int32_t* peer_token_idx, const int32_t* num_rows, int max_rows, int row_begin,
                                         int row_end, int row_divisor, int64_t hidden, void* dst,
                                         const uint64_t* row_scale_ptrs_host, float* row_scale_out, int blocks,
                                         int32_t* done_counter, void* q_out, void* q_sc_out, int64_t index_limit,
                                         int32_t* status, void* stream) {
    return dispatch_rows_impl(src_ptrs_host, ep_size, peer_rank, peer_token_idx, num_rows, max_rows, row_begin, row_end, row_divisor,
                              hidden, dst, row_scale_ptrs_host, row_scale_out, blocks, static_cast<cudaStream_t>(stream), done_counter,
                              q_out, q_sc_out, index_limit, status);
}

extern "C" int mokb_dispatch_rows_quant(const uint64_t* src_ptrs_host, int ep_size, const int32_t* peer_rank, const int32_t* peer_token_idx,
                                        const int32_t* num_rows, int max_rows, int row_begin, int row_end, int row_divisor, int64_t hidden,
                                        const uint64_t* row_scale_ptrs_host, float* row_scale_out, void* q, void* sc, void* qt, void* sct,
                                        int64_t t_rows, int blocks, int32_t* ticket, int32_t* window_ready, int window_rows,
                                        int64_t index_limit, int32_t* status, void* stream) {
    return pull_quant_rows_impl(src_ptrs_host, ep_size, peer_rank, peer_token_idx, num_rows, max_rows, row_begin, row_end, row_divisor, hidden,
                                row_scale_ptrs_host, row_scale_out, q, sc, qt, sct, t_rows, blocks, static_cast<cudaStream_t>(stream), ticket,
                                window_ready, window_rows, index_limit, status);
}

extern "C" int mokb_combine_rows(const void* src, const uint64_t* dst_ptrs_host, int ep_size,
                                 const int32_t* peer_rank, const int32_t* peer_token_idx,
                                 const int32_t* num_rows, int max_rows, int64_t hidden,
                                 const float* row_values, const uint64_t* value_ptrs_host, void* stream) {
    return combine_rows_impl(src, dst_ptrs_host, ep_size, peer_rank, peer_token_idx, num_rows, max_rows, 0, max_rows, hidden,
                             row_values, value_ptrs_host, 0, static_cast<cudaStream_t>(stream), nullptr, 0, nullptr);
}

extern "C" int mokb_combine_rows_window(const void* src, const uint64_t* dst_ptrs_host, int ep_size,
                                        const int32_t* peer_rank, const int32_t* peer_token_idx,
                                        const int32_t* num_rows, int max_rows, int row_begin, int row_end, int64_t hidden,
                                        const float* row_values, const uint64_t* value_ptrs_host, int blocks,
                                        const int32_t* wait_counter, int arrivals_per_row_block, int32_t* status,
                                        int64_t index_limit, void* stream) {
    return combine_rows_impl(src, dst_ptrs_host, ep_size, peer_rank, peer_token_idx, num_rows, max_rows, row_begin, row_end, hidden,
                             row_values, value_ptrs_host, blocks, static_cast<cudaStream_t>(stream), wait_counter,
                             arrivals_per_row_block, status, index_limit);
}
