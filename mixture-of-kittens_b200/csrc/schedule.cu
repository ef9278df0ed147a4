// Routing schedule builder.
//
// Produces exactly the schedule of the reference (csrc/scheduler.cuh:35-147):
// per-expert segments padded to 256 rows, and inside a segment the routes of
// the R source ranks interleaved round-robin, where the j-th route of a
// (rank, expert) pair is counted in the order in which a 1024-thread block
// strides over that rank's route list (thread index first, then iteration).
//
// The reference launches E_l*R blocks that each re-read one rank's whole route
// list twice.  Here two launches of about 128 blocks do it:
//   view a rank's routes as a matrix [iteration][1024 threads]; the reference
//   order is column-major over that matrix.  A block owns a contiguous range of
//   columns, i.e. a contiguous range of the order.
//   1. count : every block histograms its routes by local expert.
//   2. place : every block adds up all blocks' histograms (totals per rank and
//              expert, and what the blocks before it hold), scans the padded
//              totals into segment bases, ranks its routes -- a warp takes 32 in
//              order at a time, lanes of the same expert are ranked by a vote --
//              and writes each one's row with the closed form of
//              scheduler.cuh:134-139.  Rows without a route are written by the
//              same launch, so nothing is cleared beforehand.
// Bound by latency (about 1 MB moves): what counts is the number of dependent launches and
// round trips: 14 us for 131072 routes over 32 experts, 7 us for 2048 over 8.  (As three clears and four kernels
// with a scan of per-thread counters in memory: 38 and 16 us.)
#include "common.cuh"

namespace mokb {
namespace {

constexpr int kThreadsOrder = 1024;   // the reference's block size, which defines the order
constexpr int kPad = 256;             // expert segment padding
constexpr int kSchedThreads = 512;
constexpr int kSchedWarps = kSchedThreads / 32;
constexpr int kMaxColumnBlocks = 128;

struct SchedParams {
    const int32_t* topk_all;  // [R, routes]
    int R, routes, E_l, C, rank;
    int NB;                   // blocks per rank: a power of two; each owns 1024 / NB columns
    int P;                    // ceil(routes / 1024): rows of the matrix
    int32_t* blkcnt;          // [R, NB, E_l]
    int32_t* peer_rank;
    int32_t* peer_token_idx;
    int32_t* num_tokens;
    int32_t* tokens_per_expert;
    int32_t* status;
};

__global__ void __launch_bounds__(kSchedThreads) count_kernel(SchedParams p) {
    extern __shared__ int32_t hist[];     // [E_l]
    const int t = threadIdx.x, r = blockIdx.y, b = blockIdx.x;
    for (int e = t; e < p.E_l; e += kSchedThreads) hist[e] = 0;
    __syncthreads();
    const uint32_t cols = kThreadsOrder / p.NB, c0 = b * cols, shift = 31 - __clz(cols);
    const int first = p.rank * p.E_l;
    const int32_t* routes = p.topk_all + static_cast<size_t>(r) * p.routes;
    const uint32_t items = p.P * cols;           // any order will do here: row by row
#pragma unroll 4
    for (uint32_t i = t; i < items; i += kSchedThreads) {
        const uint32_t idx = (i >> shift) * kThreadsOrder + c0 + (i & (cols - 1));
        if (idx < static_cast<uint32_t>(p.routes)) {
            const int e = __ldg(routes + idx) - first;
            if (e >= 0 && e < p.E_l) atomicAdd(&hist[e], 1);
        }
    }
    __syncthreads();
    int32_t* out = p.blkcnt + (static_cast<size_t>(r) * p.NB + b) * p.E_l;
    for (int e = t; e < p.E_l; e += kSchedThreads) out[e] = hist[e];
}

__global__ void __launch_bounds__(kSchedThreads) place_kernel(SchedParams p) {
    extern __shared__ int32_t sm[];
    int32_t* const tot = sm;                              // [R][E_l]  routes of a rank to an expert
    int32_t* const ctr = tot + p.R * p.E_l;               // [warps][E_l]
    int32_t* const before = ctr + kSchedWarps * p.E_l;    // [E_l]     routes of this rank in the blocks before this one
    int32_t* const base = before + p.E_l;                 // [E_l + 1] first row of a segment
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, r = blockIdx.y, b = blockIdx.x;
    const int E_l = p.E_l, first = p.rank * E_l;
    for (int i = t; i < (p.R + kSchedWarps + 1) * E_l; i += kSchedThreads) sm[i] = 0;
    __syncthreads();

    for (int rr = 0; rr < p.R; ++rr) {
        const int32_t* c = p.blkcnt + static_cast<size_t>(rr) * p.NB * E_l;
        const int n = p.NB * E_l, mine = rr == r ? b * E_l : 0;     // entries below `mine`: earlier blocks of this rank
#pragma unroll 4
        for (int i = t; i < n; i += kSchedThreads) {
            const int v = __ldg(c + i);
            if (v) {
                const int e = i % E_l;
                atomicAdd(&tot[rr * E_l + e], v);
                if (i < mine) atomicAdd(&before[e], v);
            }
        }
    }
    // this block's part of the order, a contiguous piece of it per warp
    const uint32_t cols = kThreadsOrder / p.NB, c0 = b * cols, P = p.P;
    const int32_t* routes = p.topk_all + static_cast<size_t>(r) * p.routes;
    const uint32_t items = P * cols;             // at most routes + 1023 * cols, routes < 2^31
    const uint32_t per_warp = (items + kSchedThreads - 1) / kSchedThreads * 32;
    const uint32_t l0 = warp * per_warp, l1 = min(l0 + per_warp, items);
    auto expert_of = [&](uint32_t l, int* index) {          // position in the order -> local expert, or -1
        const uint32_t cc = l / P;
        const uint32_t idx = (l - cc * P) * kThreadsOrder + c0 + cc;
        *index = static_cast<int>(idx);
        if (l >= l1 || idx >= static_cast<uint32_t>(p.routes)) return -1;
        const int e = __ldg(routes + idx) - first;
        return e >= 0 && e < E_l ? e : -1;
    };
    int index;
    for (uint32_t l = l0 + lane; l < l1; l += 32) {
        const int e = expert_of(l, &index);
        if (e >= 0) atomicAdd(&ctr[warp * E_l + e], 1);
    }
    __syncthreads();

    if (warp == 0) {          // segment bases: exclusive scan of the padded totals
        int carry = 0;
        for (int e0 = 0; e0 < E_l; e0 += 32) {
            const int e = e0 + lane;
            int padded = 0;
            if (e < E_l) {
                int n = 0;
                for (int rr = 0; rr < p.R; ++rr) n += tot[rr * E_l + e];
                padded = (n + kPad - 1) / kPad * kPad;
                if (b == 0 && r == 0) p.tokens_per_expert[e] = padded;
            }
            int inc = padded;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (e < E_l) base[e] = carry + inc - padded;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) {
            base[E_l] = carry;
            if (b == 0 && r == 0) {
                p.num_tokens[0] = carry;
                if (carry > p.C) atomicCAS(p.status, MOKB_ST_OK, MOKB_ST_SCHEDULE_OVERFLOW);
            }
        }
    } else {                  // where each warp's routes of an expert start counting
        for (int e = t - 32; e < E_l; e += kSchedThreads - 32) {
            int run = before[e];
            for (int w = 0; w < kSchedWarps; ++w) {
                const int n = ctr[w * E_l + e];
                ctr[w * E_l + e] = run;
                run += n;
            }
        }
    }
    __syncthreads();

    // rows without a route: all of them if the schedule does not fit, otherwise the end of every segment and of the arrays
    const int total = base[E_l];
    const bool overflow = total > p.C;
    const int block = r * p.NB + b, nblocks = p.NB * p.R;
    for (int64_t i = (overflow ? 0 : total) + static_cast<int64_t>(block) * kSchedThreads + t; i < p.C; i += static_cast<int64_t>(nblocks) * kSchedThreads)
        p.peer_rank[i] = p.peer_token_idx[i] = -1;
    if (overflow) return;
    for (int e = block * kSchedWarps + warp; e < E_l; e += nblocks * kSchedWarps) {
        int n = 0;
        for (int rr = 0; rr < p.R; ++rr) n += tot[rr * E_l + e];
        for (int i = base[e] + n + lane; i < base[e + 1]; i += 32) p.peer_rank[i] = p.peer_token_idx[i] = -1;
    }

    int32_t* const count = ctr + warp * E_l;
    for (uint32_t lb = l0; lb < l1; lb += 32) {            // whole warp: the same number of trips in every lane
        const int e = expert_of(lb + lane, &index);
        const unsigned same = __match_any_sync(0xffffffffu, e);
        int j = 0;
        if (e >= 0) j = count[e] + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (e >= 0 && lane == 31 - __clz(same)) count[e] = j + 1;
        __syncwarp();
        if (e >= 0) {
            int dst = base[e];
            for (int rr = 0; rr < p.R; ++rr) {
                const int n = tot[rr * E_l + e];
                dst += min(n, j) + ((rr < r && n > j) ? 1 : 0);
            }
            p.peer_rank[dst] = r;
            p.peer_token_idx[dst] = index;
        }
    }
}

// Blocks: about 128 over all ranks, fewer where the histograms that every block of the second launch adds up would
// otherwise exceed 16384 words (32 per thread).
int launch_schedule(SchedParams p, cudaStream_t stream) {
    const int E = p.R * p.E_l;
    p.P = (p.routes + kThreadsOrder - 1) / kThreadsOrder;
    p.NB = kMaxColumnBlocks;
    while (p.NB > 1 && (p.NB * p.R > kMaxColumnBlocks || static_cast<int64_t>(p.NB) * E > 16384)) p.NB /= 2;
    const size_t smem = (static_cast<size_t>(E) + static_cast<size_t>(kSchedWarps + 2) * p.E_l + 1) * 4;
    if (smem > 48 * 1024) MOKB_CUDA(cudaFuncSetAttribute(place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    const dim3 grid(static_cast<unsigned>(p.NB), static_cast<unsigned>(p.R));
    count_kernel<<<grid, kSchedThreads, static_cast<size_t>(p.E_l) * 4, stream>>>(p);
    place_kernel<<<grid, kSchedThreads, smem, stream>>>(p);
    MOKB_CUDA(cudaGetLastError());
    note_launch(2);
    return MOKB_OK;
}

}  // namespace
}  // namespace mokb

using namespace mokb;

extern "C" size_t mokb_schedule_scratch_bytes(int ep_size, int num_local_experts) {
    // an upper bound with room to spare (the histograms take at most a 64th of it); callers may have been sized by it
    return static_cast<size_t>(ep_size) * num_local_experts * (kThreadsOrder * 8 + 2) * 4;
}

extern "C" int mokb_schedule(const int32_t* topk_all, int ep_size, int num_local_tokens, int topk,
                             int num_local_experts, int schedule_capacity, int rank,
                             int32_t* peer_rank, int32_t* peer_token_idx, int32_t* num_tokens,
                             int32_t* tokens_per_expert, void* scratch, int32_t* status, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    TraceScope trace(stream, "schedule");
    MOKB_REQUIRE(topk_all && peer_rank && peer_token_idx && num_tokens && tokens_per_expert && scratch && status,
                 "schedule: null pointer");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP, "schedule: ep_size %d out of range", ep_size);
    MOKB_REQUIRE(rank >= 0 && rank < ep_size, "schedule: rank %d not in [0, %d)", rank, ep_size);
    MOKB_REQUIRE(num_local_tokens > 0 && topk > 0 && num_local_experts > 0, "schedule: sizes must be positive");
    MOKB_REQUIRE(schedule_capacity > 0 && schedule_capacity % kPad == 0, "schedule: capacity must be a positive multiple of 256");
    const long long routes_ll = 1LL * num_local_tokens * topk;
    MOKB_REQUIRE(routes_ll * ep_size < (1LL << 31), "schedule: too many routes");
    MOKB_REQUIRE(static_cast<size_t>(num_local_experts) * 32 * 4 <= 160 * 1024, "schedule: too many local experts");

    SchedParams p;
    p.topk_all = topk_all;
    p.R = ep_size; p.routes = static_cast<int>(routes_ll); p.E_l = num_local_experts;
    p.C = schedule_capacity; p.rank = rank;
    p.blkcnt = static_cast<int32_t*>(scratch);
    p.peer_rank = peer_rank; p.peer_token_idx = peer_token_idx;
    p.num_tokens = num_tokens; p.tokens_per_expert = tokens_per_expert; p.status = status;
    return launch_schedule(p, stream);
}

// ---------------------------------------------------------------------------
// Routing schedule for callers that must not allocate device memory.
//
// Some hosts of this library run where cudaMalloc is off limits: inside a
// framework that owns the whole device heap through its own pool, in a
// latency-critical step loop where an allocation would serialise the device,
// or in a process that pre-commits all memory at start-up.  For them the work
// area of the schedule builder lives in the library image itself: a fixed
// __device__ array that every GPU loading the library carries until exit.
// The price is a size limit and shared state (see the header).
namespace mokb {
namespace {

// the histograms of every block of the first launch, for the most experts that this entry point takes
constexpr size_t kStaticSchedBytes = static_cast<size_t>(MOKB_SCHEDULE_NOALLOC_MAX_EXPERTS) * kMaxColumnBlocks * 4;
static __device__ __align__(256) unsigned char g_static_sched_scratch[kStaticSchedBytes];

// Device address of the array above, per device.  In host code the array's name is only a
// handle for the runtime; the address a kernel can use comes from cudaGetSymbolAddress,
// asked for with that device current.
void* g_static_sched_ptr[64] = {nullptr};

int static_sched_scratch(void** out) {
    int dev = -1;
    MOKB_CUDA(cudaGetDevice(&dev));
    MOKB_REQUIRE(dev >= 0 && dev < 64, "schedule_noalloc: device index %d out of range", dev);
    if (g_static_sched_ptr[dev] == nullptr) {
        void* p = nullptr;
        MOKB_CUDA(cudaGetSymbolAddress(&p, g_static_sched_scratch));
        MOKB_REQUIRE(p != nullptr, "schedule_noalloc: cudaGetSymbolAddress returned a null address");
        g_static_sched_ptr[dev] = p;
    }
    *out = g_static_sched_ptr[dev];
    return MOKB_OK;
}

}  // namespace
}  // namespace mokb

extern "C" int mokb_schedule_noalloc(const int32_t* topk_all, int ep_size, int num_local_tokens, int topk,
                                     int num_local_experts, int schedule_capacity, int rank,
                                     int32_t* peer_rank, int32_t* peer_token_idx, int32_t* num_tokens,
                                     int32_t* tokens_per_expert, int32_t* status, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    MOKB_REQUIRE(topk_all && peer_rank && peer_token_idx && num_tokens && tokens_per_expert && status,
                 "schedule_noalloc: null pointer");
    MOKB_REQUIRE(ep_size >= 1 && ep_size <= MOKB_MAX_EP, "schedule_noalloc: ep_size %d out of range", ep_size);
    MOKB_REQUIRE(rank >= 0 && rank < ep_size, "schedule_noalloc: rank %d not in [0, %d)", rank, ep_size);
    MOKB_REQUIRE(num_local_tokens > 0 && topk > 0 && num_local_experts > 0, "schedule_noalloc: sizes must be positive");
    MOKB_REQUIRE(schedule_capacity > 0 && schedule_capacity % kPad == 0,
                 "schedule_noalloc: capacity must be a positive multiple of 256");
    const long long routes_ll = 1LL * num_local_tokens * topk;
    MOKB_REQUIRE(routes_ll * ep_size < (1LL << 31), "schedule_noalloc: too many routes");
    const size_t E = static_cast<size_t>(ep_size) * num_local_experts;
    MOKB_REQUIRE(E <= MOKB_SCHEDULE_NOALLOC_MAX_EXPERTS,
                 "schedule_noalloc: ep_size * num_local_experts = %zu exceeds the built-in work area's limit of %d experts; "
                 "use mokb_schedule with caller-provided scratch", E, MOKB_SCHEDULE_NOALLOC_MAX_EXPERTS);
    MOKB_REQUIRE(static_cast<size_t>(num_local_experts) * 32 * 4 <= 160 * 1024, "schedule_noalloc: too many local experts");

    void* scratch = nullptr;
    MOKB_TRY(static_sched_scratch(&scratch));

    SchedParams p;
    p.topk_all = topk_all;
    p.R = ep_size; p.routes = static_cast<int>(routes_ll); p.E_l = num_local_experts;
    p.C = schedule_capacity; p.rank = rank;
    // the area keeps whatever the previous call left; every word that is read is written by this call's first launch
    p.blkcnt = static_cast<int32_t*>(scratch);
    p.peer_rank = peer_rank; p.peer_token_idx = peer_token_idx;
    p.num_tokens = num_tokens; p.tokens_per_expert = tokens_per_expert; p.status = status;
    return launch_schedule(p, stream);
}
