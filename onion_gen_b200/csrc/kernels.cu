// Key-search kernels for sm_100a. See kernels.cuh for the schemes and the
// candidate numbering; field.cuh for the arithmetic.
#include <algorithm>

#include "field.cuh"
#include "kernels.cuh"
#include "search_common.cuh"
#include "suffix_match.cuh"

// Register budget of the search kernels: at most OG_LB_THREADS threads per
// block and at least OG_LB_MIN_BLOCKS resident blocks per SM. 128 x 4 gives
// them 128 registers (16 warps per SM); the paired kernel runs 49.9 ms a launch
// of 3.1e9 candidates so, 51.9 at 96 registers (20 warps) and 51.9 at 168 (12);
// 9.7e7 candidates 1.74, 1.86 and 1.75. ptxas reports 244 bytes of spill stores
// and 120 of loads at 128.
#ifndef OG_LB_MIN_BLOCKS
#define OG_LB_MIN_BLOCKS 4
#endif

namespace og {

namespace {

__global__ void __launch_bounds__(OG_LB_THREADS) init_kernel(const InitArgs a, const Pow2Table stride) {
    first_centre(words_fe(a.bx), words_fe(a.by), words_fe(a.bz), words_fe(a.bt), stride,
                 blockIdx.x * blockDim.x + threadIdx.x, a.lanes, a.lanes_n);
}

// The search, bound by the multiply-add pipe. Persistent: each CTA takes the
// next block of lanes until none is left; its scratch belongs to the CTA, not
// the lanes. On B200 at half 2048, 757 760 lanes and one 6-symbol prefix a
// launch takes 49.9 ms (6.2e10 keys/s); ten multiplications a pair took 147.
template <SinkKind Kind>
__global__ void __launch_bounds__(OG_LB_THREADS, OG_LB_MIN_BLOCKS) paired_kernel(const PairedArgs a) {
    __shared__ uint32_t item_s;
    const size_t L = a.lanes_n;
    const uint32_t nitems = (a.lanes_n + OG_LB_THREADS - 1) / OG_LB_THREADS;
    const Sink sink{a.bitmap, a.bits,   a.hits,  a.counter, a.cap,     a.search,          a.sbitmap,
                    a.sbits,  a.failed, a.limit, a.lanes_n, 2 * a.half + 1};
    const PairTable tab = pair_table_at(a.table, a.half);
    uint4* const scr = a.scratch + (size_t)blockIdx.x * cta_scratch_uint4(a.half, Kind) + threadIdx.x;
    MatrixUnit mu;
    RoundShared* sh = nullptr;
    if constexpr (Kind != SINK_FULL) {
        __shared__ __align__(128) RoundShared shared;
        sh = &shared;
        matrix_open(*sh);
    }
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) item_s = atomicAdd(a.work, 1u);
        __syncthreads();
        const uint32_t item = item_s;
        if (item >= nitems) break;
        const uint32_t lane = item * OG_LB_THREADS + threadIdx.x;
        const bool active = lane < a.lanes_n;
        uint4* const centre = a.lanes + (active ? lane : 0);
        if constexpr (Kind != SINK_FULL)
            paired_rounds<Kind == SINK_SUFFIX, true, false>(centre, L, a.between, a.last, tab, a.half, a.rounds, scr, sink,
                                                      *sh, mu, lane, active);
        else
            paired_rounds_full<true>(centre, L, a.between, a.last, tab, a.half, a.rounds, scr, sink, lane, active);
    }
    if constexpr (Kind != SINK_FULL) matrix_close(*sh);
}

// The per-entry part of a PairTable.
__global__ void __launch_bounds__(OG_LB_THREADS) pair_entry_kernel(uint4* table, uint32_t half, const Pow2Table eight) {
    fill_pair_entry(pair_table_at<const uint4>(table, half), groups_of(half) * GROUP, eight,
                    blockIdx.x * blockDim.x + threadIdx.x);
}

// The per-group part of a PairTable whose q, v and s are in place.
__global__ void __launch_bounds__(128) group_table_kernel(uint4* table, uint32_t half) {
    fill_group_table(pair_table_at(table, half), groups_of(half), blockIdx.x * blockDim.x + threadIdx.x);
}

// The filter a suffix-bitmap survivor matches (suffix_match), with the
// survivor's scalar offset over 8 decoded from its record.
__device__ __noinline__ uint32_t suffix_owner(const MatchArgs& a, const HitRec& r) {
    const uint64_t k = a.first + (((uint64_t)r.step << 32) | r.lane);
    const SuffixTables t{a.suffixes, a.nsuffix, a.mul8};
    bool bad = false;
    const uint32_t j = suffix_match(t, a.sx, a.sy, a.sz, a.st, k, r.y, bad);
    if (bad) atomicAdd(a.mismatch, 1u);
    return j == 0xffffffffu ? j : a.prefix_count + j;
}

// Exact match of one advance's bitmap survivors (grid-stride; the survivor
// count is read on the device, so the launch needs no host round trip).
__global__ void __launch_bounds__(128) match_kernel(const MatchArgs a) {
    const uint32_t n = min(*a.surv_count, a.surv_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const HitRec r = a.surv[i];
        uint32_t owner = (a.t.nbuckets || a.t.npatterns) ? exact_owner(a.t, r.y) : 0xffffffffu;
        if (owner == 0xffffffffu && a.sbitmap) {
            const uint32_t slot = suffix_slot(r.y[6], r.y[7], a.sbits);
            if ((__ldg(a.sbitmap + (slot >> 5)) >> (slot & 31)) & 1u) owner = suffix_owner(a, r);
        }
        if (owner != 0xffffffffu) {
            const uint32_t idx = atomicAdd(a.out_count, 1u);
            if (idx < a.out_cap) {
                const uint64_t k = a.first + (((uint64_t)r.step << 32) | r.lane);
                uint4* dst = reinterpret_cast<uint4*>(a.out + idx);
                dst[0] = make_uint4((uint32_t)(8 * k), (uint32_t)((8 * k) >> 32), r.y[0], r.y[1]);
                dst[1] = make_uint4(r.y[2], r.y[3], r.y[4], r.y[5]);
                dst[2] = make_uint4(r.y[6], r.y[7], owner, 0u);
            }
        }
    }
}

}  // namespace

cudaError_t launch_match(const MatchArgs& a, int grid, cudaStream_t s) {
    match_kernel<<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_init(const InitArgs& a, const Pow2Table& stride, cudaStream_t s) {
    init_kernel<<<(a.lanes_n + OG_LB_THREADS - 1) / OG_LB_THREADS, OG_LB_THREADS, 0, s>>>(a, stride);
    return cudaGetLastError();
}

cudaError_t launch_paired(const PairedArgs& a, SinkKind kind, int grid, cudaStream_t s) {
    if (grid <= 0) return cudaErrorInvalidValue;
    if (kind == SINK_PREFIX)
        paired_kernel<SINK_PREFIX><<<grid, OG_LB_THREADS, 0, s>>>(a);
    else if (kind == SINK_SUFFIX)
        paired_kernel<SINK_SUFFIX><<<grid, OG_LB_THREADS, 0, s>>>(a);
    else
        paired_kernel<SINK_FULL><<<grid, OG_LB_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pair_table(uint4* table, uint32_t half, const Pow2Table& eight, cudaStream_t s) {
    pair_entry_kernel<<<(groups_of(half) * GROUP + OG_LB_THREADS - 1) / OG_LB_THREADS, OG_LB_THREADS, 0, s>>>(table, half, eight);
    group_table_kernel<<<(groups_of(half) * 36 + 127) / 128, 128, 0, s>>>(table, half);
    return cudaGetLastError();
}

cudaError_t matrix_blocks_per_sm(const void* fn, size_t smem, int* blocks) {
    cudaFuncAttributes attr;
    int device = 0, regs = 0, shared = 0, reserved = 0;
    cudaError_t e = cudaFuncGetAttributes(&attr, fn);
    if (e == cudaSuccess) e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&regs, cudaDevAttrMaxRegistersPerMultiprocessor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&shared, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
    if (e != cudaSuccess) return e;
    const int warp_regs = (attr.numRegs * 32 + 255) / 256 * 256;  // allocated 256 at a time
    const size_t block_shared = (attr.sharedSizeBytes + smem + reserved + 127) / 128 * 128;
    *blocks = std::min({regs / (warp_regs * (OG_LB_THREADS / 32)), (int)(shared / block_shared),
                        (int)(512 / TMEM_COLUMNS)});
    return cudaSuccess;
}

cudaError_t paired_blocks_per_sm(SinkKind kind, int* blocks) {
    if (kind == SINK_PREFIX) return matrix_blocks_per_sm((const void*)paired_kernel<SINK_PREFIX>, 0, blocks);
    if (kind == SINK_SUFFIX) return matrix_blocks_per_sm((const void*)paired_kernel<SINK_SUFFIX>, 0, blocks);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, paired_kernel<SINK_FULL>, OG_LB_THREADS, 0);
}

}  // namespace og
