// Key-search kernels for sm_100a. See kernels.cuh for the schemes and the
// candidate numbering; field.cuh for the arithmetic.
#include <algorithm>

#include "field.cuh"
#include "kernels.cuh"
#include "search_common.cuh"
#include "suffix_match.cuh"

// Register budget of the search kernels: at most OG_LB_THREADS threads per
// block and at least OG_LB_MIN_BLOCKS resident blocks per SM. 128 x 4 gives
// them 128 registers (16 warps per SM); the paired kernel ran 52.6 ms a launch
// of 3.1e9 candidates so, 54.3 at 96 registers (20 warps), 56.0 at 168.
#ifndef OG_LB_THREADS
#define OG_LB_THREADS 128
#endif
#ifndef OG_LB_MIN_BLOCKS
#define OG_LB_MIN_BLOCKS 4
#endif
// with two blocks of lanes an item: the blocks per SM of its launches
#ifndef OG_LB2_MIN_BLOCKS
#define OG_LB2_MIN_BLOCKS 4
#endif

namespace og {

namespace {

__global__ void __launch_bounds__(128) init_kernel(const InitArgs a) {
    const uint32_t lane = blockIdx.x * blockDim.x + threadIdx.x;
    if (lane >= a.lanes_n) return;
    const size_t L = a.lanes_n;
    fe X = words_fe(a.bx), Y = words_fe(a.by), Z = words_fe(a.bz), T = words_fe(a.bt);
    for (uint32_t k = 0; k < a.nbits; k++) {
        if ((lane >> k) & 1u) {
            const uint4* p = a.pow2 + (size_t)k * 6;
            const fe ypx = load_fe(p + 0, 1), ymx = load_fe(p + 2, 1), t2d = load_fe(p + 4, 1);
            add_cached(X, Y, Z, T, ypx, ymx, t2d);
        }
    }
    if (a.affine_out) {
        const fe zi = fe_invert(Z);
        store_fe(a.lanes + 0 * L + lane, L, fe_mulv(X, zi));
        store_fe(a.lanes + 2 * L + lane, L, fe_mulv(Y, zi));
    } else {
        store_fe(a.lanes + 0 * L + lane, L, X);
        store_fe(a.lanes + 2 * L + lane, L, Y);
        store_fe(a.lanes + 4 * L + lane, L, Z);
        store_fe(a.lanes + 6 * L + lane, L, T);
    }
}

// The paired search, bound by the multiply-add pipe. Persistent: each CTA
// takes the next PerItem blocks of lanes until none is left; its scratch
// belongs to the CTA, not the lanes. On B200 at half 2048, 757 760 lanes and
// one 6-symbol prefix a launch takes 52.6 ms (5.9e10 keys/s); ten
// multiplications a pair took 147.
// Narrow: a prefix bitmap of at most 24 bits (sink_is_narrow).
template <int PerItem, bool Narrow>
__global__ void __launch_bounds__(OG_LB_THREADS, PerItem == 2 ? OG_LB2_MIN_BLOCKS : OG_LB_MIN_BLOCKS)
    paired_kernel(const PairedArgs a) {
    __shared__ uint32_t item_s;
    const size_t L = a.lanes_n;
    constexpr uint32_t per_item = OG_LB_THREADS * PerItem;
    const uint32_t nitems = (a.lanes_n + per_item - 1) / per_item;
    const Sink sink{a.bitmap, a.bits, a.hits, a.counter, a.cap, a.search, a.sbitmap, a.sbits, false, a.failed};
    const PairTable tab = pair_table_at(a.table, a.half);
    uint4* const scr = a.scratch + (size_t)blockIdx.x * cta_scratch_uint4(a.half) + threadIdx.x;
    MatrixUnit mu;
    RoundShared* sh = nullptr;
    if constexpr (Narrow) {
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
#pragma unroll 1
        for (uint32_t k = 0; k < PerItem; k++) {
            const uint32_t lane = item * per_item + k * OG_LB_THREADS + threadIdx.x;
            const bool active = lane < a.lanes_n;
            uint4* const centre = a.lanes + (active ? lane : 0);
            if constexpr (Narrow)
                paired_rounds<true>(centre, L, a.wx, a.wy, a.wdt, tab, a.half, a.rounds, scr, sink, *sh, mu, lane, active);
            else
                paired_rounds_full<true>(centre, L, a.wx, a.wy, a.wdt, tab, a.half, a.rounds, scr, sink, lane, active);
        }
    }
    if constexpr (Narrow) matrix_close(*sh);
}

// The per-group part of a PairTable whose q, v and s are in place.
__global__ void __launch_bounds__(128) group_table_kernel(uint4* table, uint32_t half) {
    fill_group_table(pair_table_at(table, half), groups_of(half), blockIdx.x * blockDim.x + threadIdx.x);
}

// The chain kernel (the config-1 contract) keeps 96 registers: at 80 it
// spills. Persistent like the paired kernel: each CTA takes the next block
// of lanes until none is left, and the scratch is indexed by the CTA's
// slot, so any number of waves of lanes costs the scratch of one. A prefix
// bitmap of up to 16 bits (8 KiB) is staged in shared memory per CTA and
// tested there: 9.445e9 against 9.355e9 keys/s on B200 for config 2's index
// at n = 1024. (The paired kernel reads the table Q_m through L1, and the
// 8 KiB more a block cost it more than the bitmap read saves, so it keeps
// the map in global memory.) The scratch is one region per CTA whose rows
// hold the CTA's threads, so that a CTA's accesses stay within a few pages:
// 9.57e9 against 9.49e9 keys/s with rows across the whole grid.
__global__ void __launch_bounds__(OG_LB_THREADS, 5) chain_kernel(const ChainArgs a) {
    static_assert(CHAIN_ROW >= OG_LB_THREADS, "a row holds every thread of a block");
    __shared__ uint32_t item_s;
    const size_t L = a.lanes_n;
    const uint32_t nblocks = a.lanes_n / blockDim.x;
    const bool staged = a.bitmap && a.bits <= STAGED_BITMAP_BITS;
    const Sink sink{a.bitmap, a.bits, a.hits, a.counter, a.cap, a.search, a.sbitmap, a.sbits, staged};
    if (staged) {
        extern __shared__ uint32_t og_bitmap_s[];
        const uint32_t words = (1u << a.bits) / 32u;
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) og_bitmap_s[i] = a.bitmap[i];
        // the loop's first barrier orders these stores before any test
    }
    uint4* const scr = a.scratch + (size_t)blockIdx.x * (CHAIN_ROW * 4) * a.n + threadIdx.x;
#define SCR(e, w) (scr + ((size_t)(e) * 4 + (w) * 2) * CHAIN_ROW)
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) item_s = atomicAdd(a.work, 1u);
        __syncthreads();
        const uint32_t item = item_s;
        if (item >= nblocks) break;
        const uint32_t lane = item * blockDim.x + threadIdx.x;
        fe X = load_fe(a.lanes + 0 * L + lane, L);
        fe Y = load_fe(a.lanes + 2 * L + lane, L);
        fe Z = load_fe(a.lanes + 4 * L + lane, L);
        fe T = load_fe(a.lanes + 6 * L + lane, L);
        for (uint32_t r = 0; r < a.rounds; r++) {
            fe run = fe_one();
#pragma unroll 1
            for (uint32_t t = 0; t < a.n; t++) {
                store_fe(SCR(t, 0), CHAIN_ROW, fe_mulv(Y, run));
                store_fe(SCR(t, 1), CHAIN_ROW, Z);
                run = fe_mulv(run, Z);
                add_cached(X, Y, Z, T, words_fe(a.step_ypx), words_fe(a.step_ymx), words_fe(a.step_t2d));
            }
            if (L > 1) add_cached(X, Y, Z, T, words_fe(a.jump_ypx), words_fe(a.jump_ymx), words_fe(a.jump_t2d));
            fe acc = block_invert(run);  // one inversion for the block's lanes
            const uint32_t base_step = r * a.n;
#pragma unroll 1
            for (uint32_t t = a.n; t-- > 0;) {
                const fe v = fe_mulv(load_fe(SCR(t, 0), CHAIN_ROW), acc);
                acc = fe_mulv(acc, load_fe(SCR(t, 1), CHAIN_ROW));
                test_emit(sink, v, lane, base_step + t);
            }
        }
        store_fe(a.lanes + 0 * L + lane, L, X);
        store_fe(a.lanes + 2 * L + lane, L, Y);
        store_fe(a.lanes + 4 * L + lane, L, Z);
        store_fe(a.lanes + 6 * L + lane, L, T);
    }
#undef SCR
}

// The filter a suffix-bitmap survivor matches (suffix_match), with the
// survivor's scalar offset over 8 decoded from its record.
__device__ __noinline__ uint32_t suffix_owner(const MatchArgs& a, const HitRec& r) {
    const uint64_t w = a.window0 + (uint64_t)(r.step / a.slots) * a.lanes + r.lane;
    const uint64_t k = w * a.slots + (a.paired ? 1u : 0u) + r.step % a.slots;
    const SuffixTables t{a.suffixes, a.nsuffix, a.pow8};
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
            fe y;
#pragma unroll
            for (int q = 0; q < 8; q++) y.v[q] = r.y[q];
            const uint32_t slot = suffix_slot(y, a.sbits);
            if ((__ldg(a.sbitmap + (slot >> 5)) >> (slot & 31)) & 1u) owner = suffix_owner(a, r);
        }
        if (owner != 0xffffffffu) {
            const uint32_t idx = atomicAdd(a.out_count, 1u);
            if (idx < a.out_cap) {
                // window w = window0 + round * lanes + lane; candidate i of it
                const uint64_t w = a.window0 + (uint64_t)(r.step / a.slots) * a.lanes + r.lane;
                const uint64_t k = w * a.slots + (a.paired ? 1u : 0u) + r.step % a.slots;
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

cudaError_t launch_init(const InitArgs& a, int block, cudaStream_t s) {
    const unsigned grid = (a.lanes_n + block - 1) / block;
    init_kernel<<<grid, block, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_paired(const PairedArgs& a, int grid, cudaStream_t s) {
    const uint32_t n = a.lanes_per_thread;
    constexpr int block = OG_LB_THREADS;
    if ((n != 1 && n != 2) || grid <= 0) return cudaErrorInvalidValue;
    const bool narrow = sink_is_narrow(a.bitmap != nullptr, a.bits, a.sbitmap != nullptr);
    if (n == 2 && narrow)
        paired_kernel<2, true><<<grid, block, 0, s>>>(a);
    else if (n == 2)
        paired_kernel<2, false><<<grid, block, 0, s>>>(a);
    else if (narrow)
        paired_kernel<1, true><<<grid, block, 0, s>>>(a);
    else
        paired_kernel<1, false><<<grid, block, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_group_table(uint4* table, uint32_t half, cudaStream_t s) {
    group_table_kernel<<<(groups_of(half) * 48 + 127) / 128, 128, 0, s>>>(table, half);
    return cudaGetLastError();
}

cudaError_t launch_chain(const ChainArgs& a, int block, int grid, cudaStream_t s) {
    if (a.lanes_n % block != 0 || block % 32 != 0 || grid < 1 || (uint32_t)grid * block != a.slots_n)
        return cudaErrorInvalidValue;
    const size_t smem = (a.bitmap && a.bits <= STAGED_BITMAP_BITS) ? (size_t)(1u << a.bits) / 8u : 0;
    chain_kernel<<<grid, block, smem, s>>>(a);
    return cudaGetLastError();
}

static cudaError_t info_of(const void* fn, int block, size_t smem, KernelInfo* info) {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, fn);
    if (e != cudaSuccess) return e;
    info->regs = attr.numRegs;
    info->max_threads = attr.maxThreadsPerBlock;
    info->local_bytes = attr.localSizeBytes;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&info->blocks_per_sm, fn, block, smem);
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

cudaError_t paired_info(bool narrow, uint32_t lanes_per_thread, KernelInfo* info) {
    const void* const fn[2][2] = {{(const void*)paired_kernel<1, false>, (const void*)paired_kernel<1, true>},
                                  {(const void*)paired_kernel<2, false>, (const void*)paired_kernel<2, true>}};
    const void* const f = fn[lanes_per_thread == 2][narrow];
    const cudaError_t e = info_of(f, OG_LB_THREADS, 0, info);
    return e == cudaSuccess && narrow ? matrix_blocks_per_sm(f, 0, &info->blocks_per_sm) : e;
}

// sized for a staged 16-bit bitmap, the most a chain launch takes
cudaError_t chain_info(int block, KernelInfo* info) {
    return info_of((const void*)chain_kernel, block, (size_t)(1u << STAGED_BITMAP_BITS) / 8u, info);
}

}  // namespace og
