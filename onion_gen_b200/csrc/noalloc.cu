// og_search_noalloc: the paired search without any device allocation.
//
// Some callers cannot allocate device memory: code running inside another
// framework's memory pool that forbids cudaMalloc behind its back, callers
// that must not synchronise the device (cudaMalloc and cudaFree can), and
// processes that reserve all device memory up front. This entry point lets
// them run the search: they pass the inputs (start point, bitmap) and the
// outputs (survivor records and their counter) in device memory they own,
// and everything else — lane state, the rounds' products and the tables —
// lives in one file-scope device array, `og_noalloc_scratch`, sized
// OG_NOALLOC_SCRATCH_BYTES. Every GPU that loads the library holds that array
// until the process exits.
//
// Host code must not use the array's name as a device address (in host code
// it is a host-side stand-in); it takes the address once per device with
// cudaGetSymbolAddress, on the first call made on that device, and passes it
// to the kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/onion_gen_b200.h"
#include "host/common.h"
#include "search_common.cuh"

namespace og {

Stride stride_of(const Pt& w);    // engine.cu
Pow2Table pow2_table(Pt p);       // engine.cu
const Pow2Table& powers_of_8g();  // engine.cu

namespace {

constexpr size_t SCRATCH_BYTES = OG_NOALLOC_SCRATCH_BYTES;
constexpr uint32_t NBLOCK = 128;
static_assert(NBLOCK == SCRATCH_ROW, "a row of a CTA's scratch holds its threads");
constexpr int MAX_DEVICES = 64;

static __device__ __align__(256) uint4 og_noalloc_scratch[SCRATCH_BYTES / sizeof(uint4)];

// The limit callers are told, in uint4 units: lanes * (2 half + 3) * 64 +
// half * 96 bytes. The call lays the array out for a tiling of its own.
size_t need_uint4(uint32_t lanes, uint32_t half) {
    return (size_t)half * 6 + (size_t)lanes * 4 + (size_t)lanes * (2 * (size_t)half + 2) * 4;
}

// How the search covers its candidates: `ctas` blocks, a lane a thread, each
// lane `rounds` windows of 2 half + 1 candidates.
struct NoAllocTile {
    uint32_t half, ctas, rounds;
};

// uint4 the array holds for a tile: the PairTable, the lane centres (four a
// lane) and the CTAs' scratch.
size_t tile_uint4(uint32_t half, uint32_t ctas, SinkKind kind) {
    return pair_table_uint4(half) + (size_t)ctas * (NBLOCK * 4 + cta_scratch_uint4(half, kind));
}

// All `resident` blocks, in one round where the array holds the scratch of
// windows that long, else in as many as it takes (a round's own cost is that of
// about 10 groups of three pairs, so the longest windows that fit: on 592 CTAs 12
// groups; while room was kept to compute every key in full, 8, and 4.05e7 candidates
// took 1.77 ms for 1.60). Windows of at least two groups.
NoAllocTile plan_tile(uint64_t candidates, uint32_t resident, SinkKind kind) {
    const uint64_t threads = (uint64_t)resident * NBLOCK, window = (candidates + threads - 1) / threads;
    uint32_t groups = 2;
    while (2ULL * GROUP * groups + 1 < window &&
           tile_uint4(GROUP * (groups + 1), resident, kind) * sizeof(uint4) <= SCRATCH_BYTES)
        groups++;
    NoAllocTile t{GROUP * groups, resident, 1};
    const uint64_t lane = 2ULL * t.half + 1;
    t.ctas = (uint32_t)std::min<uint64_t>(resident, (candidates + lane * NBLOCK - 1) / (lane * NBLOCK));
    t.rounds = (uint32_t)((candidates + lane * NBLOCK * t.ctas - 1) / (lane * NBLOCK * t.ctas));
    return t;
}

struct NoAllocArgs {
    uint4* table;
    uint4* lanes;
    uint4* scratch;
    FeWords bx, by, bz, bt;  // first centre, extended
    Stride stride;           // between rounds
    uint64_t limit;          // candidates
    uint32_t out_lanes;      // the caller's shape, in which the records are numbered
    uint32_t out_slots;
    uint32_t table_blocks;   // blocks of the first kernel that write the table; the others the lanes
    const uint32_t* bitmap;
    uint32_t bits;
    HitRec* hits;
    uint32_t* counter;
    uint32_t cap;
    uint32_t lanes_n;  // of the tile, as half and rounds
    uint32_t half;
    uint32_t rounds;
};

// The table's entries on the first blocks, the lanes' first centres on the
// others: neither needs the other. The power tables travel as launch parameters: a
// copy from pageable host memory would wait for the work already queued on the
// caller's stream.
__global__ void __launch_bounds__(NBLOCK) noalloc_start_kernel(const NoAllocArgs a, const Pow2Table eight,
                                                               const Pow2Table stride) {
    if (blockIdx.x < a.table_blocks)
        fill_pair_entry(pair_table_at<const uint4>(a.table, a.half), groups_of(a.half) * GROUP, eight,
                        blockIdx.x * NBLOCK + threadIdx.x);
    else
        first_centre(words_fe(a.bx), words_fe(a.by), words_fe(a.bz), words_fe(a.bt), stride,
                     (blockIdx.x - a.table_blocks) * NBLOCK + threadIdx.x, a.lanes, a.lanes_n);
}

// The production paired kernel with its scratch in the file-scope array; the
// table is read through L1 as in the single engine.
template <bool Narrow>
__global__ void __launch_bounds__(NBLOCK, 4) noalloc_paired_kernel(const NoAllocArgs a) {
    const uint32_t lane = blockIdx.x * blockDim.x + threadIdx.x;
    const Sink sink{a.bitmap, a.bits,  a.hits,    a.counter, a.cap,           0,           nullptr,
                    0,        nullptr, a.limit,   a.lanes_n,       2 * a.half + 1, a.out_lanes,
                    a.out_slots};
    const PairTable tab = pair_table_at<const uint4>(a.table, a.half);
    uint4* const scr = a.scratch + (size_t)blockIdx.x * cta_scratch_uint4(a.half, Narrow ? SINK_PREFIX : SINK_FULL) + threadIdx.x;
    if constexpr (Narrow) {
        __shared__ __align__(128) RoundShared sh;
        MatrixUnit mu;
        matrix_open(sh);
        paired_rounds<false, false, true>(a.lanes + lane, a.lanes_n, a.stride, a.stride, tab, a.half, a.rounds, scr, sink, sh, mu, lane, true);
        if (threadIdx.x == 0 && sh.failed) atomicOr(a.counter, OG_NOALLOC_FAILED);
        matrix_close(sh);
    } else {
        paired_rounds_full<true>(a.lanes + lane, a.lanes_n, a.stride, a.stride, tab, a.half, a.rounds, scr, sink, lane, true);
    }
}

__global__ void __launch_bounds__(NBLOCK) noalloc_groups_kernel(const NoAllocArgs a) {
    fill_group_table(pair_table_at<const uint4>(a.table, a.half), groups_of(a.half), blockIdx.x * blockDim.x + threadIdx.x);
}

// The array's device address, per device, taken on the first call there.
std::mutex g_mu;
uint4* g_addr[MAX_DEVICES];

}  // namespace
}  // namespace og

using namespace og;

extern "C" int og_search_noalloc(int ordinal, const uint8_t start[128], uint32_t lanes, uint32_t half, uint32_t rounds,
                                 const uint32_t* d_bitmap, uint32_t bits, og_hit_record* d_hits, uint32_t cap,
                                 uint32_t* d_count, void* stream, char* err, size_t errlen) {
    if (!start || !d_hits || !d_count) return fail(err, errlen, OG_E_ARG, "null argument");
    if (ordinal < 0 || ordinal >= MAX_DEVICES) return fail(err, errlen, OG_E_ARG, "device %d", ordinal);
    if (lanes == 0 || lanes % NBLOCK)
        return fail(err, errlen, OG_E_ARG, "lanes %u: a positive multiple of %u", lanes, NBLOCK);
    if (half == 0 || half > 2048) return fail(err, errlen, OG_E_ARG, "half %u outside 1..2048", half);
    if (rounds == 0) return fail(err, errlen, OG_E_ARG, "zero rounds");
    if ((uint64_t)rounds * (2ULL * half + 1) > 0xffffffffULL) return fail(err, errlen, OG_E_ARG, "too many rounds");
    if (d_bitmap && (bits < 8 || bits > 32)) return fail(err, errlen, OG_E_ARG, "bitmap width %u outside 8..32", bits);
    if (lanes >= (1u << POW2)) return fail(err, errlen, OG_E_ARG, "lanes %u", lanes);
    const size_t need = need_uint4(lanes, half) * sizeof(uint4);
    if (need > SCRATCH_BYTES)
        return fail(err, errlen, OG_E_CAPACITY,
                    "%u lanes at half %u need %zu bytes of scratch; the fixed array holds %zu "
                    "(lanes * (2 half + 3) * 64 + half * 96 must stay within it)",
                    lanes, half, need, SCRATCH_BYTES);
    const Pt A = point_from_bytes(start);
    if (!point_valid(A)) return fail(err, errlen, OG_E_ARG, "the start point is not on the curve");
    cudaError_t e = cudaSetDevice(ordinal);
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "cudaSetDevice: %s", cuda_text(e).c_str());
    uint4* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!g_addr[ordinal]) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, og_noalloc_scratch);
            if (e != cudaSuccess || !p)
                return fail(err, errlen, OG_E_DEVICE, "cudaGetSymbolAddress: %s", cuda_text(e).c_str());
            g_addr[ordinal] = static_cast<uint4*>(p);
        }
        base = g_addr[ordinal];
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const SinkKind kind = sink_kind(d_bitmap ? bits : 0, 0);
    const bool narrow = kind == SINK_PREFIX;
    const uint32_t slots = 2 * half + 1;
    const uint64_t candidates = (uint64_t)lanes * rounds * slots;
    int per_sm = 0, sms = 0;
    e = narrow ? matrix_blocks_per_sm((const void*)noalloc_paired_kernel<true>, 0, &per_sm)
               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, noalloc_paired_kernel<false>, NBLOCK, 0);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ordinal);
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "device attributes: %s", cuda_text(e).c_str());
    const NoAllocTile tile = plan_tile(candidates, (uint32_t)(std::max(1, per_sm) * sms), kind);
    const uint32_t window = 2 * tile.half + 1;
    if ((uint64_t)tile.rounds * window > 0xffffffffULL) return fail(err, errlen, OG_E_ARG, "too many rounds");
    NoAllocArgs a;
    std::memset(&a, 0, sizeof a);
    a.lanes_n = tile.ctas * NBLOCK;
    a.half = tile.half;
    a.rounds = tile.rounds;
    a.table = base;
    a.lanes = a.table + pair_table_uint4(tile.half);
    a.scratch = a.lanes + (size_t)a.lanes_n * 4;
    // constants computed on the host and passed as launch parameters: the
    // first centre and the round stride
    const Pt first = pt_add(A, base_mult_u64(8ULL * (tile.half + 1)));
    a.bx = to_words(first.X);
    a.by = to_words(first.Y);
    a.bz = to_words(first.Z);
    a.bt = to_words(first.T);
    a.stride = stride_of(base_mult_u64(8ULL * window * a.lanes_n));
    a.limit = candidates;
    a.out_lanes = lanes;
    a.out_slots = slots;
    a.bitmap = d_bitmap;
    a.bits = bits;
    a.hits = reinterpret_cast<HitRec*>(d_hits);
    a.counter = d_count;
    a.cap = cap;
    const uint32_t groups = groups_of(tile.half);
    a.table_blocks = (groups * GROUP + NBLOCK - 1) / NBLOCK;
    // the counter starts at zero on every call
    e = cudaMemsetAsync(d_count, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "memset: %s", cuda_text(e).c_str());
    noalloc_start_kernel<<<a.table_blocks + tile.ctas, NBLOCK, 0, s>>>(
        a, powers_of_8g(), pow2_table(base_mult_u64(8ULL * window)));
    if (narrow) {
        noalloc_groups_kernel<<<(groups * 36 + NBLOCK - 1) / NBLOCK, NBLOCK, 0, s>>>(a);
        noalloc_paired_kernel<true><<<tile.ctas, NBLOCK, 0, s>>>(a);
    } else {
        noalloc_paired_kernel<false><<<tile.ctas, NBLOCK, 0, s>>>(a);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "launch: %s", cuda_text(e).c_str());
    return OG_OK;
}
