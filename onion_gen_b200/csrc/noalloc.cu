// og_search_noalloc: the paired search without any device allocation.
//
// Some callers cannot allocate device memory: code running inside another
// framework's memory pool that forbids cudaMalloc behind its back, callers
// that must not synchronise the device (cudaMalloc and cudaFree can), and
// processes that reserve all device memory up front. This entry point lets
// them run the search: they pass the inputs (start point, bitmap) and the
// outputs (survivor records and their counter) in device memory they own,
// and everything else — lane state, the Montgomery scratch and the tables —
// lives in one file-scope device array, `og_noalloc_scratch`, sized
// OG_NOALLOC_SCRATCH_BYTES. Every GPU that loads the library holds that array
// until the process exits.
//
// Host code must not use the array's name as a device address (in host code
// it is a host-side stand-in); it takes the address once per device with
// cudaGetSymbolAddress, on the first call made on that device, and passes it
// to the kernels.
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "../../include/onion_gen_b200.h"
#include "host/common.h"
#include "search_common.cuh"

namespace og {

Stride stride_of(const Pt& w);  // engine.cu

namespace {

constexpr size_t SCRATCH_BYTES = OG_NOALLOC_SCRATCH_BYTES;
constexpr uint32_t NBLOCK = 128;
static_assert(NBLOCK == SCRATCH_ROW, "a row of a CTA's scratch holds its threads");
constexpr uint32_t POW2 = 24;
constexpr int MAX_DEVICES = 64;

static __device__ __align__(256) uint4 og_noalloc_scratch[SCRATCH_BYTES / sizeof(uint4)];

// The limit callers are told, in uint4 units: lanes * (2 half + 3) * 64 +
// half * 96 bytes. Inside it lie the PairTable, the lane centres (lanes * 4)
// and the CTAs' scratch: 600 g + lanes * (4 + 6 g) for g = groups_of(half),
// which is less for every half and at least one block of lanes.
size_t need_uint4(uint32_t lanes, uint32_t half) {
    return (size_t)half * 6 + (size_t)lanes * 4 + (size_t)lanes * (2 * (size_t)half + 2) * 4;
}
constexpr bool layout_fits(uint32_t half) {
    return pair_table_uint4(half) + NBLOCK * 4 + cta_scratch_uint4(half) <=
               half * 6 + NBLOCK * 4 + (size_t)NBLOCK * (2 * half + 2) * 4 &&
           cta_scratch_uint4(half) <= (size_t)NBLOCK * (2 * half + 2) * 4;
}
static_assert(layout_fits(1) && layout_fits(2) && layout_fits(4) && layout_fits(2048),
              "the arrays fit in what the limit allows");

// 2^k p for k < POW2 in cached form (y + x, y - x, 2 d x y; Z = 1), passed to
// the kernels by value as a launch parameter (2304 bytes), so that the call
// copies nothing from host memory: a host-to-device copy from pageable
// memory would wait for the work already queued on the caller's stream.
struct Pow2Table {
    uint4 v[POW2 * 6];
};

struct NoAllocArgs {
    uint4* table;
    uint4* lanes;
    uint4* scratch;
    FeWords bx, by, bz, bt;  // first centre, extended
    FeWords ex, ey, ez, et;  // 8G, extended (table entry 1)
    Stride stride;           // between rounds
    const uint32_t* bitmap;
    uint32_t bits;
    HitRec* hits;
    uint32_t* counter;
    uint32_t cap;
    uint32_t lanes_n;
    uint32_t half;
    uint32_t rounds;
};

// The paired round's table (PairTable) of Q_m = m * 8G, m = 1..half. Entry
// m - 1 starts from 8G and adds 2^k * 8G (from `pow8`) for every bit k of
// m - 1.
__global__ void __launch_bounds__(NBLOCK) noalloc_table_kernel(const NoAllocArgs a, const Pow2Table pow8) {
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n = groups_of(a.half) * GROUP;
    if (m >= n) return;
    fe X = words_fe(a.ex), Y = words_fe(a.ey), Z = words_fe(a.ez), T = words_fe(a.et);
    for (uint32_t k = 0; k < POW2; k++)
        if ((m >> k) & 1u) {
            const uint4* p = pow8.v + (size_t)k * 6;
            add_cached(X, Y, Z, T, load_fe(p + 0, 1), load_fe(p + 2, 1), load_fe(p + 4, 1));
        }
    // of the affine (x, y): v = 1/y = Z (Z^2 + X^2) i, s = x / (1 + x^2) = X Y Z i and
    // q = v^2 / d, with i = 1 / (Y (Z^2 + X^2))
    const fe den = fe_add(fe_sqv(Z), fe_sqv(X));
    const fe zi = fe_mulv(Z, fe_invert(fe_mulv(Y, den)));
    const fe v = fe_canon(fe_mulv(den, zi));
    store_fe(a.table + (size_t)m * 2, 1, fe_canon(fe_mulv(fe_sqv(v), const_inv_d())));
    uint4* const vs = a.table + (size_t)n * 2 + (size_t)m * 4;
    store_fe(vs + 0, 1, v);
    store_fe(vs + 2, 1, fe_canon(fe_mulv(fe_mulv(X, Y), zi)));
}

// Lane l starts on the centre of window l: the first centre plus 2^k times
// the lane stride (from `pow2`) for every bit k of l.
__global__ void __launch_bounds__(NBLOCK) noalloc_init_kernel(const NoAllocArgs a, const Pow2Table pow2) {
    const uint32_t lane = blockIdx.x * blockDim.x + threadIdx.x;
    if (lane >= a.lanes_n) return;
    const size_t L = a.lanes_n;
    fe X = words_fe(a.bx), Y = words_fe(a.by), Z = words_fe(a.bz), T = words_fe(a.bt);
    for (uint32_t k = 0; k < POW2; k++)
        if ((lane >> k) & 1u) {
            const uint4* p = pow2.v + (size_t)k * 6;
            add_cached(X, Y, Z, T, load_fe(p + 0, 1), load_fe(p + 2, 1), load_fe(p + 4, 1));
        }
    const fe zi = fe_invert(Z);
    store_fe(a.lanes + 0 * L + lane, L, fe_mulv(X, zi));
    store_fe(a.lanes + 2 * L + lane, L, fe_mulv(Y, zi));
}

// The production paired kernel with its scratch in the file-scope array; the
// table is read through L1 as in the single engine.
template <bool Narrow>
__global__ void __launch_bounds__(NBLOCK, 4) noalloc_paired_kernel(const NoAllocArgs a) {
    const uint32_t lane = blockIdx.x * blockDim.x + threadIdx.x;
    const Sink sink{a.bitmap, a.bits, a.hits, a.counter, a.cap, 0, nullptr, 0};
    const PairTable tab = pair_table_at<const uint4>(a.table, a.half);
    uint4* const scr = a.scratch + (size_t)blockIdx.x * cta_scratch_uint4(a.half) + threadIdx.x;
    if constexpr (Narrow) {
        __shared__ __align__(128) RoundShared sh;
        MatrixUnit mu;
        matrix_open(sh);
        paired_rounds<true>(a.lanes + lane, a.lanes_n, a.stride, a.stride, tab, a.half, a.rounds, scr, sink, sh, mu, lane, true);
        // a wait that ran out leaves a count beyond any room
        if (threadIdx.x == 0 && sh.failed) atomicOr(a.counter, 0x80000000u);
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

// 2^k * p for k < POW2 in cached form.
void pow2_into(Pt p, uint4* out) {
    for (uint32_t k = 0; k < POW2; k++) {
        const Niels c = pt_niels(p);
        put_fe(out + k * 6 + 0, 1, c.ypx);
        put_fe(out + k * 6 + 2, 1, c.ymx);
        put_fe(out + k * 6 + 4, 1, c.xy2d);
        p = pt_dbl(p);
    }
}

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
    NoAllocArgs a;
    std::memset(&a, 0, sizeof a);
    a.table = base;
    a.lanes = a.table + pair_table_uint4(half);
    a.scratch = a.lanes + (size_t)lanes * 4;
    const uint32_t slots = 2 * half + 1;
    // constants computed on the host and passed as launch parameters: the
    // first centre, 8G, the round stride
    const Pt first = pt_add(A, base_mult_u64(8ULL * (half + 1)));
    a.bx = to_words(first.X);
    a.by = to_words(first.Y);
    a.bz = to_words(first.Z);
    a.bt = to_words(first.T);
    const Pt eight = base_mult_u64(8);
    a.ex = to_words(eight.X);
    a.ey = to_words(eight.Y);
    a.ez = to_words(eight.Z);
    a.et = to_words(eight.T);
    a.stride = stride_of(base_mult_u64(8ULL * slots * lanes));
    a.bitmap = d_bitmap;
    a.bits = bits;
    a.hits = reinterpret_cast<HitRec*>(d_hits);
    a.counter = d_count;
    a.cap = cap;
    a.lanes_n = lanes;
    a.half = half;
    a.rounds = rounds;
    // the two power-of-two tables travel as launch parameters
    Pow2Table pow2, pow8;
    pow2_into(base_mult_u64(8ULL * slots), pow2.v);
    pow2_into(eight, pow8.v);
    // the counter starts at zero on every call
    e = cudaMemsetAsync(d_count, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "memset: %s", cuda_text(e).c_str());
    const uint32_t groups = groups_of(half);
    noalloc_table_kernel<<<(groups * GROUP + NBLOCK - 1) / NBLOCK, NBLOCK, 0, s>>>(a, pow8);
    noalloc_init_kernel<<<lanes / NBLOCK, NBLOCK, 0, s>>>(a, pow2);
    if (sink_is_narrow(d_bitmap != nullptr, bits, false)) {
        noalloc_groups_kernel<<<(groups * 48 + NBLOCK - 1) / NBLOCK, NBLOCK, 0, s>>>(a);
        noalloc_paired_kernel<true><<<lanes / NBLOCK, NBLOCK, 0, s>>>(a);
    } else {
        noalloc_paired_kernel<false><<<lanes / NBLOCK, NBLOCK, 0, s>>>(a);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err, errlen, OG_E_DEVICE, "launch: %s", cuda_text(e).c_str());
    return OG_OK;
}
