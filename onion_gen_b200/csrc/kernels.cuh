// Device kernels of the key search and the host-side launch interface.
//
// A lane holds an affine centre P. One round yields y(P + Q_m) and y(P - Q_m)
// for the table Q_m = 8m G, m = 1..half, plus y(P) itself, from a formula in
// which both have the same denominator (search_common.cuh), and moves P to
// the next centre P + W. Every denominator of the round is inverted with one
// field inversion (Montgomery's trick): nine multiplications for three pairs.
//
// Candidate numbering. The kernels number the candidates of a launch from 0:
// lane l of L in round r covers the window w = r L + l of 2 half + 1
// candidates, index w (2 half + 1) + i; i = half is the centre, i = half + m is
// P + Q_m, i = half - m is P - Q_m. An engine's kernel stops at the number of
// candidates of one advance, whatever half and lanes it runs at, so the
// tiling is free: both enumeration schemes run on it. With k the index in all
// advances, the scalar offset is
//   paired: 8 (k + 1), where lane l's window of user shape (half, lanes) is
//           k = w (2 half + 1) + i;
//   chain:  8 k, k = w n + t for step t of lane l (the contract of src/batch.rs).
// Offsets never collide, and every candidate of a launch is covered once.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#ifndef OG_LB_THREADS
#define OG_LB_THREADS 128  // the most threads a block of the search kernels has
#endif

namespace og {

// One bitmap survivor: 48 bytes, three 16-byte stores.
struct HitRec {
    uint32_t lane;  // the lane; or (Sink::limit) the low word of the candidate's index
    uint32_t step;  // round-in-launch * slots + candidate index; or the index's high word
    uint32_t search;
    uint32_t pad;
    uint32_t y[8];  // canonical y, little-endian limbs (the packed key, sign bit clear)
};
static_assert(sizeof(HitRec) == 48, "HitRec layout");

// A device exact match in the caller's layout (og_match): the candidate's
// scalar offset, its canonical y limbs (the packed key's little-endian
// bytes) and the filter it matched. The match kernel decodes the offset, so
// the host copies the records through unchanged.
struct MatchRec {
    uint64_t offset;
    uint32_t y[8];
    uint32_t filter;
    uint32_t pad;
};
static_assert(sizeof(MatchRec) == 48, "MatchRec layout");

// Entries of the table of multiples of 8G (add_multiple_8g): 16 digits of four bits.
constexpr uint32_t MULTIPLES_8G = 16 * 16;

struct FeWords {
    uint32_t v[8];
};

// 2^k p for k < POW2 in cached form (y + x, y - x, 2 d x y; Z = 1), passed to
// kernels by value as a launch parameter (2304 bytes), so that nothing is copied
// from host memory for it.
constexpr uint32_t POW2 = 24;
struct Pow2Table {
    uint4 v[POW2 * 6];  // (k * 3 + {ypx,ymx,t2d}) * 2 + q
};

// A stride W between centres: affine x and y, and d x y.
struct Stride {
    FeWords x, y, dt;
};

// Rows of a CTA's scratch hold this many threads (the largest block).
constexpr uint32_t SCRATCH_ROW = OG_LB_THREADS;

// The tables of one half, for G = ceil(half / 3) groups. Per entry (3 G of
// them) q (two uint4) and v, s (four), for the full products; per group s1,
// s2 = the sums of products, e0 = s3 - s1 s2 (six uint4) and the constants of
// its matrix product.
struct PairTable {
    const uint4* q;
    const uint4* vs;
    const uint4* cubic;
    const uint4* constants;
};

constexpr uint32_t GROUP = 3;                     // pairs per group
constexpr uint32_t GROUP_CONSTANTS = 12 * 48;     // uint4 a group

__host__ __device__ constexpr uint32_t groups_of(uint32_t half) { return (half + GROUP - 1) / GROUP; }
// uint4 of a PairTable in one array: q, vs, cubic, constants.
__host__ __device__ constexpr size_t pair_table_uint4(uint32_t half) {
    return (size_t)groups_of(half) * (GROUP * 6 + 6 + GROUP_CONSTANTS);
}
template <class T>
__host__ __device__ PairTable pair_table_at(T* base, uint32_t half) {
    const size_t g = groups_of(half);
    return PairTable{base, base + g * GROUP * 2, base + g * GROUP * 6, base + g * (GROUP * 6 + 6)};
}
// How a sink's keys are tested: by paired_rounds, whose matrix product gives a
// key's low 24 bits and its bits from 231 on, or in full. A suffix bitmap of 24
// bits reads one bit more, and paired_rounds looks both of its values up: twice
// the possible survivors to compute, but 9.7e7 candidates against 40 eight-symbol
// suffixes (0.24 % of them survive) took 3.45 ms in full and take 2.43. A width of 0 stands for no bitmap.
enum SinkKind { SINK_PREFIX, SINK_SUFFIX, SINK_FULL };
__host__ __device__ inline SinkKind sink_kind(uint32_t prefix_bits, uint32_t suffix_bits) {
    if (prefix_bits > 24 || suffix_bits > 24 || (!prefix_bits && !suffix_bits)) return SINK_FULL;
    return suffix_bits ? SINK_SUFFIX : SINK_PREFIX;
}

// uint4 of a CTA's scratch: paired_rounds keeps a prefix product and E per group and
// thread, paired_rounds_full a prefix product per pair.
__host__ __device__ constexpr size_t cta_scratch_uint4(uint32_t half, SinkKind kind) {
    return (size_t)groups_of(half) * (kind == SINK_FULL ? 2 * GROUP : 4) * SCRATCH_ROW;
}

struct PairedArgs {
    const uint4* table;      // PairTable of Q_m, m = 1..half (pair_table_at)
    uint4* lanes;            // affine centres: ({x,y} * 2 + q) * L + lane
    uint4* scratch;          // cta_scratch_uint4(half, kind) per CTA
    uint32_t* work;          // next block of lanes to take, zero at launch
    const uint32_t* bitmap;  // prefix bitmap as 32-bit words (nullptr: none)
    uint32_t bits;
    HitRec* hits;
    uint32_t* counter;
    uint32_t cap;
    uint32_t search;         // copied into every record
    const uint32_t* sbitmap; // suffix bitmap (nullptr: none); with neither bitmap every candidate survives
    uint32_t sbits;
    Stride between;          // L (2 half + 1) 8 G, after every round but the last
    Stride last;             // after the last round: to the lane's first centre of the next launch
    uint64_t limit;          // candidates of a launch: indexes at and above it are none
    uint32_t lanes_n;        // L
    uint32_t half;
    uint32_t rounds;         // rounds per launch
    uint32_t* failed;        // set to 1 when a wait of the kernel ran out
};

// Lane start points: lane l starts at base + l * stride, affine, built from
// the binary expansion of l over the Pow2Table of the stride.
struct InitArgs {
    uint4* lanes;            // ({x,y} * 2 + q) * L + lane
    FeWords bx, by, bz, bt;  // base point, extended
    uint32_t lanes_n;
};

// Exact-match tables of a literal-prefix filter set in the form the device
// searches (FilterSet::match_key, src/filter.rs:2194-2213, with the length
// buckets of :2645-2700): one bucket per distinct filter length of at most
// 12 symbols, each a sorted run of masked 64-bit key heads (bytes 0..7 of the
// packed key, big-endian) with the owning filter's index.
constexpr int MAX_MATCH_BUCKETS = 12;
struct MatchTables {
    const uint64_t* keys;
    const uint32_t* owners;
    uint32_t nbuckets;
    uint32_t bucket_bits[MAX_MATCH_BUCKETS];
    uint32_t bucket_off[MAX_MATCH_BUCKETS];
    uint32_t bucket_len[MAX_MATCH_BUCKETS];
    // prefixes with wildcards or classes, walked after the buckets: per
    // pattern PATTERN_WORDS words, its filter index, the key-only symbols it
    // fixes (at most 49) and one symbol set per position
    const uint32_t* patterns;
    uint32_t npatterns;
};
constexpr uint32_t PATTERN_WORDS = 2 + 49;

// The single engine's exact match over one advance's bitmap survivors:
// matching records are copied to `out` with `pad` = the filter's index.
// Prefixes are matched on the key (MatchTables). A survivor whose slot is
// set in the suffix bitmap has its full key recomputed from its offset
// (start + k 8G), sign bit and checksum included, and is matched on its
// address against every suffix.
constexpr uint32_t MAX_SUFFIX_SYMBOLS = 56;
struct MatchArgs {
    const HitRec* surv;
    const uint32_t* surv_count;
    uint32_t surv_cap;
    MatchTables t;           // nbuckets = 0: no prefixes
    const uint32_t* sbitmap; // suffix bitmap, nullptr: no suffixes
    uint32_t sbits;
    const uint32_t* suffixes;  // per suffix 57 words: its length, then one symbol set per position
    uint32_t nsuffix;
    uint32_t prefix_count;     // filter index of suffix j is prefix_count + j
    FeWords sx, sy, sz, st;    // the engine's start point, extended
    const uint4* mul8;         // multiples of 8G (add_multiple_8g)
    uint64_t first;            // scalar offset over 8 of the advance's candidate 0
    MatchRec* out;
    uint32_t* out_count;
    uint32_t out_cap;
    uint32_t* mismatch;        // survivors whose recomputed key differs from their record
};

cudaError_t launch_init(const InitArgs& a, const Pow2Table& stride, cudaStream_t s);
cudaError_t launch_match(const MatchArgs& a, int grid, cudaStream_t s);
// The search kernel is persistent: `grid` CTAs of OG_LB_THREADS (at most the
// resident ones) take the lanes a block at a time from `work`, so the scratch
// covers only the lanes in flight and no SM idles in a tail wave.
// `kind` is that of its bitmaps, or SINK_FULL, which takes any bitmaps and any start.
cudaError_t launch_paired(const PairedArgs& a, SinkKind kind, int grid, cudaStream_t s);
// Writes a PairTable of `half` from the Pow2Table of 8G.
cudaError_t launch_pair_table(uint4* table, uint32_t half, const Pow2Table& eight, cudaStream_t s);

// Resident blocks per SM of the search kernel.
cudaError_t paired_blocks_per_sm(SinkKind kind, int* blocks);
// The same of a kernel that allocates tensor memory, from its registers,
// shared memory and tensor memory: the occupancy calculator counts one block
// per SM for such a kernel.
cudaError_t matrix_blocks_per_sm(const void* fn, size_t dynamic_shared, int* blocks);

}  // namespace og
