// Device building blocks shared by the single-search and the batched
// kernels: device-layout loads and stores, the survivor test and append, the
// cached point addition, and one lane's paired rounds.
#pragma once
#include "field.cuh"
#include "kernels.cuh"

namespace og {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ fe load_fe(const uint4* p, size_t qstride) {
    const uint4 a = p[0];
    const uint4 b = p[qstride];
    fe r;
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
    return r;
}

__device__ __forceinline__ void store_fe(uint4* p, size_t qstride, const fe& v) {
    p[0] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    p[qstride] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
}

__device__ __forceinline__ fe words_fe(const FeWords& w) {
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = w.v[k];
    return r;
}

// Where survivors go: the bitmaps, the record buffer and its counter.
struct Sink {
    const uint32_t* bitmap;  // prefix bitmap in global or in the block's shared memory, or nullptr
    uint32_t bits;
    HitRec* hits;
    uint32_t* counter;
    uint32_t cap;
    uint32_t search;
    const uint32_t* sbitmap;  // suffix bitmap, or nullptr
    uint32_t sbits;
    uint32_t* failed = nullptr;  // set when a wait of the search kernel ran out
    // With `limit` set, a record holds its candidate's index in the launch
    // (lane the low word, step the high one) instead of its lane and step, and
    // candidates at `limit` and above are none: lane l of `lanes` covers in
    // round r the `slots` candidates from (r lanes + l) slots on.
    uint64_t limit = 0;
    uint32_t lanes = 0;
    uint32_t slots = 0;
    // the caller's lanes and slots, when its records are to hold the lane and
    // step that the index has among those instead
    uint32_t out_lanes = 0;
    uint32_t out_slots = 0;
};

// Prefix bitmaps of at most this many bits (8 KiB) can be staged in shared
// memory.
constexpr uint32_t STAGED_BITMAP_BITS = 16;

// Slot of a canonical key, from its limbs 6 and 7, in the suffix bitmap: base32 bits
// [255 - sbits, 255) of the packed key, i.e. bits 1..sbits of its last eight
// bytes read big-endian (BitmapIndex::slot with offset 255 - sbits,
// src/filter.rs:2536-2549). The sign bit (bit 7 of byte 31) is clear in the
// packed key and the bitmap holds both of its values.
__device__ __forceinline__ uint32_t suffix_slot(uint32_t y6, uint32_t y7, uint32_t sbits) {
    const uint32_t lo = __byte_perm(y7, 0, 0x0123), hi = __byte_perm(y6, 0, 0x0123);
    const uint32_t w = (lo >> 1) | (hi << 31);
    return sbits >= 32 ? w : w & ((1u << sbits) - 1u);
}

// Slot in the prefix bitmap of a key whose canonical low limb is `y0`: bytes
// 0..3 of the key, big-endian, are the top of the slot.
__device__ __forceinline__ uint32_t prefix_slot(const Sink& k, uint32_t y0) {
    return __byte_perm(y0, 0, 0x0123) >> (32 - k.bits);  // bits is 8..32
}

__device__ __forceinline__ bool prefix_hit(const Sink& k, uint32_t y0) {
    const uint32_t slot = prefix_slot(k, y0);
    return (k.bitmap[slot >> 5] >> (slot & 31)) & 1u;
}

// Whether the slot of a key with the limbs 6 and 7 is set in the sink's suffix
// bitmap.
__device__ __forceinline__ bool suffix_hit(const Sink& k, uint32_t y6, uint32_t y7) {
    const uint32_t slot = suffix_slot(y6, y7, k.sbits);
    return (__ldg(k.sbitmap + (slot >> 5)) >> (slot & 31)) & 1u;
}

// Tests a candidate's slots in the prefix bitmap and in the suffix bitmap
// (either lets it through; with neither, every candidate survives) and
// appends a record for every lane of the warp that hit, canonicalised, with
// one atomic per warp. Lanes with `valid` false have no candidate. Every
// lane of the warp calls this together.
__device__ __forceinline__ void test_emit(const Sink& k, const fe& yraw, uint32_t lane, uint32_t step,
                                          bool valid = true) {
    // The canonical limbs the bitmaps read (0, 6 and 7), without the full
    // canonicalisation. Folding bit 255 adds 19 to limb 0; its carry reaches
    // limb 6 only through limbs 1..5 all ones, and the value can be p or
    // more only with limbs 1..6 all ones (a carry out of limb 0 leaves it
    // below 19, too small for that). Outside that case, which a uniform key
    // meets with probability 2^-160, the canonical limbs are these.
    fe y;
    y.v[0] = yraw.v[0] + ((yraw.v[7] >> 31) ? 19u : 0u);
    y.v[6] = yraw.v[6];
    y.v[7] = yraw.v[7] & 0x7fffffffu;
    if ((yraw.v[1] & yraw.v[2] & yraw.v[3] & yraw.v[4] & yraw.v[5]) == 0xffffffffu) y = fe_canon(yraw);
    bool hit = valid;
    if (k.bitmap || k.sbitmap) {
        hit = false;
        if (k.bitmap && valid) hit = prefix_hit(k, y.v[0]);
        if (k.sbitmap && valid) hit |= suffix_hit(k, y.v[6], y.v[7]);
    }
    if (k.limit && hit) {
        const uint64_t index = ((uint64_t)(step / k.slots) * k.lanes + lane) * k.slots + step % k.slots;
        hit = index < k.limit;
        lane = (uint32_t)index;
        step = (uint32_t)(index >> 32);
        if (k.out_slots) {
            const uint64_t window = index / k.out_slots;
            lane = (uint32_t)(window % k.out_lanes);
            step = (uint32_t)(window / k.out_lanes * k.out_slots + index % k.out_slots);
        }
    }
    const unsigned mask = __ballot_sync(FULL, hit);
    if (mask == 0) return;
    const unsigned me = threadIdx.x & 31u;
    const unsigned leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (me == leader) base = atomicAdd(k.counter, (uint32_t)__popc(mask));
    base = __shfl_sync(FULL, base, leader);
    if (hit) {
        const uint32_t idx = base + (uint32_t)__popc(mask & ((1u << me) - 1u));
        if (idx < k.cap) {
            y = fe_canon(yraw);
            uint4* rec = reinterpret_cast<uint4*>(k.hits + idx);
            rec[0] = make_uint4(lane, step, k.search, 0u);
            rec[1] = make_uint4(y.v[0], y.v[1], y.v[2], y.v[3]);
            rec[2] = make_uint4(y.v[4], y.v[5], y.v[6], y.v[7]);
        }
    }
}

// Symbol `pos` (five bits, most significant first) of a canonical key held
// as eight little-endian limbs, i.e. of its 32 packed bytes.
__device__ __forceinline__ uint32_t key_symbol(const uint32_t y[8], uint32_t pos) {
    const uint32_t bit = pos * 5, byte = bit / 8;
    const uint32_t b0 = (y[byte / 4] >> (8 * (byte % 4))) & 0xffu;
    const uint32_t b1 = byte + 1 < 32 ? (y[(byte + 1) / 4] >> (8 * ((byte + 1) % 4))) & 0xffu : 0u;
    return (((b0 << 8) | b1) >> (11 - bit % 8)) & 31u;
}

// The filter a canonical key matches, or 0xffffffff: per length bucket of
// the literal prefixes a binary search of the sorted masked heads (first 12
// symbols at most; no kept literal is a prefix of another, so at most one
// matches), then the patterns in order, on their key-only symbols.
__device__ __forceinline__ uint32_t exact_owner(const MatchTables& t, const uint32_t y[8]) {
    const uint64_t head = ((uint64_t)__byte_perm(y[0], 0, 0x0123) << 32) | (uint64_t)__byte_perm(y[1], 0, 0x0123);
    for (uint32_t b = 0; b < t.nbuckets; b++) {
        const uint64_t probe = head & (~0ULL << (64 - t.bucket_bits[b]));
        const uint64_t* k = t.keys + t.bucket_off[b];
        uint32_t lo = 0, hi = t.bucket_len[b];
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (k[mid] < probe) lo = mid + 1;
            else hi = mid;
        }
        if (lo < t.bucket_len[b] && k[lo] == probe) return t.owners[t.bucket_off[b] + lo];
    }
    for (uint32_t j = 0; j < t.npatterns; j++) {
        const uint32_t* p = t.patterns + (size_t)j * PATTERN_WORDS;
        bool ok = true;
        for (uint32_t i = 0; i < p[1] && ok; i++) ok = (p[2 + i] >> key_symbol(y, i)) & 1u;
        if (ok) return p[0];
    }
    return 0xffffffffu;
}

__device__ __forceinline__ fe shfl_up_fe(const fe& v, unsigned d) {
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = __shfl_up_sync(FULL, v.v[k], d);
    return r;
}

__device__ __forceinline__ fe shfl_down_fe(const fe& v, unsigned d) {
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = __shfl_down_sync(FULL, v.v[k], d);
    return r;
}

__device__ __forceinline__ fe select_fe(bool c, const fe& a, const fe& b) {
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = c ? a.v[k] : b.v[k];
    return r;
}

// 1/v for every thread of the block with one field inversion for the whole
// block: Montgomery's trick across its lanes. A warp executes an inversion
// at the cost of all its lanes whether one lane or 32 need it, so one
// inversion a block instead of one a warp saves three of every four on
// 128-thread blocks. Within a warp, inclusive prefix and suffix products by
// shuffles (five levels each, the missing neighbours taken as 1); across
// warps, their totals in shared memory; thread 0 inverts the block's total;
// then 1/v_i = (product before i) (product after i) / total. The inverse is
// unique, so the result equals fe_invert's modulo p (0 when some v of the
// block is 0, which the search's denominators never are). Every thread of
// the block calls it together; blocks hold at most OG_LB_THREADS threads.
// Not inlined, like fe_invert, so that the search loops' register
// allocation does not change around it.
static __device__ __noinline__ fe block_invert(const fe& v) {
    __shared__ fe warp_total_s[OG_LB_THREADS / 32];
    __shared__ fe inv_total_s;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const fe one = fe_one();
    fe pre = v, suf = v;
#pragma unroll
    for (unsigned d = 1; d < 32; d <<= 1) {
        const fe lo = shfl_up_fe(pre, d), hi = shfl_down_fe(suf, d);
        pre = fe_mulv(pre, select_fe(lane >= d, lo, one));
        suf = fe_mulv(suf, select_fe(lane + d < 32, hi, one));
    }
    // exclusive: the products strictly before and after this lane
    const fe before = select_fe(lane > 0, shfl_up_fe(pre, 1), one);
    const fe after = select_fe(lane < 31, shfl_down_fe(suf, 1), one);
    __syncthreads();  // earlier readers of the shared words are done
    if (lane == 31) warp_total_s[warp] = pre;
    __syncthreads();
    if (threadIdx.x == 0) {
        fe total = warp_total_s[0];
        for (unsigned w = 1; w < nwarps; w++) total = fe_mulv(total, warp_total_s[w]);
        inv_total_s = fe_invert(total);
    }
    // the other warps' totals, before and after this warp (the same in every lane)
    fe others = one;
    for (unsigned w = 0; w < nwarps; w++)
        if (w != warp) others = fe_mulv(others, warp_total_s[w]);
    __syncthreads();
    return fe_mulv(fe_mulv(before, after), fe_mulv(others, inv_total_s));
}

// p3 + cached addend with Z = 1: seven multiplications
// (the formulas of src/curve.rs:130-175 with the addend's Z scaled away).
__device__ __forceinline__ void add_cached(fe& X, fe& Y, fe& Z, fe& T, const fe& ypx, const fe& ymx,
                                           const fe& t2d) {
    const fe a = fe_mulv(fe_add(Y, X), ypx);
    const fe b = fe_mulv(fe_sub(Y, X), ymx);
    const fe c = fe_mulv(T, t2d);
    const fe d = fe_add(Z, Z);
    const fe x3 = fe_sub(a, b), y3 = fe_add(a, b), z3 = fe_add(d, c), t3 = fe_sub(d, c);
    X = fe_mulv(x3, t3);
    Y = fe_mulv(y3, z3);
    Z = fe_mulv(z3, t3);
    T = fe_mulv(x3, y3);
}

// Adds k 8G from a table of d 16^w 8G (w < 16, d < 16; 0 is the identity) in
// cached form, (((w * 16 + d) * 3 + {ypx,ymx,t2d}) * 2 + q). Four bits an
// addition: the lanes' k differ in every digit, so a warp would take all the
// additions of a table of powers of two, a chain of 3 500 clocks for each bit of
// the longest k. The table, 24 KB, stays in L1.
__device__ __forceinline__ void add_multiple_8g(fe& X, fe& Y, fe& Z, fe& T, const uint4* table, uint64_t k) {
#pragma unroll 1
    for (; k; k >>= 4, table += 16 * 6) {
        const uint4* p = table + (k & 15u) * 6;
        add_cached(X, Y, Z, T, load_fe(p + 0, 1), load_fe(p + 2, 1), load_fe(p + 4, 1));
    }
}

// ---- the paired round ---------------------------------------------------
//
// For a centre P = (x, y) and a table point Q = (x2, y2) of odd order, the
// curve equation -x^2 + y^2 = 1 + d x^2 y^2 lets the denominators of
// y(P + Q) and y(P - Q) be one and the same:
//
//     y(P +- Q) = (z v +- c s) / (q - X),
//     X = x^2, z = y (1/d - X), c = (1 + 1/d) x          (the lane's)
//     q = 1 / (d y2^2), v = 1 / y2, s = x2 / (1 + x2^2)  (the table's)
//
// (substitute y^2 = (1 + x^2) / (1 - d x^2) into the addition formula's
// numerators and 1 -+ d x x2 y y2; the common factors cancel). Its
// denominator is (1/y2^2 - d x^2) / d, which has no zero because d is not a
// square. Only z can be 0, for the two centres of order four, (+-sqrt(-1), 0):
// no s B + 8 k G is one, but a caller's start point may lead to them, and the 0
// would take the whole block's inversion with it. With AnyStart, such a lane's
// round runs with 1 for z (then e = c), and its g_k are set to 0 where they are
// stored. The batch's starts are multiples of the base point, and the engine tells
// by its start which rounds to run (may_meet_order_four), because the test costs
// them 1 to 2 %: the default advance 53.2 -> 54.5 ms.
//
// The denominators are taken three at a time. With D_i = q_i - X, i = 1..3,
// and E = D_1 D_2 D_3, the product is a cubic in X whose coefficients are
// the table's: E = (X^2 + s2) (s1 - X) + e0, one multiplication. With one
// inversion for the round's E (Montgomery's trick, the prefix products P
// started from z, and e = c / z):
//
//     h = P I [= z / E],  I <- I E,  g_k = X^k h,  f_k = e g_k,  k = 0..2
//
// and every key of the group is a sum of the six with constant coefficients,
//
//     y(P +- Q_i) = v (q'q'' g_0 - (q' + q'') g_1 + g_2) +- s (the same in f),
//
// q' and q'' the other two. So three pairs take nine multiplications, and
// the six keys are products of lane values with a table of constants: a
// matrix product, of which only what the bitmap reads is computed, on the
// tensor cores (test_group).

__device__ __forceinline__ fe const_inv_d() {  // 1/d
    return fe{{0xcdc9f843u, 0x25e0f276u, 0x4279542eu, 0x0b5dd698u, 0xcdb9cf66u, 0x2b162114u, 0x14d5ce43u, 0x40907ed2u}};
}

__device__ __forceinline__ fe const_inv_d_plus_1() {  // 1 + 1/d
    return fe{{0xcdc9f844u, 0x25e0f276u, 0x4279542eu, 0x0b5dd698u, 0xcdb9cf66u, 0x2b162114u, 0x14d5ce43u, 0x40907ed2u}};
}

// Candidates that may survive, collected per warp in shared memory: h, f_0
// and X (96 bytes), the candidate's lane and step, and its table entry with
// the sign (0: the centre, whose y is in h's place). stage_flush computes
// their keys, a lane each, tests them exactly and appends the survivors. The
// search loop itself holds neither the full products nor the record writes.
constexpr uint32_t STAGE_RECORDS = 24;
constexpr uint32_t STAGE_WORDS = 7;  // uint4 a record

struct WarpStage {
    uint4* recs;  // this warp's STAGE_RECORDS records in shared memory
    uint32_t n;   // records held; the same in every lane of the warp
};

static __device__ __noinline__ void stage_flush(const Sink& k, const PairTable& tab, const uint4* recs, uint32_t n) {
    if (n == 0) return;
    __syncwarp();
    const unsigned me = threadIdx.x & 31u;
    const bool valid = me < n;
    const uint4* r = recs + (valid ? me : 0) * STAGE_WORDS;
    const fe h = load_fe(r, 1), X = load_fe(r + 4, 1);
    const uint4 id = r[6];
    const uint32_t m = id.z & 0x7fffffffu, i = m ? m - 1 : 0, g = i / GROUP * GROUP;
    // 1 / D_i = (the group's other two D) / E
    const fe others = fe_mulv(fe_sub(load_fe(tab.q + (size_t)(g + (i - g + 1) % GROUP) * 2, 1), X),
                              fe_sub(load_fe(tab.q + (size_t)(g + (i - g + 2) % GROUP) * 2, 1), X));
    const uint4* t = tab.vs + (size_t)i * 4;
    const fe A = fe_mulv(load_fe(t, 1), h), B = fe_mulv(load_fe(t + 2, 1), load_fe(r + 2, 1));
    const fe key = fe_mulv(select_fe(id.z >> 31, fe_sub(A, B), fe_add(A, B)), others);
    const fe y = select_fe(m == 0, h, key);
    test_emit(k, y, id.x, id.y, valid);
    __syncwarp();
}

// A lane's group values in shared memory, a row of the matrix product's left
// operand: g_0, g_1, g_2, f_0, f_1, f_2, whose limbs are its 192 bytes, in
// twelve 16-byte parts. Part c of row r is at c ROWS + r, so that a warp's
// stores are contiguous and eight rows of a part are the 128 contiguous bytes
// the matrix unit reads at once.
constexpr uint32_t ROWS = 128;
constexpr uint32_t ROW_PARTS = 12;
static_assert(OG_LB_THREADS <= ROWS, "a row for every thread of a block");

__device__ __forceinline__ void store_row(uint4* row, uint32_t element, const fe& v) {
    store_fe(row + element * 2 * ROWS, ROWS, v);
}

// Adds the candidates of the lanes with `hit` set, from their rows. Every lane
// of the warp calls it together.
__device__ __forceinline__ void stage_push(const Sink& k, const PairTable& tab, WarpStage& st, bool hit,
                                           const uint4* row, const fe& X, uint32_t lane, uint32_t step, uint32_t entry) {
    for (unsigned mask = __ballot_sync(FULL, hit); mask; mask = __ballot_sync(FULL, hit)) {
        if (st.n == STAGE_RECORDS) {
            stage_flush(k, tab, st.recs, st.n);
            st.n = 0;
        }
        const uint32_t at = st.n + (uint32_t)__popc(mask & ((1u << (threadIdx.x & 31u)) - 1u));
        if (hit && at < STAGE_RECORDS) {
            uint4* r = st.recs + at * STAGE_WORDS;
            r[0] = row[0];
            r[1] = row[ROWS];
            r[2] = row[6 * ROWS];
            r[3] = row[7 * ROWS];
            store_fe(r + 4, 1, X);
            r[6] = make_uint4(lane, step, entry, 0u);
            hit = false;
        }
        st.n = min(STAGE_RECORDS, st.n + (uint32_t)__popc(mask));
    }
}

// ---- the matrix product of a group --------------------------------------
//
// For the block's 128 lanes, rows (lanes) x 192 bytes times 192 x 48
// constants (eight columns for each of the group's six keys): six tcgen05.mma of
// kind::i8, unsigned, K = 32, issued by one thread, sums in 48 columns of tensor memory, read back a lane's row by its own thread. It
// runs while the warps multiply for the next group. The constants come by a
// bulk copy, 9 KB a group for the whole block. Measured on B200 at 3.1e9
// candidates a launch when it came in: 52.6 ms (49.9 now), 47.0 with the products
// left out; by mma.sync a warp, which shares registers and issue slots with the
// multiplications, 64.2; with the keys' low limbs by multiply-adds, four
// multiplications and two partial ones a pair, 70.3.
constexpr uint32_t KEY_COLUMNS = 8;
constexpr uint32_t COLUMNS = 48;
constexpr uint32_t TMEM_COLUMNS = 64;  // an allocation is a power of two
static_assert(GROUP_CONSTANTS == ROW_PARTS * COLUMNS, "the constants of a group are one right operand");

// Shared memory of a block for paired_rounds.
struct RoundShared {
    uint4 rows[ROW_PARTS * ROWS];
    uint4 constants[GROUP_CONSTANTS];  // part c of column n at c COLUMNS + n
    uint4 stage[(OG_LB_THREADS / 32) * STAGE_RECORDS * STAGE_WORDS];
    uint64_t product_done, constants_here;  // mbarriers
    uint32_t tmem;
    uint32_t failed;  // a wait ran out: the block goes on without products, and the launch has failed
};

// The block's use of the matrix unit: the phases its two barriers are in.
struct MatrixUnit {
    uint32_t product_phase = 0, constants_phase = 0;
};

__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Called by every thread of the block, before the first round and after the
// last one.
__device__ __forceinline__ void matrix_open(RoundShared& sh) {
    __syncwarp();  // the allocation takes the whole warp, and some of its lanes may come from a branch
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_addr(&sh.tmem)),
                     "r"(TMEM_COLUMNS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_addr(&sh.product_done)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_addr(&sh.constants_here)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sh.failed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void matrix_close(RoundShared& sh) {
    // after a failed wait a copy or a product may still be under way: a
    // millisecond for it to end
    if (*(volatile uint32_t*)&sh.failed)
        for (uint32_t i = 0; i < 1000; i++) __nanosleep(1000);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(TMEM_COLUMNS));
    }
}

// Waits for the barrier's phase, a bounded number of times (a product takes
// about a microsecond; the bound is at least tens of milliseconds). If it runs
// out the block is marked failed, and so is the launch (Sink::failed).
__device__ __forceinline__ void bounded_wait(RoundShared& sh, const Sink& sink, const uint64_t* bar, uint32_t phase) {
    constexpr uint32_t LIMIT = 1u << 15;
    const uint32_t addr = shared_addr(bar);
    if (*(volatile uint32_t*)&sh.failed) return;
    for (uint32_t i = 0; i < LIMIT; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(phase)
            : "memory");
        if (done) return;
    }
    *(volatile uint32_t*)&sh.failed = 1;
    if (sink.failed) atomicExch(sink.failed, 1u);
}

// Fetches group j's constants (one thread; the product that read the last ones
// is done).
__device__ __forceinline__ void fetch_constants(RoundShared& sh, const uint4* constants) {
    const uint32_t bar = shared_addr(&sh.constants_here);
    constexpr uint32_t bytes = GROUP_CONSTANTS * 16;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     shared_addr(sh.constants)),
                 "l"(constants), "r"(bytes), "r"(bar)
                 : "memory");
}

// Every thread's row is written: starts the product (thread 0 issues it).
__device__ __forceinline__ void start_product(RoundShared& sh, const Sink& sink, MatrixUnit& mu) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        bounded_wait(sh, sink, &sh.constants_here, mu.constants_phase);
        if (!sh.failed) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // K-major operands without swizzle: 8 rows of 16 bytes contiguous,
            // 8-row groups 128 bytes apart (bits 32..45), the 16-byte parts a
            // part's size apart (bits 16..29), all in units of 16 bytes
            constexpr uint64_t common = (8ull << 32) | (1ull << 46);
            uint64_t a = common | ((uint64_t)ROWS << 16) | (shared_addr(sh.rows) >> 4);
            uint64_t b = common | ((uint64_t)COLUMNS << 16) | (shared_addr(sh.constants) >> 4);
            // 32-bit sums, unsigned 8-bit operands, N = 48, M = 128
            constexpr uint32_t idesc = (2u << 4) | ((COLUMNS / 8) << 17) | ((ROWS / 16) << 24);
#pragma unroll
            for (uint32_t k = 0; k < ROW_PARTS / 2; k++) {
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(sh.tmem),
                    "l"(a), "l"(b), "r"(idesc), "r"(k)
                    : "memory");
                a += 2 * ROWS;
                b += 2 * COLUMNS;
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             shared_addr(&sh.product_done))
                         : "memory");
        }
    }
    mu.constants_phase ^= 1;
}

// Waits for the product.
__device__ __forceinline__ void finish_product(RoundShared& sh, const Sink& sink, MatrixUnit& mu) {
    bounded_wait(sh, sink, &sh.product_done, mu.product_phase);
    mu.product_phase ^= 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Tests the six keys of the group whose first entry is m0 (entries past `half`
// belong to no key of the round) from the finished product: whether each may be
// in the sink's bitmaps. With the key T = sum of byte_j rho_j, rho_j the
// coefficient times 2^(8 j) mod p, a key's first three columns sum the bytes
// against the low 24 bits of rho_j and the others against
// floor(2^40 rho_j / p), byte by byte. The latter add up to K = 2^40 T / p less
// an error below 192 * 255 < 2^16. So k = floor(T / p) is K >> 40, unless bits
// 16..39 of K are all ones (such a key counts as a hit), and the key's low limb
// is that of T + 19 k; and K's bits 16..39, or those plus one, are the key's
// bits 231..254 (2^255 T / p modulo 2^255 exceeds the key by less than 19). The
// bitmap's words are loaded for all keys before the first is looked at, and no
// key takes a branch: with a branch a key a launch of 3.1e9 candidates took
// 59 ms, so 52.
template <bool Suffixes>
__device__ __forceinline__ void test_group(RoundShared& sh, const Sink& sink, const PairTable& tab, WarpStage& st,
                                           const fe& X, uint32_t lane, bool active, uint32_t mid, uint32_t m0,
                                           uint32_t half) {
    constexpr int KEYS = 2 * GROUP;
    const uint32_t from = sh.tmem + ((threadIdx.x / 32) << 21);  // 32 lanes a warp, in bits 16 and up
    uint32_t slot[KEYS], top[KEYS], hits = 0;
    // the loads take the whole warp, whose lanes left the wait one by one; thread
    // 0 has fetched and issued besides
    __syncwarp();
#pragma unroll
    for (int i = 0; i < (int)GROUP; i++) {
        uint32_t c[2 * KEY_COLUMNS];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
            "%15}, [%16];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]),
              "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15])
            : "r"(from + i * 2 * KEY_COLUMNS)
            : "memory");
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t* k = c + j * KEY_COLUMNS;
            const uint32_t t0 = k[4] + (k[3] >> 8), t1 = k[5] + (t0 >> 8), t2 = k[6] + (t1 >> 8), t3 = k[7] + (t2 >> 8);
            const uint32_t low = k[0] + (k[1] << 8) + (k[2] << 16) + 19u * (t3 >> 8);
            slot[2 * i + j] = prefix_slot(sink, low);
            hits |= (t1 & t2 & t3 & 255u) == 255u ? 1u << (2 * i + j) : 0u;
            // the top limb down to bit 231
            if (Suffixes) top[2 * i + j] = (t3 & 255u) << 23 | (t2 & 255u) << 15 | (t1 & 255u) << 7;
        }
    }
    if (!Suffixes || sink.bitmap) {
        uint32_t word[KEYS];
#pragma unroll
        for (int k = 0; k < KEYS; k++) word[k] = sink.bitmap[slot[k] >> 5];
#pragma unroll
        for (int k = 0; k < KEYS; k++) hits |= (word[k] >> (slot[k] & 31) & 1u) << k;
    }
    if (Suffixes) {
#pragma unroll
        for (int k = 0; k < KEYS; k++)
            hits |= suffix_hit(sink, 0u, top[k]) | suffix_hit(sink, 0u, (top[k] + 128u) & 0x7fffffffu) ? 1u << k : 0u;
        // a 24-bit slot's bit 23 is the key's bit 224, which the sums do not give
        if (sink.sbits > 23) {
#pragma unroll
            for (int k = 0; k < KEYS; k++)
                hits |= suffix_hit(sink, 0u, top[k] | 1u) | suffix_hit(sink, 0u, ((top[k] + 128u) & 0x7fffffffu) | 1u)
                            ? 1u << k
                            : 0u;
        }
    }
    const uint32_t entries = min(GROUP, half - m0 + 1);
    hits &= active ? (1u << (2 * entries)) - 1u : 0u;
    const uint4* row = sh.rows + threadIdx.x;
    // Each lane pushes a hit of its own at a time, whichever keys they are: at
    // 5 % of candidates surviving that is two pushes a group where one per key
    // was five (22.0 ms for 7.8e8 candidates, now 20.3; 1.9e8 at 0.95 % 4.17,
    // now 3.98), and the shorter loop gave 2 % at any density.
    while (__any_sync(FULL, hits != 0)) {
        const uint32_t key = __ffs(hits) - 1, m = m0 + key / 2;
        stage_push(sink, tab, st, hits != 0, row, X, lane, key & 1u ? mid - m : mid + m, key & 1u ? m | 0x80000000u : m);
        hits &= hits - 1;
    }
}

// Whether a centre has order four: its y is 0 modulo p.
__device__ __forceinline__ bool order_four(const fe& y) {
    const fe v = fe_canon(y);
    return (v.v[0] | v.v[1] | v.v[2] | v.v[3] | v.v[4] | v.v[5] | v.v[6] | v.v[7]) == 0;
}

// What a lane's round keeps for its second pass.
struct RoundState {
    fe X, e, I;
};

// The part of a round between its passes: the inversion, e = c / z and
// I = 1 / prod E, and the next centre. The stride is added by the complete
// addition: with k = d x y xW yW, x(P + W) = (x yW + y xW) / (1 + k) and
// y(P + W) = (y yW + x xW) / (1 - k); 1 - k^2 joins the inversion.
__device__ __forceinline__ void turn_round(RoundState& s, const fe& x, const fe& y, const fe& z, const fe& run,
                                           uint4* centre, size_t cstride, bool active, const Stride& w) {
    const fe k = fe_mulv(fe_mulv(x, y), words_fe(w.dt));
    const fe one_k2 = fe_sub(fe_one(), fe_sqv(k));
    const fe total = fe_mulv(fe_mulv(run, z), one_k2);
    const fe U = block_invert(total);
    const fe a = fe_mulv(U, one_k2);
    s.e = fe_mulv(fe_mulv(const_inv_d_plus_1(), x), fe_mulv(a, run));
    s.I = fe_mulv(fe_sqv(z), a);
    const fe inv = fe_mulv(run, fe_mulv(z, U));  // 1 / (1 - k^2)
    const fe nx = fe_mulv(fe_add(fe_mulv(x, words_fe(w.y)), fe_mulv(y, words_fe(w.x))),
                          fe_mulv(fe_sub(fe_one(), k), inv));
    const fe ny = fe_mulv(fe_add(fe_mulv(y, words_fe(w.y)), fe_mulv(x, words_fe(w.x))),
                          fe_mulv(fe_add(fe_one(), k), inv));
    if (active) {
        store_fe(centre, cstride, nx);
        store_fe(centre + 2 * cstride, cstride, ny);
    }
}

// A block's `rounds` paired rounds, a lane each, against bitmaps of at most 24
// bits (sink_kind); see kernels.cuh for the candidate numbering. `centre` points
// at the lane's affine centre in the lane state (x, then y, 16-byte halves
// `cstride` apart), which is left on the centre after the last round: `between`
// is the stride after every round but the last, `last` the stride after that
// one. `scr` is the thread's column of its CTA's scratch: group j's prefix
// product, then E, half q at scr + (4 j + 2 e + q) SCRATCH_ROW. With Ahead, a
// group's two are read a group ahead, under the five multiplications of the one
// before, at the cost of 16 registers: the engine's kernel 50.3 -> 49.8 ms for
// 3.1e9 candidates (prefetch hints to L1 or L2 instead: 51.0); the batched one,
// with less to spare, ran some mixes 1 % faster and others 3.34 -> 3.57 ms a
// step, and the no-allocation one 1.68 -> 1.72 ms a call, so they go without. A
// thread that is not `active` has no lane: it takes part with another's centre
// and reports nothing. Every thread of the block calls it together, between
// matrix_open and matrix_close.
template <bool Suffixes, bool Ahead, bool AnyStart>
__device__ __forceinline__ void paired_rounds(uint4* centre, size_t cstride, const Stride& between, const Stride& last,
                                              const PairTable& tab, uint32_t half, uint32_t rounds, uint4* scr,
                                              const Sink& sink, RoundShared& sh, MatrixUnit& mu, uint32_t lane,
                                              bool active) {
    const uint32_t slots = 2 * half + 1, groups = groups_of(half);
    uint4* const row = sh.rows + threadIdx.x;
    WarpStage st{sh.stage + threadIdx.x / 32 * STAGE_RECORDS * STAGE_WORDS, 0};
    for (uint32_t r = 0; r < rounds; r++) {
        RoundState s;
        const uint32_t mid = r * slots + half;
        bool four;
        if (threadIdx.x == 0 && !sh.failed) fetch_constants(sh, tab.constants + (size_t)(groups - 1) * GROUP_CONSTANTS);
        {
            const fe x = load_fe(centre, cstride), y = load_fe(centre + 2 * cstride, cstride);
            s.X = fe_sqv(x);
            four = AnyStart && order_four(y);
            const fe X2 = fe_sqv(s.X), z = select_fe(four, fe_one(), fe_mulv(y, fe_sub(const_inv_d(), s.X)));
            fe run = z;
#pragma unroll 1
            for (uint32_t j = 0; j < groups; j++) {
                const uint4* t = tab.cubic + (size_t)j * 6;
                uint4* const p = scr + (size_t)j * (4 * SCRATCH_ROW);
                store_fe(p, SCRATCH_ROW, run);
                const fe E = fe_add(fe_mulv(fe_add(X2, load_fe(t + 2, 1)), fe_sub(load_fe(t, 1), s.X)),
                                    load_fe(t + 4, 1));
                store_fe(p + 2 * SCRATCH_ROW, SCRATCH_ROW, E);
                run = fe_mulv(run, E);
            }
            turn_round(s, x, y, z, run, centre, cstride, active, r + 1 < rounds ? between : last);
            // the centre's own key: its low limb is exact with bit 255
            // folded, unless y is p or more, and its high limbs unless the
            // fold carries that far
            bool hit = (y.v[7] & 0x7fffffffu) == 0x7fffffffu || (Suffixes && y.v[1] == 0xffffffffu);
            if (!Suffixes || sink.bitmap) hit |= prefix_hit(sink, y.v[0] + ((y.v[7] >> 31) ? 19u : 0u));
            if (Suffixes) hit |= suffix_hit(sink, y.v[6], y.v[7] & 0x7fffffffu);
            hit &= active;
            store_row(row, 0, y);
            stage_push(sink, tab, st, hit, row, s.X, lane, mid, 0u);
        }
        fe P, E;
        const auto load_group = [&](uint32_t j) {
            const uint4* p = scr + (size_t)j * (4 * SCRATCH_ROW);
            P = load_fe(p, SCRATCH_ROW);
            E = load_fe(p + 2 * SCRATCH_ROW, SCRATCH_ROW);
        };
        if (Ahead) load_group(groups - 1);
#pragma unroll 1
        for (uint32_t j = groups; j-- > 0;) {
            if (!Ahead) load_group(j);
            const fe h = fe_mulv(P, s.I);
            s.I = fe_mulv(s.I, E);
            if (j + 1 < groups) {
                // the product of the group before, which ran meanwhile
                finish_product(sh, sink, mu);
                if (threadIdx.x == 0 && !sh.failed) fetch_constants(sh, tab.constants + (size_t)j * GROUP_CONSTANTS);
                test_group<Suffixes>(sh, sink, tab, st, s.X, lane, active, mid, (j + 1) * GROUP + 1, half);
            }
            if (Ahead && j > 0) load_group(j - 1);
            store_row(row, 0, h);
            store_row(row, 3, fe_mulv(s.e, h));
            const fe g1 = fe_mulv(s.X, h);
            store_row(row, 1, g1);
            store_row(row, 4, fe_mulv(s.e, g1));
            const fe g2 = fe_mulv(s.X, g1);
            store_row(row, 2, g2);
            store_row(row, 5, fe_mulv(s.e, g2));
            if (AnyStart && four) {
                for (uint32_t k = 0; k < 3; k++) store_row(row, k, fe_zero());
            }
            start_product(sh, sink, mu);
        }
        finish_product(sh, sink, mu);
        test_group<Suffixes>(sh, sink, tab, st, s.X, lane, active, mid, 1, half);
    }
    stage_flush(sink, tab, st.recs, st.n);
}

// The same rounds with every key computed in full: for sinks with wider bitmaps
// than paired_rounds reads, or with none (every candidate survives), and for any
// start. A pair takes six multiplications: per pair the prefix product, w = P I
// [= z / D], I <- I D, f = e w and y = v w +- s f. 3.9e8 candidates against a
// bitmap of 25 bits 13.4 ms, of 24 bits by paired_rounds 6.9.
template <bool AnyStart>
__device__ __forceinline__ void paired_rounds_full(uint4* centre, size_t cstride, const Stride& between,
                                                   const Stride& last, const PairTable& tab, uint32_t half,
                                                   uint32_t rounds, uint4* scr, const Sink& sink, uint32_t lane,
                                                   bool active) {
    const uint32_t slots = 2 * half + 1;
    for (uint32_t r = 0; r < rounds; r++) {
        RoundState s;
        const uint32_t mid = r * slots + half;
        bool four;
        {
            const fe x = load_fe(centre, cstride), y = load_fe(centre + 2 * cstride, cstride);
            s.X = fe_sqv(x);
            four = AnyStart && order_four(y);
            const fe z = select_fe(four, fe_one(), fe_mulv(y, fe_sub(const_inv_d(), s.X)));
            fe run = z;
#pragma unroll 1
            for (uint32_t m = 0; m < half; m++) {
                store_fe(scr + (size_t)m * (2 * SCRATCH_ROW), SCRATCH_ROW, run);
                run = fe_mulv(run, fe_sub(load_fe(tab.q + (size_t)m * 2, 1), s.X));
            }
            turn_round(s, x, y, z, run, centre, cstride, active, r + 1 < rounds ? between : last);
            test_emit(sink, y, lane, mid, active);
        }
#pragma unroll 1
        for (uint32_t m = half; m >= 1; m--) {
            const fe w = fe_mulv(load_fe(scr + (size_t)(m - 1) * (2 * SCRATCH_ROW), SCRATCH_ROW), s.I);
            s.I = fe_mulv(s.I, fe_sub(load_fe(tab.q + (size_t)(m - 1) * 2, 1), s.X));
            const uint4* t = tab.vs + (size_t)(m - 1) * 4;
            const fe B = fe_mulv(load_fe(t + 2, 1), fe_mulv(s.e, w));
            fe A = fe_mulv(load_fe(t, 1), w);
            if (AnyStart && four) A = fe_zero();
#pragma unroll 1
            for (uint32_t sign = 0; sign < 2; sign++)
                test_emit(sink, sign ? fe_sub(A, B) : fe_add(A, B), lane, sign ? mid - m : mid + m, active);
        }
    }
}

// p (extended) plus k times the point of a Pow2Table, k < 2^POW2.
__device__ __forceinline__ void add_multiple(fe& X, fe& Y, fe& Z, fe& T, const Pow2Table& table, uint32_t k) {
    for (const uint4* p = table.v; k; k >>= 1, p += 6)
        if (k & 1u) add_cached(X, Y, Z, T, load_fe(p + 0, 1), load_fe(p + 2, 1), load_fe(p + 4, 1));
}

// Entry m of the per-entry part of a PairTable of `n` entries, Q_m+1 = 8 (m + 1) G
// from the Pow2Table of 8G, m the thread's number. Every thread of the block calls
// it; those past the table write nothing.
__device__ __forceinline__ void fill_pair_entry(const PairTable& tab, uint32_t n, const Pow2Table& eight, uint32_t thread) {
    const uint32_t m = min(thread, n - 1);
    fe X = fe_zero(), Y = fe_one(), Z = fe_one(), T = fe_zero();
    add_multiple(X, Y, Z, T, eight, m + 1);
    // of the affine (x, y): v = 1/y = Z (Z^2 + X^2) i, s = x / (1 + x^2) = X Y Z i and
    // q = v^2 / d, with i = 1 / (Y (Z^2 + X^2)); y and 1 + x^2 are never 0 for a point
    // of odd order
    const fe den = fe_add(fe_sqv(Z), fe_sqv(X));
    const fe zi = fe_mulv(Z, block_invert(fe_mulv(Y, den)));
    const fe v = fe_canon(fe_mulv(den, zi));
    if (thread >= n) return;
    store_fe(const_cast<uint4*>(tab.q) + (size_t)m * 2, 1, fe_canon(fe_mulv(fe_sqv(v), const_inv_d())));
    uint4* const vs = const_cast<uint4*>(tab.vs) + (size_t)m * 4;
    store_fe(vs + 0, 1, v);
    store_fe(vs + 2, 1, fe_canon(fe_mulv(fe_mulv(X, Y), zi)));
}

// The affine centre of lane `lane`: a base point (extended) plus that many times
// the point of a Pow2Table. Every thread of the block calls it.
__device__ __forceinline__ void first_centre(fe X, fe Y, fe Z, fe T, const Pow2Table& stride, uint32_t lane,
                                             uint4* lanes, uint32_t lanes_n) {
    const size_t L = lanes_n;
    add_multiple(X, Y, Z, T, stride, lane);
    const fe zi = block_invert(Z);  // Z is never 0
    if (lane < lanes_n) {
        store_fe(lanes + 0 * L + lane, L, fe_mulv(X, zi));
        store_fe(lanes + 2 * L + lane, L, fe_mulv(Y, zi));
    }
}

// Fills the per-group part of a PairTable from its q, v and s, one thread for
// each (group, key, element) of six keys and six elements; the threads of
// element 0 and key 0 write the cubic. `tab` is the table being written.
__device__ inline void fill_group_table(const PairTable& tab, uint32_t groups, uint32_t thread) {
    const uint32_t g = thread / 36, key = thread / 6 % 6, elem = thread % 6;
    if (g >= groups) return;
    const uint32_t i = key / 2;  // the key's pair
    fe q[GROUP];
    for (uint32_t j = 0; j < GROUP; j++) q[j] = load_fe(tab.q + (size_t)(g * GROUP + j) * 2, 1);
    if (key == 0 && elem == 0) {
        const fe s1 = fe_add(fe_add(q[0], q[1]), q[2]), q01 = fe_mulv(q[0], q[1]);
        const fe s2 = fe_add(q01, fe_mulv(q[2], fe_add(q[0], q[1])));
        uint4* const t = const_cast<uint4*>(tab.cubic) + (size_t)g * 6;
        store_fe(t, 1, s1);
        store_fe(t + 2, 1, s2);
        store_fe(t + 4, 1, fe_sub(fe_mulv(q01, q[2]), fe_mulv(s1, s2)));
    }
    const uint4* vs = tab.vs + (size_t)(g * GROUP + i) * 4;
    const fe zero = fe_zero(), qa = q[(i + 1) % GROUP], qb = q[(i + 2) % GROUP];
    fe c = load_fe(elem < 3 ? vs : vs + 2, 1);
    if (elem % 3 == 0) c = fe_mulv(c, fe_mulv(qa, qb));
    if (elem % 3 == 1) c = fe_sub(zero, fe_mulv(c, fe_add(qa, qb)));
    if (elem >= 3 && (key & 1)) c = fe_sub(zero, c);
    uint32_t* const out = reinterpret_cast<uint32_t*>(const_cast<uint4*>(tab.constants) + (size_t)g * GROUP_CONSTANTS);
    const fe times256 = fe{{256u, 0u, 0u, 0u, 0u, 0u, 0u, 0u}};
    for (uint32_t word = 0; word < 8; word++) {
        uint32_t col[KEY_COLUMNS] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (uint32_t byte = 0; byte < 4; byte++) {
            const fe rho = fe_canon(c);
            // floor(2^40 rho / p), or one less
            const uint64_t frac = (((uint64_t)rho.v[7] << 32) | rho.v[6]) >> 23;
            for (uint32_t n = 0; n < 3; n++) col[n] |= (rho.v[0] >> (8 * n) & 255u) << (8 * byte);
            for (uint32_t n = 0; n < 5; n++) col[3 + n] |= (uint32_t)(frac >> (8 * n) & 255u) << (8 * byte);
            c = fe_mulv(c, times256);
        }
        for (uint32_t n = 0; n < KEY_COLUMNS; n++)
            out[((elem * 2 + word / 4) * COLUMNS + key * KEY_COLUMNS + n) * 4 + word % 4] = col[n];
    }
}

}  // namespace og
