// Device building blocks shared by the single-search and the batched
// kernels: device-layout loads and stores, the survivor test and append, the
// cached point addition, and one lane's paired rounds.
#pragma once
#include "field.cuh"
#include "kernels.cuh"

namespace og {

constexpr unsigned FULL = 0xffffffffu;

#ifndef OG_LB_THREADS
#define OG_LB_THREADS 128  // the most threads a block of the search kernels has
#endif

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
    const uint32_t* bitmap;
    uint32_t bits;
    HitRec* hits;
    uint32_t* counter;
    uint32_t cap;
    uint32_t search;
    const uint32_t* sbitmap;  // suffix bitmap, or nullptr
    uint32_t sbits;
    // the prefix bitmap is read from the block's copy in shared memory
    // (og_bitmap_s, staged by the kernel), not through L1
    bool staged = false;
};

// Prefix bitmaps of at most this many bits (8 KiB) can be staged in shared
// memory by a kernel that sets Sink::staged.
constexpr uint32_t STAGED_BITMAP_BITS = 16;

// Slot of a canonical key in the suffix bitmap: base32 bits
// [255 - sbits, 255) of the packed key, i.e. bits 1..sbits of its last eight
// bytes read big-endian (BitmapIndex::slot with offset 255 - sbits,
// src/filter.rs:2536-2549). The sign bit (bit 7 of byte 31) is clear in the
// packed key and the bitmap holds both of its values.
__device__ __forceinline__ uint32_t suffix_slot(const fe& y, uint32_t sbits) {
    const uint32_t lo = __byte_perm(y.v[7], 0, 0x0123), hi = __byte_perm(y.v[6], 0, 0x0123);
    const uint32_t w = (lo >> 1) | (hi << 31);
    return sbits >= 32 ? w : w & ((1u << sbits) - 1u);
}

// Whether the slot of a key whose canonical low limb is `y0` is set in the
// sink's prefix bitmap: bytes 0..3 of the key, big-endian, are the top of the
// slot.
__device__ __forceinline__ bool prefix_hit(const Sink& k, uint32_t y0) {
    const uint32_t head = __byte_perm(y0, 0, 0x0123);
    const uint32_t slot = k.bits >= 32 ? head : head >> (32 - k.bits);
    if (k.staged) {
        extern __shared__ uint32_t og_bitmap_s[];
        return (og_bitmap_s[slot >> 5] >> (slot & 31)) & 1u;
    }
    return (__ldg(k.bitmap + (slot >> 5)) >> (slot & 31)) & 1u;
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
        if (k.sbitmap && valid) {
            const uint32_t slot = suffix_slot(y, k.sbits);
            hit |= ((__ldg(k.sbitmap + (slot >> 5)) >> (slot & 31)) & 1u) != 0;
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
// square, so no centre is exceptional; z is 0 only for the two centres of
// order four. With one inversion for the round's denominators (Montgomery's
// trick), the prefix products started from z and e = c / z, a pair costs
// four multiplications,
//
//     P_m = P_(m-1) (q - X),   w = P_(m-1) I  [= z / (q - X)],
//     I <- I (q - X),          f = e w,
//
// and y(P +- Q) = v w +- s f, of which only what the bitmap reads is
// computed (low_product below): about a third of a multiplication each.
// Only P_m is kept between the passes, 32 bytes a pair.

// The table of one half: q per entry (two uint4), then v and s per entry
// (four), in one array of 6 half uint4.
struct PairTable {
    const uint4* q;
    const uint4* vs;
};

__device__ __forceinline__ fe const_inv_d() {  // 1/d
    return fe{{0xcdc9f843u, 0x25e0f276u, 0x4279542eu, 0x0b5dd698u, 0xcdb9cf66u, 0x2b162114u, 0x14d5ce43u, 0x40907ed2u}};
}

__device__ __forceinline__ fe const_inv_d_plus_1() {  // 1 + 1/d
    return fe{{0xcdc9f844u, 0x25e0f276u, 0x4279542eu, 0x0b5dd698u, 0xcdb9cf66u, 0x2b162114u, 0x14d5ce43u, 0x40907ed2u}};
}

// What the low limb of a canonical product needs. With T = a b < 2^512 and
// k = floor(T / p), T mod p = T - k p, and p = -19 (mod 2^32), so its low
// limb is lo + 19 k with lo = a0 b0 (mod 2^32). T / p is
// T / 2^255 + 19 T / 2^510 (the next term is below 2^-240), so in units of
// 2^-31 it is the product's words 7 and 8 plus 38 times its word 15: `acc`
// holds these from the products of columns 7 and 8 (mod 2^64), the high
// halves of column 6 and the high half of a7 b7. What is left out: column
// 6's low halves (below 7), column 5 (below 6) and lower; 38 times the rest
// of word 15 (below 3.01): the true value is in [acc, acc + 128).
// About 21 multiply-add slots against 74 for the multiplication.
struct LowProduct {
    uint64_t acc;
    uint32_t lo;
};

constexpr uint32_t LOW_PRODUCT_ERROR = 128;

__device__ __forceinline__ LowProduct low_product(const fe& a, const fe& b) {
    uint64_t acc = 0, c6 = 0;
    uint32_t c8 = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) acc += (uint64_t)a.v[i] * b.v[7 - i];
#pragma unroll
    for (int i = 0; i < 7; i++) c6 += __umulhi(a.v[i], b.v[6 - i]);
#pragma unroll
    for (int i = 1; i < 8; i++) c8 += a.v[i] * b.v[8 - i];
    acc += c6 + 38ull * __umulhi(a.v[7], b.v[7]) + ((uint64_t)c8 << 32);
    return LowProduct{acc, a.v[0] * b.v[0]};
}

// Whether a key that is the sum (or difference) of two low products may be
// in the prefix bitmap: its low limb is exact unless the sum's uncertainty
// (2 LOW_PRODUCT_ERROR above `acc`) reaches the next k, once in 2^23 keys;
// those count as hits and are decided by the full product.
__device__ __forceinline__ bool low_may_hit(const Sink& k, uint64_t acc, uint32_t lo) {
    const uint32_t q = __funnelshift_l((uint32_t)acc, (uint32_t)(acc >> 32), 1);  // acc >> 31
    const bool unsure = ((uint32_t)acc & 0x7fffffffu) >= 0x80000000u - 2u * LOW_PRODUCT_ERROR;
    return unsure | prefix_hit(k, lo + 19u * q);
}

// Candidates that may survive, collected per warp in shared memory: w and f
// (64 bytes), the candidate's lane and step, and its table entry with the
// sign (0: the centre, whose y is w). stage_flush computes their keys with
// 32 lanes at once, tests them exactly and appends the survivors. The search
// loop itself holds neither the full products nor the record writes, and an
// index that passes one candidate in a hundred costs it no more than a rare
// one.
constexpr uint32_t STAGE_RECORDS = 32;
constexpr uint32_t STAGE_WORDS = 5;  // uint4 a record

struct WarpStage {
    uint4* recs;  // this warp's STAGE_RECORDS records in shared memory
    uint32_t n;   // records held; the same in every lane of the warp
};

static __device__ __noinline__ void stage_flush(const Sink& k, const uint4* vs, const uint4* recs, uint32_t n) {
    if (n == 0) return;
    __syncwarp();
    const unsigned me = threadIdx.x & 31u;
    const bool valid = me < n;
    const uint4* r = recs + (valid ? me : 0) * STAGE_WORDS;
    const fe w = load_fe(r, 1), f = load_fe(r + 2, 1);
    const uint4 id = r[4];
    const uint32_t m = id.z & 0x7fffffffu;
    const uint4* t = vs + (size_t)(m ? m - 1 : 0) * 4;
    const fe A = fe_mulv(load_fe(t, 1), w), B = fe_mulv(load_fe(t + 2, 1), f);
    const fe sum = fe_add(A, B), diff = fe_sub(A, B);
    const fe y = select_fe(m == 0, w, select_fe(id.z >> 31, diff, sum));
    test_emit(k, y, id.x, id.y, valid);
    __syncwarp();
}

// Adds the candidates of the warp's lanes with `hit` set.
__device__ __forceinline__ void stage_push(const Sink& k, const uint4* vs, WarpStage& st, bool hit, const fe& w,
                                           const fe& f, uint32_t lane, uint32_t step, uint32_t entry) {
    const unsigned mask = __ballot_sync(FULL, hit);
    if (mask == 0) return;
    const uint32_t count = (uint32_t)__popc(mask);
    if (st.n + count > STAGE_RECORDS) {
        stage_flush(k, vs, st.recs, st.n);
        st.n = 0;
    }
    if (hit) {
        uint4* r = st.recs + (st.n + (uint32_t)__popc(mask & ((1u << (threadIdx.x & 31u)) - 1u))) * STAGE_WORDS;
        store_fe(r, 1, w);
        store_fe(r + 2, 1, f);
        r[4] = make_uint4(lane, step, entry, 0u);
    }
    st.n += count;
}

// Rows of a CTA's scratch hold this many threads (the largest block).
constexpr uint32_t SCRATCH_ROW = OG_LB_THREADS;

// One lane's `rounds` paired rounds; see kernels.cuh for the candidate
// numbering. `centre` points at the lane's affine centre in the lane state
// (x, then y, 16-byte halves `cstride` apart), which is left on the centre
// after the last round. `wdt` is d xW yW of the stride W. `scr` is the
// thread's column of its CTA's scratch: prefix product m, half q at
// scr + (2 m + q) SCRATCH_ROW. Candidates that may survive go to `st`.
// OneInversion: one field inversion for the block's lanes (block_invert),
// else one a lane.
template <bool OneInversion>
__device__ __forceinline__ void paired_rounds(uint4* centre, size_t cstride, const FeWords& wx, const FeWords& wy,
                                              const FeWords& wdt, const PairTable& tab, uint32_t half, uint32_t rounds,
                                              uint4* scr, const Sink& sink, WarpStage& st, uint32_t lane) {
    const uint32_t slots = 2 * half + 1;
    const bool approx = sink.bitmap && !sink.sbitmap;
    for (uint32_t r = 0; r < rounds; r++) {
        fe X, e, I;
        const uint32_t mid = r * slots + half;
        {
            const fe x = load_fe(centre, cstride), y = load_fe(centre + 2 * cstride, cstride);
            X = fe_sqv(x);
            const fe z = fe_mulv(y, fe_sub(const_inv_d(), X));
            fe run = z;
#pragma unroll 1
            for (uint32_t m = 0; m < half; m++) {
                store_fe(scr + (size_t)m * (2 * SCRATCH_ROW), SCRATCH_ROW, run);
                run = fe_mulv(run, fe_sub(load_fe(tab.q + (size_t)m * 2, 1), X));
            }
            // the stride by the complete addition: with k = d x y xW yW,
            // x(P + W) = (x yW + y xW) / (1 + k), y(P + W) = (y yW + x xW) / (1 - k);
            // 1 - k^2 joins the round's inversion
            const fe k = fe_mulv(fe_mulv(x, y), words_fe(wdt));
            const fe E = fe_sub(fe_one(), fe_sqv(k));
            const fe total = fe_mulv(fe_mulv(run, z), E);  // z^2 E prod(q - X)
            const fe U = OneInversion ? block_invert(total) : fe_invert(total);
            const fe a = fe_mulv(U, E);
            e = fe_mulv(fe_mulv(const_inv_d_plus_1(), x), fe_mulv(a, run));  // c / z
            I = fe_mulv(fe_sqv(z), a);
            const fe invE = fe_mulv(run, fe_mulv(z, U));
            const fe nx = fe_mulv(fe_add(fe_mulv(x, words_fe(wy)), fe_mulv(y, words_fe(wx))),
                                  fe_mulv(fe_sub(fe_one(), k), invE));
            const fe ny = fe_mulv(fe_add(fe_mulv(y, words_fe(wy)), fe_mulv(x, words_fe(wx))),
                                  fe_mulv(fe_add(fe_one(), k), invE));
            store_fe(centre, cstride, nx);
            store_fe(centre + 2 * cstride, cstride, ny);
            // the centre's own key: its low limb is exact with bit 255
            // folded, unless y is p or more
            const bool hit = !approx || (y.v[7] & 0x7fffffffu) == 0x7fffffffu ||
                             prefix_hit(sink, y.v[0] + ((y.v[7] >> 31) ? 19u : 0u));
            stage_push(sink, tab.vs, st, hit, y, y, lane, mid, 0u);
        }
#pragma unroll 1
        for (uint32_t m = half; m >= 1; m--) {
            const fe w = fe_mulv(load_fe(scr + (size_t)(m - 1) * (2 * SCRATCH_ROW), SCRATCH_ROW), I);
            I = fe_mulv(I, fe_sub(load_fe(tab.q + (size_t)(m - 1) * 2, 1), X));
            const fe f = fe_mulv(e, w);
            bool plus = true, minus = true;
            if (approx) {
                const uint4* t = tab.vs + (size_t)(m - 1) * 4;
                const LowProduct A = low_product(load_fe(t, 1), w), B = low_product(load_fe(t + 2, 1), f);
                plus = low_may_hit(sink, A.acc + B.acc, A.lo + B.lo);
                minus = low_may_hit(sink, A.acc - B.acc - LOW_PRODUCT_ERROR, A.lo - B.lo);
            }
            if (__any_sync(FULL, plus | minus)) {
                stage_push(sink, tab.vs, st, plus, w, f, lane, mid + m, m);
                stage_push(sink, tab.vs, st, minus, w, f, lane, mid - m, m | 0x80000000u);
            }
        }
    }
}

}  // namespace og
