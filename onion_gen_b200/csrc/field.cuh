// GF(2^255-19) on sm_100a: eight 32-bit limbs, least significant first.
//
// Every value is held below 2^256 and congruent to the field element; only
// fe_canon() produces the unique representative below p. Multiplication and
// squaring are exact 32x32->64 partial products on the integer multiply-add
// pipe with PTX carry chains (field_asm.cuh); addition and subtraction are
// carry chains on the integer ALU, folded with 2^256 = 38 (mod p).
//
// The representation and folding constant follow the arithmetic of
// src/field.rs (radix 2^64 there, radix 2^32 here) and the device field of
// cuda-kernel/src/field_asm.rs; the code is written for this engine.
#pragma once
#include <cstdint>

#include "field_asm.cuh"

struct fe {
    uint32_t v[8];
};

#define OG_FE_MUL_ASM fe_mul_asm

__device__ __forceinline__ void fe_mul(fe& r, const fe& a, const fe& b) { OG_FE_MUL_ASM(r.v, a.v, b.v); }
__device__ __forceinline__ void fe_sq(fe& r, const fe& a) { fe_sq_asm(r.v, a.v); }

__device__ __forceinline__ fe fe_mulv(const fe& a, const fe& b) {
    fe r;
    OG_FE_MUL_ASM(r.v, a.v, b.v);
    return r;
}

__device__ __forceinline__ fe fe_sqv(const fe& a) {
    fe r;
    fe_sq_asm(r.v, a.v);
    return r;
}

// r = a + b. A carry out of bit 256 is worth 38; a second fold cannot carry.
__device__ __forceinline__ fe fe_add(const fe& a, const fe& b) {
    fe r;
    asm("{\n\t.reg .u32 c, m;\n\t"
        "add.cc.u32 %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.cc.u32 %7, %15, %23;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "neg.s32 m, c;\n\t"
        "and.b32 m, m, 38;\n\t"
        "add.cc.u32 %0, %0, m;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\t"
        "addc.cc.u32 %7, %7, 0;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "neg.s32 m, c;\n\t"
        "and.b32 m, m, 38;\n\t"
        "add.u32 %0, %0, m;\n\t"
        "}"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
          "=r"(r.v[6]), "=r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
          "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]));
    return r;
}

// r = a - b. A borrow out of the top means the value wrapped by 2^256, which
// is worth 38, so 38 is taken off again; a second borrow leaves the value near
// 2^256 and the third subtraction cannot borrow.
__device__ __forceinline__ fe fe_sub(const fe& a, const fe& b) {
    fe r;
    asm("{\n\t.reg .u32 c, m;\n\t"
        "sub.cc.u32 %0, %8, %16;\n\t"
        "subc.cc.u32 %1, %9, %17;\n\t"
        "subc.cc.u32 %2, %10, %18;\n\t"
        "subc.cc.u32 %3, %11, %19;\n\t"
        "subc.cc.u32 %4, %12, %20;\n\t"
        "subc.cc.u32 %5, %13, %21;\n\t"
        "subc.cc.u32 %6, %14, %22;\n\t"
        "subc.cc.u32 %7, %15, %23;\n\t"
        "subc.u32 c, 0, 0;\n\t"
        "and.b32 m, c, 38;\n\t"
        "sub.cc.u32 %0, %0, m;\n\t"
        "subc.cc.u32 %1, %1, 0;\n\t"
        "subc.cc.u32 %2, %2, 0;\n\t"
        "subc.cc.u32 %3, %3, 0;\n\t"
        "subc.cc.u32 %4, %4, 0;\n\t"
        "subc.cc.u32 %5, %5, 0;\n\t"
        "subc.cc.u32 %6, %6, 0;\n\t"
        "subc.cc.u32 %7, %7, 0;\n\t"
        "subc.u32 c, 0, 0;\n\t"
        "and.b32 m, c, 38;\n\t"
        "sub.u32 %0, %0, m;\n\t"
        "}"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
          "=r"(r.v[6]), "=r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
          "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]));
    return r;
}

// a + c for a small c, carried through all limbs; the caller guarantees
// that the sum stays below 2^256.
__device__ __forceinline__ fe fe_add_small(const fe& a, uint32_t c) {
    fe r;
    asm("add.cc.u32 %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, 0;\n\t"
        "addc.cc.u32 %2, %10, 0;\n\t"
        "addc.cc.u32 %3, %11, 0;\n\t"
        "addc.cc.u32 %4, %12, 0;\n\t"
        "addc.cc.u32 %5, %13, 0;\n\t"
        "addc.cc.u32 %6, %14, 0;\n\t"
        "addc.u32 %7, %15, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
          "=r"(r.v[6]), "=r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
          "r"(a.v[7]), "r"(c));
    return r;
}

// The unique representative below p = 2^255 - 19.
// Bit 255 is folded first (2^255 = 19), which leaves a value below
// 2^255 + 19; then q = (v + 19) >> 255 says whether one p comes off, and
// v - q p = (v + 19 q) mod 2^255.
__device__ __forceinline__ fe fe_canon(const fe& a) {
    fe v = a;
    const uint32_t top = v.v[7] >> 31;
    v.v[7] &= 0x7fffffffu;
    v = fe_add_small(v, top * 19u);
    fe s = fe_add_small(v, 19u);
    const bool q = (s.v[7] >> 31) != 0;
    s.v[7] &= 0x7fffffffu;
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = q ? s.v[k] : v.v[k];
    return r;
}

__device__ __forceinline__ fe fe_zero() { return fe{{0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u}}; }

__device__ __forceinline__ fe fe_one() {
    fe r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.v[k] = k == 0 ? 1u : 0u;
    return r;
}

// x^-1 modulo p (0 for a multiple of p), by division steps (Bernstein and Yang,
// "Fast constant-time gcd computation and modular inversion", 2019), until g is
// 0. The pair (f, g) starts as (p, x); a step with g even halves g;
// with g odd it first takes g + f, or, when delta > 0, (f, g) <- (g, g - f) and
// delta <- -delta; every halving adds one to delta. 742 steps bring any x below
// 2^256 to g = 0, f = +-gcd; a random one takes some 540. Thirty steps at a time
// are decided by the low words alone and gathered in a matrix (u v; q r), which
// then goes onto (f, g), exactly divisible by 2^30, and onto (d, e) from (0, 1),
// divisible after adding a multiple of p, so that d x = f (mod p) throughout.
// Numbers are nine signed limbs of 30 bits, the layout of libsecp256k1's 32-bit
// modular inversion, of which the names of the matrix and the sums are too; p =
// 2^15 2^240 - 19 has two of them.
// |d| and |e| grow by at most p / 2 in thirty steps, below 13 p. One thread's
// latency is what counts (block_invert): on B200 29 000 clocks (35 000 with the
// steps' zeros counted instead of taken one by one), the power x^(p - 2) by 254
// squarings and 11 multiplications 90 000.
static __device__ __noinline__ fe fe_invert(const fe& x) {
    constexpr int32_t M30 = 0x3fffffff;
    constexpr uint32_t NEG_INV_P = 0x286bca1bu;  // -1/p modulo 2^30
    int32_t f[9], g[9], d[9], e[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const int w = 30 * i / 32, sh = 30 * i % 32;
        const uint32_t hi = sh > 2 && w < 7 ? x.v[w + 1] : 0u;
        f[i] = i == 0 ? M30 - 18 : i < 8 ? M30 : 0x7fff;
        g[i] = (int32_t)(__funnelshift_r(x.v[w], hi, sh) & M30);
        d[i] = 0;
        e[i] = i == 0;
    }
    int32_t delta = 1;
#pragma unroll 1
    for (int batch = 0; batch < 25; batch++) {
        int32_t any = 0;
#pragma unroll
        for (int i = 0; i < 9; i++) any |= g[i];
        if (any == 0) break;
        int32_t u = 1, v = 0, q = 0, r = 1;
        uint32_t fw = (uint32_t)f[0] | (uint32_t)f[1] << 30, gw = (uint32_t)g[0] | (uint32_t)g[1] << 30;
        // every step the same instructions: a single thread sees each branch and
        // each count of zeros at its full latency
#pragma unroll 10
        for (int step = 0; step < 30; step++) {
            const bool odd = gw & 1u, swap = odd && delta > 0;
            const int32_t sign = odd ? (delta > 0 ? -1 : 1) : 0;
            const uint32_t nf = swap ? gw : fw;
            const int32_t nu = swap ? q : u, nv = swap ? r : v;
            gw = (gw + (uint32_t)sign * fw) >> 1;
            q += sign * u;
            r += sign * v;
            fw = nf;
            u = nu << 1;
            v = nv << 1;
            delta = (swap ? -delta : delta) + 1;
        }
        int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0], cg = (int64_t)q * f[0] + (int64_t)r * g[0];
        int64_t cd = (int64_t)u * d[0] + (int64_t)v * e[0], ce = (int64_t)q * d[0] + (int64_t)r * e[0];
        // the multiples of p that make the sums divisible, from -2^29 on
        const int32_t md = (int32_t)((uint32_t)cd * NEG_INV_P << 2) >> 2, me = (int32_t)((uint32_t)ce * NEG_INV_P << 2) >> 2;
        cf >>= 30;
        cg >>= 30;
        cd = (cd - (int64_t)19 * md) >> 30;
        ce = (ce - (int64_t)19 * me) >> 30;
#pragma unroll
        for (int i = 1; i < 9; i++) {
            cf += (int64_t)u * f[i] + (int64_t)v * g[i];
            cg += (int64_t)q * f[i] + (int64_t)r * g[i];
            cd += (int64_t)u * d[i] + (int64_t)v * e[i] + (i == 8 ? (int64_t)32768 * md : 0);
            ce += (int64_t)q * d[i] + (int64_t)r * e[i] + (i == 8 ? (int64_t)32768 * me : 0);
            f[i - 1] = (int32_t)cf & M30;
            g[i - 1] = (int32_t)cg & M30;
            d[i - 1] = (int32_t)cd & M30;
            e[i - 1] = (int32_t)ce & M30;
            cf >>= 30;
            cg >>= 30;
            cd >>= 30;
            ce >>= 30;
        }
        f[8] = (int32_t)cf;
        g[8] = (int32_t)cg;
        d[8] = (int32_t)cd;
        e[8] = (int32_t)ce;
    }
    // f is 1 or -1, unless x is a multiple of p
    const int32_t sign = f[8] >> 31;
    int32_t other = (f[0] ^ (sign & M30)) ^ (sign ? 0 : 1);
#pragma unroll
    for (int i = 1; i < 8; i++) other |= f[i] ^ (sign & M30);
    other |= f[8] ^ sign;
    // +-d + 16 p, from 0 to 2^260: limbs back to 0..2^30 - 1
    uint32_t w[9];
    int64_t c = -16 * 19;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        c += (d[i] ^ sign) - sign + (i == 8 ? 16 * 32768 : 0);
        w[i] = i == 8 ? (uint32_t)c : (uint32_t)c & M30;
        c >>= 30;
    }
    fe r, top;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int i = 32 * k / 30, sh = 32 * k % 30;  // word k starts in limb i at bit sh
        uint64_t bits = (uint64_t)w[i] >> sh | (uint64_t)w[i + 1] << (30 - sh);
        if (i + 2 < 9) bits |= (uint64_t)w[i + 2] << (60 - sh);
        r.v[k] = other ? 0u : (uint32_t)bits;
        top.v[k] = 0;
    }
    top.v[0] = other ? 0u : 38u * (w[8] >> 16);
    return fe_add(r, top);
}
