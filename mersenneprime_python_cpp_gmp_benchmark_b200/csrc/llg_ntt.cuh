// Arithmetic in GF(q), q = 2^64 - 2^32 + 1 ("Goldilocks"), and the in-register radix passes of
// the number-theoretic transforms (exact IBDWT; the reference's CUDA engine, cuda/ll_ntt.cu:38-61
// and 100-127, does the same field with radix-2 stages and a 128-bit-free u64 multiply).
//
// The integer ALU bounds these kernels (a 32-bit add, shift or select takes 2 cycles of a warp
// scheduler's ALU, multiply-adds issue beside them), so every primitive is written for the fewest
// 32-bit ALU instructions:
//   * products are Montgomery products a b 2^-64 mod q (mul). With q = 2^64 - 2^32 + 1 the
//     reduction needs no multiplication: for X = a b = xh 2^64 + r1 2^32 + r0 and
//     t + e 2^32 = r0 + r1, X 2^-64 == xh + r1 - (t 2^32 + e (2^32 - 1)), one 64-bit difference with
//     one correction. Every constant (twiddles, weights) is stored as c 2^64 mod q ("Montgomery
//     form"), so mul(value, constant) is the plain product and the values themselves stay plain.
//     29 cycles a warp product per scheduler, against 41 with the 128-bit reduction it replaces;
//   * a sum is a difference with the negative (add), canonical without a compare;
//   * 2 has order 192, so w_8 = 7^((q-1)/8) = 2^120 and w_4 = 2^48: the twiddles inside a radix-8
//     butterfly are shifts with their own short reductions (rot24, rot48, rot72). A radix-8
//     butterfly takes 41 cycles a value, against 63 before.
// "any" below means any 64-bit value standing for itself mod q; canonical means < q.
#pragma once

#include <cstdint>

namespace llg {
namespace gl {

constexpr uint64_t Q = 0xFFFFFFFF00000001ull;
constexpr uint64_t ONE = 0xFFFFFFFFull;           // 2^64 mod q: 1 in Montgomery form
constexpr uint64_t HALF = 0x8000000000000000ull;  // 2^63: 1/2 in Montgomery form

// a - b for any a and b <= q: on a borrow, a - b + 2^64 - (2^32 - 1) = a - b + q. The result is
// canonical when a is.
__device__ __forceinline__ uint64_t sub(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("{\n\t.reg .u32 a0, a1, b0, b1, m;\n\t"
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "sub.cc.u32 a0, a0, b0;\n\t"
        "subc.cc.u32 a1, a1, b1;\n\t"
        "subc.u32 m, 0, 0;\n\t"  // 0, or 0xFFFFFFFF = 2^64 - q after a borrow
        "sub.cc.u32 a0, a0, m;\n\t"
        "subc.u32 a1, a1, 0;\n\t"
        "mov.b64 %0, {a0, a1};\n\t}"
        : "=l"(r)
        : "l"(a), "l"(b));
    return r;
}

// a + b for any a and canonical b: a - (q - b); canonical when a is.
__device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) { return sub(a, Q - b); }

// Montgomery product a b 2^-64 mod q; canonical when a or b is (then xh <= q - 1, so xh + r1 does
// not overflow), any otherwise excluded: one operand must be canonical.
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
    const uint64_t lo = a * b, hi = __umul64hi(a, b);
    uint64_t r;
    asm("{\n\t.reg .u32 r0, r1, r2, r3, t, m, e;\n\t"
        "mov.b64 {r0, r1}, %1;\n\t"
        "mov.b64 {r2, r3}, %2;\n\t"
        "add.cc.u32 t, r1, r0;\n\t"
        "addc.u32 e, 0, 0;\n\t"
        "neg.s32 e, e;\n\t"
        "add.cc.u32 r2, r2, r1;\n\t"
        "addc.u32 r3, r3, 0;\n\t"
        "sub.cc.u32 r2, r2, e;\n\t"
        "subc.cc.u32 r3, r3, t;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 r2, r2, m;\n\t"
        "subc.u32 r3, r3, 0;\n\t"
        "mov.b64 %0, {r2, r3};\n\t}"
        : "=l"(r)
        : "l"(lo), "l"(hi));
    return r;
}

// x 2^24, canonical for any x: x 2^24 = lo + h 2^64 with h < 2^24, and -h 2^64 == q - h (2^32 - 1)
// = (~h) 2^32 + h + 1 takes two instructions.
__device__ __forceinline__ uint64_t rot24(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32), h = x1 >> 8;
    const uint64_t lo = ((uint64_t)__funnelshift_l(x0, x1, 24) << 32) | (x0 << 24);
    return sub(lo, ((uint64_t)(~h) << 32) | (h + 1u));
}

// x 2^48, canonical for any x: 2^48 == -2^16 2^-64, the negated Montgomery reduction of x 2^16.
__device__ __forceinline__ uint64_t rot48(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    uint64_t r;
    asm("{\n\t.reg .u32 t, e, m, y0, y1;\n\t"
        "add.cc.u32 t, %2, %1;\n\t"
        "addc.u32 e, 0, 0;\n\t"
        "neg.s32 e, e;\n\t"
        "add.cc.u32 y0, %3, %2;\n\t"
        "addc.u32 y1, 0, 0;\n\t"
        "sub.cc.u32 e, e, y0;\n\t"
        "subc.cc.u32 t, t, y1;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 e, e, m;\n\t"
        "subc.u32 t, t, 0;\n\t"
        "mov.b64 %0, {e, t};\n\t}"
        : "=l"(r)
        : "r"(x0 << 16), "r"(__funnelshift_l(x0, x1, 16)), "r"(x1 >> 16));
    return r;
}

// x 2^72, canonical for any x: 2^72 == -2^40 2^-64, the same with x 2^40 (its low word is zero).
__device__ __forceinline__ uint64_t rot72(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    uint64_t r;
    asm("{\n\t.reg .u32 t, y0, y1, m;\n\t"
        "add.cc.u32 y0, %2, %1;\n\t"
        "addc.u32 y1, %3, 0;\n\t"
        "sub.cc.u32 y0, 0, y0;\n\t"
        "subc.cc.u32 t, %1, y1;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 y0, y0, m;\n\t"
        "subc.u32 t, t, 0;\n\t"
        "mov.b64 %0, {y0, t};\n\t}"
        : "=l"(r)
        : "r"(x0 << 8), "r"(__funnelshift_l(x0, x1, 8)), "r"(x1 >> 24));
    return r;
}

// In-register DFT of R points over GF(q), natural order, canonical in and out:
//   X_k = sum_n x_n w_R^{+-nk}   (w_R = 7^((q-1)/R) forward, its inverse for INV; unscaled).
template <int R, bool INV>
struct NDft;

template <bool INV>
struct NDft<2, INV> {
    __device__ __forceinline__ static void run(uint64_t* v) {
        const uint64_t a = v[0], b = v[1];
        v[0] = add(a, b);
        v[1] = sub(a, b);
    }
};

template <bool INV>
struct NDft<4, INV> {
    __device__ __forceinline__ static void run(uint64_t* v) {
        const uint64_t a0 = add(v[0], v[2]), a1 = sub(v[0], v[2]);
        const uint64_t b0 = add(v[1], v[3]);
        // w_4 = 2^48, w_4^-1 = -2^48
        const uint64_t b1 = rot48(INV ? sub(v[3], v[1]) : sub(v[1], v[3]));
        v[0] = add(a0, b0);
        v[2] = sub(a0, b0);
        v[1] = add(a1, b1);
        v[3] = sub(a1, b1);
    }
};

template <bool INV>
struct NDft<8, INV> {
    __device__ __forceinline__ static void run(uint64_t* v) {
        uint64_t s[4], d[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) s[n] = add(v[n], v[n + 4]);
        d[0] = sub(v[0], v[4]);
        if constexpr (!INV) {  // w_8 = -2^24, w_8^2 = 2^48, w_8^3 = -2^72
            d[1] = rot24(sub(v[5], v[1]));
            d[2] = rot48(sub(v[2], v[6]));
            d[3] = rot72(sub(v[7], v[3]));
        } else {  // w_8^-1 = 2^72, w_8^-2 = -2^48, w_8^-3 = 2^24
            d[1] = rot72(sub(v[1], v[5]));
            d[2] = rot48(sub(v[6], v[2]));
            d[3] = rot24(sub(v[3], v[7]));
        }
        NDft<4, INV>::run(s);
        NDft<4, INV>::run(d);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[2 * k] = s[k];
            v[2 * k + 1] = d[k];
        }
    }
};

}  // namespace gl
}  // namespace llg

#include "llg_fft.cuh"

namespace llg {
namespace gl {

// log2 of the values per thread of the NTT kernels: radix-8 passes. Against the radix-16 passes
// they replace, a pass costs as much per transformed bit, but its code is a third as long (the
// unrolled radix-16 kernels waited for instruction fetch 4 to 5.5 cycles per issued instruction)
// and twice the threads share the work.
constexpr int kLogE = 3;

// Length of a geometry's twiddle table (TW_PASS order, Montgomery form): the forward passes' twiddles,
// then the inverse ones. A pass reads consecutive slots at constant offsets: no index arithmetic on
// the ALU that binds these kernels (25 of about 280 ALU instructions a value before).
template <class G>
__host__ __device__ constexpr int table_len() { return 2 * G::pass_offset(G::P - 1); }

// Radix pass S of the L-point NTT on the register array (same geometry, positions and exchange
// pattern as the FP64 passes of llg_fft.cuh; 8-byte field elements in the exchange buffer; ES and
// PADLOG as there). Values are canonical before and after.
template <class G, int S, bool INV, bool SYNC_BEFORE_STORE, class SYNC, int ES = 1, int PADLOG = 4>
__device__ __forceinline__ void radix_pass(uint64_t (&v)[G::E], uint64_t* __restrict__ buf,
                                           const uint64_t* __restrict__ qtw, int t, const SYNC& sync) {
    constexpr int R = G::radix(S);
    constexpr int L = G::len(S);
    constexpr int ST = G::stride(S);
    constexpr int B = G::E / R;
    constexpr bool LOAD = INV ? (S < G::P - 1) : (S > 0);
    constexpr bool STORE = INV ? (S > 0) : (S < G::P - 1);
#pragma unroll
    for (int h = 0; h < B; ++h) {
        const int beta = t * B + h;
        const int g = beta / ST, n2 = beta % ST;
        const int base = g * L + n2;
        uint64_t* vv = v + h * R;
        const uint64_t* w = qtw + (INV ? G::pass_offset(G::P - 1) : 0) + G::pass_offset(S) + n2;
        if constexpr (LOAD) {
#pragma unroll
            for (int n1 = 0; n1 < R; ++n1) vv[n1] = buf[physp<PADLOG>(base + n1 * ST) * ES];
        }
        if constexpr (INV && ST > 1) {
#pragma unroll
            for (int k1 = 1; k1 < R; ++k1)
                vv[k1] = mul(vv[k1], w[(k1 - 1) * ST]);
        }
        NDft<R, INV>::run(vv);
        if constexpr (!INV && ST > 1) {
#pragma unroll
            for (int k1 = 1; k1 < R; ++k1)
                vv[k1] = mul(vv[k1], w[(k1 - 1) * ST]);
        }
        if constexpr (STORE && !SYNC_BEFORE_STORE) {
#pragma unroll
            for (int k1 = 0; k1 < R; ++k1) buf[physp<PADLOG>(base + k1 * ST) * ES] = vv[k1];
        }
    }
    if constexpr (STORE && SYNC_BEFORE_STORE) {
        sync();
#pragma unroll
        for (int h = 0; h < B; ++h) {
            const int beta = t * B + h;
            const int g = beta / ST, n2 = beta % ST;
            const int base = g * L + n2;
#pragma unroll
            for (int k1 = 0; k1 < R; ++k1) buf[physp<PADLOG>(base + k1 * ST) * ES] = v[h * R + k1];
        }
    }
}

// Forward passes S .. P-1 (pass S loads from buf unless S == 0).
template <class G, int S, class SYNC = CtaSync, int ES = 1, int PADLOG = 4>
__device__ __forceinline__ void forward_from(uint64_t (&v)[G::E], uint64_t* buf, const uint64_t* qtw,
                                             int t, const SYNC& sync = SYNC()) {
    if constexpr (S < G::P) {
        radix_pass<G, S, false, false, SYNC, ES, PADLOG>(v, buf, qtw, t, sync);
        if constexpr (S < G::P - 1) sync();
        forward_from<G, S + 1, SYNC, ES, PADLOG>(v, buf, qtw, t, sync);
    }
}

// Inverse passes S down to 0, starting from registers.
template <class G, int S, bool FIRST_SYNC = true, class SYNC = CtaSync, int ES = 1, int PADLOG = 4>
__device__ __forceinline__ void inverse_from(uint64_t (&v)[G::E], uint64_t* buf, const uint64_t* qtw,
                                             int t, const SYNC& sync = SYNC()) {
    if constexpr (S >= 0) {
        radix_pass<G, S, true, FIRST_SYNC && S == G::P - 1, SYNC, ES, PADLOG>(v, buf, qtw, t, sync);
        if constexpr (S > 0) sync();
        inverse_from<G, S - 1, false, SYNC, ES, PADLOG>(v, buf, qtw, t, sync);
    }
}

// b^e for b in Montgomery form (the power too).
__device__ __forceinline__ uint64_t pow(uint64_t b, uint64_t e) {
    uint64_t r = ONE;
    while (e) {
        if (e & 1) r = mul(r, b);
        b = mul(b, b);
        e >>= 1;
    }
    return r;
}

// signed value of a canonical field element that holds an integer of magnitude below 2^62 (the
// exactness bound of the lengths): z >= 2^63 stands for z - q = z - 2^64 + 2^32 - 1
__device__ __forceinline__ long long lift(uint64_t z) {
    return (long long)(z + (uint64_t)(uint32_t)((int32_t)(uint32_t)(z >> 32) >> 31));
}
// a digit as a canonical element
__device__ __forceinline__ uint64_t from_int(int x) {
    return (uint64_t)(long long)x - (uint64_t)(uint32_t)(x >> 31);
}

// One balanced-digit step at b bits: v = x + c 2^b with x in [-2^(b-1), 2^(b-1)), the carry
// c = floor((v + 2^(b-1)) / 2^b) (lucaslehmer.cpp:299-303).
__device__ __forceinline__ int balance64(long long v, int b, long long& c) {
    c = (v + (1LL << (b - 1))) >> b;
    return (int)((uint32_t)v - ((uint32_t)c << b));
}
__device__ __forceinline__ int balance32(int v, int b, int& c) {
    c = (v + (1 << (b - 1))) >> b;
    return v - (c << b);
}

}  // namespace gl
}  // namespace llg
