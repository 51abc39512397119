// Device-side building blocks shared by the Lucas-Lehmer kernels (sm_100a):
//   * complex FP64 arithmetic on double2 and fixed-radix in-register DFTs (2, 4, 8, 16 points);
//   * twiddles from a quarter-wave table (one load and a rotation by a power of -i);
//   * round-to-nearest with the 1.5*2^52 shifter;
//   * the balanced-digit carry step of the irrational-base DWT.
//
// The arithmetic follows the IBDWT of the reference's FFT engine (lucaslehmer.cpp:257-311):
// digits x_j in a variable base of b_j = ceil((j+1)p/N) - ceil(jp/N) bits, weights
// a_j = 2^(ceil(jp/N) - jp/N), a cyclic convolution of the weighted digits, unweight, round,
// balanced carry with the "- 2" folded into digit 0 and the top carry wrapping into digit 0.
#pragma once

#include <cstdint>

namespace llg {

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
// a * (-i) and a * (+i)
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }
__device__ __forceinline__ double2 mul_pi(double2 a) { return make_double2(-a.y, a.x); }

// Multiply by e^{-2 pi i k / R} (INV=false) or e^{+2 pi i k / R} (INV=true) for a compile-time
// k / R with R in {2, 4, 8, 16}. Special angles use adds only; the rest use exact constants.
template <int R, int K, bool INV>
__device__ __forceinline__ double2 rot(double2 a) {
    constexpr int k = ((K % R) + R) % R;
    constexpr int k16 = k * (16 / R);  // angle in units of 2*pi/16
    if constexpr (k16 == 0) return a;
    constexpr double C1 = 0.92387953251128675613;  // cos(pi/8)
    constexpr double S1 = 0.38268343236508977173;  // sin(pi/8)
    constexpr double H = 0.70710678118654752440;   // cos(pi/4)
    // e^{-2 pi i k16/16} = cos(t) - i sin(t), t = k16*pi/8
    constexpr double cs[16] = {1, C1, H, S1, 0, -S1, -H, -C1, -1, -C1, -H, -S1, 0, S1, H, C1};
    constexpr double sn[16] = {0, S1, H, C1, 1, C1, H, S1, 0, -S1, -H, -C1, -1, -C1, -H, -S1};
    constexpr double c = cs[k16];
    constexpr double s = INV ? -sn[k16] : sn[k16];  // multiply by (c - i s)
    if constexpr (k16 == 4) return INV ? mul_pi(a) : mul_mi(a);
    if constexpr (k16 == 8) return make_double2(-a.x, -a.y);
    if constexpr (k16 == 12) return INV ? mul_mi(a) : mul_pi(a);
    if constexpr (k16 == 2 || k16 == 6 || k16 == 10 || k16 == 14) {
        // (a.x + i a.y)(c - i s) with |c| = |s| = H
        return make_double2(H * ((c > 0 ? a.x : -a.x) + (s > 0 ? a.y : -a.y)),
                            H * ((c > 0 ? a.y : -a.y) - (s > 0 ? a.x : -a.x)));
    }
    return make_double2(fma(a.x, c, a.y * s), fma(a.y, c, -a.x * s));
}

// rot<16, k16, INV> for a k16 known only after unrolling (the switch folds away).
template <bool INV>
__device__ __forceinline__ double2 rot16_k(double2 a, int k16) {
    switch (k16 & 15) {
        case 0: return a;
        case 1: return rot<16, 1, INV>(a);
        case 2: return rot<16, 2, INV>(a);
        case 3: return rot<16, 3, INV>(a);
        case 4: return rot<16, 4, INV>(a);
        case 5: return rot<16, 5, INV>(a);
        case 6: return rot<16, 6, INV>(a);
        case 7: return rot<16, 7, INV>(a);
        case 8: return rot<16, 8, INV>(a);
        case 9: return rot<16, 9, INV>(a);
        case 10: return rot<16, 10, INV>(a);
        case 11: return rot<16, 11, INV>(a);
        case 12: return rot<16, 12, INV>(a);
        case 13: return rot<16, 13, INV>(a);
        case 14: return rot<16, 14, INV>(a);
        default: return rot<16, 15, INV>(a);
    }
}
// Multiply by e^{-2 pi i k / R} (INV: e^{+2 pi i k / R}), R in {1, 2, 4, 8, 16}.
template <int R, bool INV>
__device__ __forceinline__ double2 rot_k(double2 a, int k) {
    if constexpr (R == 1) return a;
    else return rot16_k<INV>(a, (k & (R - 1)) * (16 / R));
}

// In-register DFT of R points, natural order in and out:
//   X_k = sum_n x_n e^{-+2 pi i nk/R}   (sign - for the forward transform, + for INV; unscaled).
template <int R, bool INV>
struct Dft;

template <bool INV>
struct Dft<1, INV> {
    __device__ __forceinline__ static void run(double2*) {}
};

template <bool INV>
struct Dft<2, INV> {
    __device__ __forceinline__ static void run(double2* v) {
        double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <bool INV>
struct Dft<4, INV> {
    __device__ __forceinline__ static void run(double2* v) {
        double2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        double2 b0 = cadd(v[1], v[3]), b1 = csub(v[1], v[3]);
        b1 = INV ? mul_pi(b1) : mul_mi(b1);
        v[0] = cadd(a0, b0);
        v[2] = csub(a0, b0);
        v[1] = cadd(a1, b1);
        v[3] = csub(a1, b1);
    }
};

// R = R1 * R2 split (decimation in frequency on the register array):
//   X[k1 + R1 k2] = sum_{n2} w_{R2}^{n2 k2} w_R^{n2 k1} sum_{n1} x[n1 R2 + n2] w_{R1}^{n1 k1}
template <int R1, int R2, bool INV>
struct DftSplit {
    static constexpr int R = R1 * R2;
    template <int N2, int K1>
    __device__ __forceinline__ static void twiddle_all(double2 (&a)[R1][R2]) {
        if constexpr (N2 < R2) {
            if constexpr (K1 < R1) {
                a[K1][N2] = rot<R, N2 * K1, INV>(a[K1][N2]);
                twiddle_all<N2, K1 + 1>(a);
            } else {
                twiddle_all<N2 + 1, 0>(a);
            }
        }
    }
    __device__ __forceinline__ static void run(double2* v) {
        double2 a[R1][R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
            double2 col[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) col[n1] = v[n1 * R2 + n2];
            Dft<R1, INV>::run(col);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) a[k1][n2] = col[k1];
        }
        twiddle_all<0, 0>(a);
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            Dft<R2, INV>::run(a[k1]);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = a[k1][k2];
        }
    }
};

template <bool INV>
struct Dft<8, INV> {
    __device__ __forceinline__ static void run(double2* v) { DftSplit<2, 4, INV>::run(v); }
};
template <bool INV>
struct Dft<16, INV> {
    __device__ __forceinline__ static void run(double2* v) { DftSplit<4, 4, INV>::run(v); }
};

// Quarter-wave tables are stored padded: entry r at qpad(r) = r + r/8, so the strided indices of
// the radix passes (multiples of 16 and of small odd numbers) spread over the shared-memory banks.
__host__ __device__ constexpr uint32_t qpad(uint32_t r) { return r + (r >> 3); }
__host__ __device__ constexpr uint32_t qpad_len(uint32_t qm) { return qm + (qm >> 3) + 1; }
// The same quarter-wave table spread further, entry r at r + r/8 + r/64: the whole-test kernel's
// twiddle reads at index n2 k1 (8 lanes of a quarter warp, strides k1 and 16 k1) and its
// digit-reversed real-FFT twiddles then land in more of the 8 bank groups of 16-byte slots.
__host__ __device__ constexpr uint32_t qpad_s(uint32_t r) { return r + (r >> 3) + (r >> 6); }
__host__ __device__ constexpr uint32_t qpad_s_len(uint32_t qm) { return qm + (qm >> 3) + (qm >> 6) + 1; }
static_assert(qpad_s(255) < qpad_s_len(256) && qpad_s(1023) < qpad_s_len(1024) && qpad_s(4095) < qpad_s_len(4096),
              "spread quarter table length");

// Twiddle e^{-2 pi i x / M} (conjugated when inv) from a padded quarter-wave table
// q[qpad(r)] = e^{-2 pi i r / M}, r < M/4.  x in [0, M).
// SPREAD: the table is in the qpad_s layout.
template <int LOG_M, bool SPREAD = false>
__device__ __forceinline__ double2 twiddle(const double2* __restrict__ q, uint32_t x, bool inv) {
    constexpr uint32_t QM = (1u << LOG_M) / 4;
    const uint32_t quad = (x / QM) & 3u;
    double2 w = q[SPREAD ? qpad_s(x % QM) : qpad(x % QM)];
    // rotate by (-i)^quad
    double2 r;
    switch (quad) {
        case 0: r = w; break;
        case 1: r = make_double2(w.y, -w.x); break;
        case 2: r = make_double2(-w.x, -w.y); break;
        default: r = make_double2(-w.y, w.x); break;
    }
    return inv ? conj2(r) : r;
}

// Round to nearest even with the 1.5*2^52 shifter (valid for |v| < 2^51).
__device__ __forceinline__ double round_shift(double v) {
    constexpr double SH = 6755399441055744.0;  // 1.5 * 2^52
    return __dsub_rn(__dadd_rn(v, SH), SH);
}

// Exact conversion of a small signed integer (|x| < 2^51) to double by the same shifter.
__device__ __forceinline__ double i2d_shift(long long x) {
    constexpr double SH = 6755399441055744.0;
    return __dsub_rn(__longlong_as_double(x + 0x4338000000000000LL), SH);
}

// Programmatic dependent launch (griddepcontrol, sm_90 and later): let the next kernel of the
// stream launch once every block of this one has executed it, and wait until the previous kernel
// has completed with its memory visible. Both are no-ops in a launch without the programmatic
// stream serialisation attribute.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asynchronous global -> shared copies (cp.async, completed by cp_async_wait_all, then a barrier
// before other threads read the data).
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async sizes");
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 2^e as a double (normal range).
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }

// Balanced split of an integer-valued double: v = x + c 2^b with |x| <= 2^(b-1) (ties to even),
// c and x exact for |v| < 2^51; inv = 2^-b, pw = 2^b. The FP64 form of the reference's carry step
// (lucaslehmer.cpp:299-303: c = floor((v + 2^(b-1)) / 2^b)); the two differ only at ties, and
// either representation of the residue is exact.
__device__ __forceinline__ double dsplit(double v, double inv, double pw, double& c) {
    constexpr double SH = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    c = __dsub_rn(__fma_rn(v, inv, SH), SH);
    return __fma_rn(-c, pw, v);
}

// The digit kinds of a test are fixed: 4 bits a value, bit 0 / 1: digit 2m / 2m+1 has q + 1 bits;
// bit 2 / 3: its weight exponent s_A + s_B wrapped past N (the weight is the table product / 2). A
// kind bit at position p (compile time) as 1 << 20 or 0, one unit of a double's exponent field: digit
// sizes and weights are then integer additions to high words, no selects and no products by 1 or 2.
__device__ __forceinline__ uint32_t kind_unit(uint32_t w, int p) {
    return (p <= 20 ? w << (20 - p) : w >> (p - 20)) & 0x100000u;
}
// x * 2 (x / 2) for m = 1 << 20, x for m = 0; x a normal number
__device__ __forceinline__ double scale_up(double x, uint32_t m) {
    return __hiloint2double(__double2hiint(x) + (int)m, __double2loint(x));
}
__device__ __forceinline__ double scale_down(double x, uint32_t m) {
    return __hiloint2double(__double2hiint(x) - (int)m, __double2loint(x));
}

// High words of 2^q and 2^-q.
struct DigitBase {
    int up, down;
    __device__ __forceinline__ explicit DigitBase(int q) : up((1023 + q) << 20), down((1023 - q) << 20) {}
};
// dsplit with a digit of q bits (m = 0) or q + 1 bits (m = 1 << 20).
__device__ __forceinline__ double dsplit_k(double v, const DigitBase& B, uint32_t m, double& c) {
    return dsplit(v, __hiloint2double(B.down - (int)m, 0), __hiloint2double(B.up + (int)m, 0), c);
}

// Largest |d| of a run of differences, to the last bit: it is compared with the round-off bound, reported
// and logged. The whole-test kernels keep two maxima side by side, for the even and the odd digits: one
// chain of compares and selects was slower there (1184 tests at N = 1024 12.42 us a squaring against
// 12.33, at 2048 20.4 against 20.3) and faster in the row kernels of 16 values a thread, which are short
// of registers (2^23 137.9 against 139.6; the others within .6% either way). A maximum of high words
// alone takes .6 to 2.7% less with many tests an SM (N = 1024 12.26, 2048 20.13, 592 tests at 4096 14.01
// against 14.37, at 6144 27.9 against 28.4) and up to 1% less in the row kernels (2^23 137.7, 2^22 64.6
// against 65.3), but holds 20 bits of mantissa and rounds down. Not-a-number counts as infinite when it
// ends a run; a transform spreads one such value to all of its outputs.
template <int CHAINS>
struct ErrMax {
    double m[CHAINS] = {};
    __device__ __forceinline__ void add(double d0, double d1) {
        put(m[0], fabs(d0));
        put(m[CHAINS - 1], fabs(d1));
    }
    __device__ __forceinline__ double value() const {
        double x = m[0];
        if (CHAINS == 2) x = x >= m[CHAINS - 1] ? x : m[CHAINS - 1];
        return x == x ? x : __longlong_as_double(0x7ff0000000000000LL);
    }
    static __device__ __forceinline__ void put(double& m, double a) { m = m >= a ? m : a; }
};

// The largest of a full warp's non-negative doubles (they order like their bit patterns).
__device__ __forceinline__ unsigned long long warp_max(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    return ((unsigned long long)mh << 32) | __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
}

// An integer-valued double with |x| < 2^31 as int32 (the low word of x + 1.5 * 2^52).
__device__ __forceinline__ int d2i_exact(double x) { return __double2loint(__dadd_rn(x, 6755399441055744.0)); }

}  // namespace llg
