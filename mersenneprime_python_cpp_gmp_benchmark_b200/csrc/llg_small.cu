// Whole-test-on-chip FP64 IBDWT Lucas-Lehmer kernel for transform lengths N = 32 .. 8192.
//
// One thread block owns one exponent and runs all of its squarings without leaving the SM: the
// residue lives in registers between iterations and shared memory is only the exchange buffer of
// the radix passes. This replaces, for small p, the reference's per-test loop of
// lucaslehmer.cpp:281-311 (FFTW r2c -> square -> c2r -> unweight/round -> carry) and the
// single-block GPU loop of cuda/ll_ntt.cu:91-163, with a different transform:
//
//   * the N real weighted digits are packed as M = N/2 complex values u_m = y_2m + i y_2m+1 and
//     transformed by an M-point complex FFT (passes of radix 2 to 16 by the values a thread holds,
//     in-register DFTs, one shared-memory exchange per pass, no bit reversal);
//   * the real-FFT split and the pointwise square are one step on the pair (k, M-k):
//       U'_k = [(3A - B)(A + B) - w^k (A - B)^2] / 4,  A = U_k, B = conj(U_{M-k}), w = e^{-2 pi i/M}
//     which equals DFT_M(z_even + i z_odd) for the cyclic square z = y * y;
//   * the inverse FFT retraces the passes (decimation in time) back to natural order, where each
//     thread holds u_m for m = t + T*i: unweight, round (1.5*2^52 shifter), max round-off,
//     balanced carry and re-weighting happen in registers. The carry chain m -> m+1 crosses from
//     thread t to t+1 (warp shuffle, one shared-memory hop per warp boundary); a thread's carry-out
//     does not depend on its carry-in (the incoming carry is folded into the first digit and its
//     small overflow left in the second), so one exchange per iteration suffices and the digits
//     stay balanced to within a few units.
//
// Round-off guard: every iteration's max |x - round(x)| is reduced into the block barrier of the
// carry exchange; above `abort_err` the test stops with status LLG_ST_ROUNDOFF and the host redoes
// it at the next larger N.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "llg_device.cuh"
#include "llg_fft.cuh"
#include "llg_internal.h"

namespace llg {

// twiddle-table layout: every pass's own twiddles (TW_PASS) where they fit beside the exchange
// buffers of the resident blocks, i.e. below 16 values a thread; else (M = 2^12) the spread quarter
// table with factored twiddles
__host__ __device__ constexpr int small_tw_layout(int le) { return le >= 4 ? TW_QUARTER_S : TW_PASS; }
// log2 of the complex values per thread. Fewer values spread a test over more warps (its squarings
// are a serial chain, and a test alone on its SM otherwise runs at one or two warps' issue rate); more
// values take fewer passes and exchanges. Measured, us a squaring (the choice first), against 16
// values everywhere but N = 1024 (8 there) before:
//   one test      N = 32 .57 (2 values), .65 (4); 64 .67, .77; 128 .77 (4), .88 (2); 256 1.07 (4),
//                 1.54 (8); 512 1.31 (4), 1.67 (8); 1024 2.05 (8), 2.04 (4); 2048 2.81 (8), 3.38 (4);
//                 4096 4.83 (8), 6.2 (16); 8192 8.6 (16), 9.2 (8)
//        before   2.9, 4.6, 4.7, 4.9, 5.1, 3.3, 5.7, 6.2, 8.6
//   1184 tests    N = 32 2.5 (4 values); 64 2.1; 128 2.7; 256 2.9 (8); 512 6.4 (8); 1024 14.9 (8);
//                 2048 25.7 (8); 592 tests: 4096 17.0 (16), 17.4 (8)
//        before   15.8, 11.2, 7.4, 10.1, 9.4, 16.9, 34.6, 17.0
// With the digits as doubles and the kinds in the exponent field, the chosen forms now: one test .54, .64,
// .73, 1.02, 1.25, 1.90, 2.65, 4.58, 8.3; 1184 tests 2.1, 1.8, 2.5, 3.1, 5.9, 14.1, 23.0, 592 at 4096 14.6.
// Above one test per SM (small_fp64_log_e) the batch form runs.
__host__ __device__ constexpr int small_log_e_alone(int log_m) {
    return log_m <= 5 ? 1 : log_m <= 8 ? 2 : log_m <= 11 ? 3 : 4;
}
__host__ __device__ constexpr int small_log_e_batch(int log_m) { return log_m <= 6 ? 2 : log_m <= 10 ? 3 : 4; }
// M = 2^LOG_M complex points, 2^LE complex values per thread
template <int LOG_M, int LE>
using SmallGeo = SmallG<LOG_M, LE, small_tw_layout(LE), true>;

// blocks per SM the kernel is built for: 128 registers a thread (80 at 8 values a thread spilled,
// and cost 10 to 20% at N = 1024 and 2048)
__host__ __device__ constexpr int small_min_blocks(int t) { return t < 32 ? 16 : 512 / t > 16 ? 16 : 512 / t; }

template <int LOG_M, int LE>
__global__ void __launch_bounds__(SmallGeo<LOG_M, LE>::T, small_min_blocks(SmallGeo<LOG_M, LE>::T))
    ll_small_fp64(const SmallJob* __restrict__ jobs, const double2* __restrict__ qtw_g,
                  int64_t* __restrict__ digits_out, SmallResult* __restrict__ results,
                  float* __restrict__ errlog, double abort_err) {
    using G = SmallGeo<LOG_M, LE>;
    constexpr int M = G::M, N = G::N, E = G::E, T = G::T, W = G::W, PL = LE;
    constexpr int PAD = M + M / E;  // exchange slots: one of padding per E
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* buf = reinterpret_cast<double2*>(smem_raw);          // exchange buffer
    double2* qtw = buf + PAD;                                   // twiddles (small_tw_layout)
    constexpr int QL = (int)twiddle_table_len<G>();
    double* wB = reinterpret_cast<double*>(qtw + QL);
    double* iwB = wB + E;
    int* sB = reinterpret_cast<int*>(iwB + E);
    double* cbuf = reinterpret_cast<double*>(sB + E + (E & 1 ? 1 : 0) + 2);  // W * E
    unsigned long long* serr = reinterpret_cast<unsigned long long*>(cbuf + W * E);  // 2
    // slot of the partner U_{M-k} of this thread's position t E + j, [j][t]: fixed for the whole
    // test, read in the real-FFT split instead of two digit reversals a value
    unsigned short* pslot = reinterpret_cast<unsigned short*>(serr + 2);  // E * T
    // TW_PASS: the split's twiddle w^freq_rev of the NB positions, [h][t]: table slot and rotation
    constexpr int NBK = E / G::RLAST;
    unsigned short* kslot = pslot + E * T;  // NBK * T

    const int t = threadIdx.x;  // blockDim.x == T (a partial warp when T < 32)
    unsigned long long t_start = 0;
    if (t == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    const SmallJob job = jobs[blockIdx.x];
    const uint64_t p = job.p;
    const uint64_t iters = job.iters;
    const int q = (int)(p >> (LOG_M + 1));          // p / N
    const int rem = (int)(p & (uint64_t)(N - 1));   // p % N

    for (int k = t; k < QL; k += blockDim.x) qtw[k] = qtw_g[k];
    for (int i = t; i < E; i += T) {
        // digit j = 2m + e with m = t + T*i: s_j = (sA(t,e) + sB(i)) mod N
        const uint64_t s = (uint64_t)(N - (int)(((uint64_t)2 * T * i * p) & (uint64_t)(N - 1))) &
                           (uint64_t)(N - 1);
        sB[i] = (int)s;
        wB[i] = exp2((double)s / (double)N);
        iwB[i] = exp2(-(double)s / (double)N) / (4.0 * (double)M);
    }
    for (int i = t; i < 2; i += T) serr[i] = 0ull;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const int kp = (M - freq_of_pos<G>(t * E + j)) & (M - 1);
        pslot[j * T + t] = (unsigned short)physp<PL>(pos_of_freq<G>(kp));
    }
    if constexpr (G::TWM == TW_PASS) {
#pragma unroll
        for (int h = 0; h < NBK; ++h) kslot[h * T + t] = split_code<M, M / E>(freq_rev<G>(t * NBK + h));
    }
    __syncthreads();

    // per-thread weight halves for the even (e=0) and odd (e=1) digit of each u_m
    int sA0 = 0, sA1 = 0;
    double wA0 = 1, wA1 = 1, iwA0 = 1, iwA1 = 1;
    {
        sA0 = (int)((uint64_t)(N - (int)(((uint64_t)(2 * t) * p) & (uint64_t)(N - 1))) & (uint64_t)(N - 1));
        sA1 = (int)((uint64_t)(N - (int)(((uint64_t)(2 * t + 1) * p) & (uint64_t)(N - 1))) & (uint64_t)(N - 1));
        wA0 = exp2((double)sA0 / (double)N);
        wA1 = exp2((double)sA1 / (double)N);
        iwA0 = exp2(-(double)sA0 / (double)N);
        iwA1 = exp2(-(double)sA1 / (double)N);
    }

    // kind of the two digits of column i, fixed for the whole test, 4 bits per column: bit 0 / 1:
    // digit 2m / 2m+1 has q + 1 bits (s < p mod N); bit 2 / 3: s_A + s_B wrapped past N (weight
    // = table product / 2, inverse weight x 2)
    uint32_t kinds[(E + 7) / 8];
#pragma unroll
    for (int w = 0; w < (E + 7) / 8; ++w) kinds[w] = 0u;
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const int sb = sB[i];
        const bool o0 = sA0 + sb >= N, o1 = sA1 + sb >= N;
        const int s0 = o0 ? sA0 + sb - N : sA0 + sb;
        const int s1 = o1 ? sA1 + sb - N : sA1 + sb;
        const uint32_t kd = (uint32_t)(s0 < rem) | ((uint32_t)(s1 < rem) << 1) | ((uint32_t)o0 << 2) | ((uint32_t)o1 << 3);
        kinds[i / 8] |= kd << (4 * (i % 8));
    }
    const DigitBase dq(q);
    auto kind = [&](int i, int bit) { return kind_unit(kinds[i / 8], 4 * (i % 8) + bit); };
    // made opaque before each use: the weights and digit sizes derived from the kinds are then
    // formed where used, not hoisted into registers held across the transforms
    auto refresh_kinds = [&]() {
#pragma unroll
        for (int w = 0; w < (E + 7) / 8; ++w) asm volatile("" : "+r"(kinds[w]));
    };

    // the weighted digits, the transform, and from the carry to the next weighting the digits: doubles
    // throughout (as integers in between they cost four FP64 conversions a value)
    double2 v[E];
    // s_0 = 4: digit 0 (thread 0, i = 0, even) has weight a_0 = 1
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = make_double2(0.0, 0.0);
    if (t == 0) v[0].x = 4.0;

    const int lane = t & 31, warp = t >> 5;
    constexpr unsigned wmask = (T >= 32) ? 0xffffffffu : ((1u << (T & 31)) - 1u);
    using Sync = typename std::conditional<(T > 32), CtaSync, WarpSync>::type;
    Sync sync;
    if constexpr (T <= 32) sync.mask = wmask;
    double maxerr = 0.0;
    uint64_t it = 0;
    uint32_t status = LLG_ST_OK;

    for (;;) {
        forward_from<G, 0, Sync, 1, PL>(v, buf, qtw, t, sync);
        // pair (k, M-k): real-FFT split + square, result scaled by 4 (folded into iwB)
#pragma unroll
        for (int j = 0; j < E; ++j) buf[physp<PL>(t * E + j)] = v[j];
        sync();
        {
            // w^k of position t E + j: one table value per j / RLAST, times w_RLAST^(j % RLAST)
            constexpr int RL = G::RLAST, NB = E / RL;
            double2 wk[NB];
#pragma unroll
            for (int h = 0; h < NB; ++h) {
                if constexpr (G::TWM == TW_PASS) wk[h] = split_twiddle(qtw, kslot[h * T + t]);
                else wk[h] = twiddle_g<G>(qtw, (uint32_t)freq_rev<G>(t * NB + h), false);
            }
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int x = pslot[j * T + t];
                const double2 A = v[j], Bc = conj2(buf[x]);  // conj(U_{M-k})
                const double2 s = cadd(A, Bc), d = csub(A, Bc);
                const double2 a3 = make_double2(3.0 * A.x - Bc.x, 3.0 * A.y - Bc.y);
                const double2 d2 = make_double2((d.x - d.y) * (d.x + d.y), 2.0 * d.x * d.y);
                v[j] = csub(cmul(a3, s), cmul(wk[j / RL], rot_k<RL, false>(d2, j % RL)));
            }
        }
        // the first inverse pass stores only after a barrier (partners may still be reading)
        inverse_from<G, G::P - 1, true, Sync, 1, PL>(v, buf, qtw, t, sync);

        // unweight, round, error, local carry (even -> odd digit); the carry-out of column i goes
        // to thread t+1 (lane shuffle) or, at a warp boundary, through cbuf after the barrier
        ErrMax<2> err;
        double lerr;
        int bad;
        refresh_kinds();
        if constexpr (W == 1) {
            // one warp: the last thread's carry-outs go to thread 0 one column on, by shuffle too
            double x0[E], x1[E], c[E];
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const double iw = iwB[i];
                const double a = v[i].x * scale_up(iwA0 * iw, kind(i, 2));
                const double b = v[i].y * scale_up(iwA1 * iw, kind(i, 3));
                const double ra = round_shift(a), rb = round_shift(b);
                err.add(a - ra, b - rb);
                double cy;
                x0[i] = dsplit_k(ra, dq, kind(i, 0), cy);
                x1[i] = dsplit_k(rb + cy, dq, kind(i, 1), c[i]);
                c[i] = __shfl_sync(wmask, c[i], (t + T - 1) & (T - 1));
            }
            const double wrap = c[E - 1];
#pragma unroll
            for (int i = E - 1; i > 0; --i) c[i] = t == 0 ? c[i - 1] : c[i];
            c[0] = t == 0 ? wrap - 2.0 : c[0];  // the "- 2" of s^2 - 2
#pragma unroll
            for (int i = 0; i < E; ++i) {
                double cy;
                v[i].x = dsplit_k(x0[i] + c[i], dq, kind(i, 0), cy);
                v[i].y = x1[i] + cy;
            }
            lerr = err.value();
            if (errlog) {
                atomicMax(&serr[it & 1], (unsigned long long)__double_as_longlong(lerr));
                __syncwarp(wmask);
            }
            bad = __any_sync(wmask, lerr > abort_err);
        } else {
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const double iw = iwB[i];
                const double a = v[i].x * scale_up(iwA0 * iw, kind(i, 2));
                const double b = v[i].y * scale_up(iwA1 * iw, kind(i, 3));
                const double ra = round_shift(a), rb = round_shift(b);
                err.add(a - ra, b - rb);
                double c;
                const double x0 = dsplit_k(ra, dq, kind(i, 0), c);
                const double x1 = dsplit_k(rb + c, dq, kind(i, 1), c);
                const double cout = c;
                if (lane == 31) cbuf[warp * E + i] = cout;
                const double cin = __shfl_up_sync(0xffffffffu, cout, 1);
                v[i] = make_double2(x0, x1);
                if (lane != 0) {
                    v[i].x = dsplit_k(x0 + cin, dq, kind(i, 0), c);
                    v[i].y = x1 + c;
                }
            }
            lerr = err.value();
            if (errlog) atomicMax(&serr[it & 1], (unsigned long long)__double_as_longlong(lerr));
            bad = __syncthreads_or(lerr > abort_err);
        }
        maxerr = fmax(maxerr, lerr);
        if (errlog && t == 0) {
            errlog[it] = (float)__longlong_as_double((long long)serr[it & 1]);
            serr[(it + 1) & 1] = 0ull;
        }
        refresh_kinds();
        if (W > 1 && lane == 0) {
#pragma unroll
            for (int i = 0; i < E; ++i) {
                double cin = (warp > 0) ? cbuf[(warp - 1) * E + i]
                                        : cbuf[(W - 1) * E + ((i + E - 1) % E)];  // m-1 wraps at m=0
                if (t == 0 && i == 0) cin -= 2.0;  // the "- 2" of s^2 - 2
                double c;
                v[i].x = dsplit_k(v[i].x + cin, dq, kind(i, 0), c);
                v[i].y += c;
            }
        }
        ++it;
        if (bad) {
            status = LLG_ST_ROUNDOFF;
            break;
        }
        if (it >= iters) break;
        refresh_kinds();
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const double w = wB[i];
            v[i].x *= scale_down(wA0 * w, kind(i, 2));
            v[i].y *= scale_down(wA1 * w, kind(i, 3));
        }
    }

    if (digits_out) {
        int64_t* out = digits_out + (size_t)blockIdx.x * N;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int m = t + T * i;
            out[2 * m] = d2i_exact(v[i].x);
            out[2 * m + 1] = d2i_exact(v[i].y);
        }
    }
    // block max of the round-off (non-negative doubles order like their bit patterns)
    __syncthreads();
    if (t == 0) serr[0] = 0ull;
    __syncthreads();
    atomicMax(&serr[0], (unsigned long long)__double_as_longlong(maxerr));
    __syncthreads();
    if (t == 0) {
        SmallResult r;
        r.max_err = __longlong_as_double((long long)serr[0]);
        r.iters_done = it;
        r.status = status;
        unsigned long long t_end;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
        r.ns = t_end - t_start;
        results[blockIdx.x] = r;
    }
}

// p < 256: s <- s^2 - 2 mod 2^p - 1 on L = ceil(p / 64) 64-bit limbs (schoolbook square, one shift
// and add for the reduction as in lucaslehmer.cpp:42-48), one block per exponent. Exact; used where
// digits of an FFT length would hold too few bits for a stable balanced carry. The limb count is a
// template parameter, so every limb is a register (a runtime limb index put them in local memory:
// 80 us for the 125 squarings of p = 127, 20 now, launch included).
template <int L>
__device__ __forceinline__ void word_test(int p, uint64_t iters, uint64_t (&out)[4]) {
    // p is odd (or 2): bit p lies inside the top limb, never at a limb boundary
    const int r = p & 63;
    const uint64_t mask = (1ull << r) - 1ull;
    uint64_t s[L];
#pragma unroll
    for (int i = 0; i < L; ++i) s[i] = 0ull;
    s[0] = 4ull;
    if (L == 1 && p < 3) s[0] = 1ull;  // 4 mod 3
    for (uint64_t k = 0; k < iters; ++k) {
        uint64_t w[2 * L];
#pragma unroll
        for (int i = 0; i < 2 * L; ++i) w[i] = 0ull;
#pragma unroll
        for (int a = 0; a < L; ++a) {
            unsigned __int128 c = 0;
#pragma unroll
            for (int b = 0; b < L; ++b) {
                c += (unsigned __int128)s[a] * s[b] + w[a + b];
                w[a + b] = (uint64_t)c;
                c >>= 64;
            }
            w[a + L] = (uint64_t)c;
        }
        // s = (w mod 2^p) + (w >> p), below 2^(p+1); then bit p folded back (2^p == 1)
        unsigned __int128 c = 0;
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const uint64_t lo = i == L - 1 ? w[i] & mask : w[i];
            const uint64_t up = L + i < 2 * L ? w[L + i] : 0ull;
            c += (unsigned __int128)lo + ((w[L - 1 + i] >> r) | (up << (64 - r)));
            s[i] = (uint64_t)c;
            c >>= 64;
        }
        c = s[L - 1] >> r;
        s[L - 1] &= mask;
#pragma unroll
        for (int i = 0; i < L; ++i) {
            c += s[i];
            s[i] = (uint64_t)c;
            c >>= 64;
        }
        // s - 2 (s may still be 2^p - 1 standing for 0)
        uint64_t rest = 0ull;
#pragma unroll
        for (int i = 1; i < L; ++i) rest |= s[i];
        if (rest || s[0] >= 2) {
            uint64_t borrow = 2ull;
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const uint64_t x = s[i];
                s[i] = x - borrow;
                borrow = x < borrow ? 1ull : 0ull;
            }
        } else {  // s in {0, 1}: s - 2 + 2^p - 1
            const uint64_t v = s[0];
#pragma unroll
            for (int i = 0; i < L; ++i) s[i] = i == L - 1 ? mask : ~0ull;
            s[0] -= 2ull - v;
        }
    }
    bool all = true;  // 2^p - 1 is 0
#pragma unroll
    for (int i = 0; i < L; ++i) all = all && s[i] == (i == L - 1 ? mask : ~0ull);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (i < L && !all) ? s[i < L ? i : 0] : 0ull;
}

__global__ void ll_word(const SmallJob* __restrict__ jobs, uint64_t* __restrict__ res) {
    const int p = (int)jobs[blockIdx.x].p;
    const uint64_t iters = jobs[blockIdx.x].iters;
    uint64_t s[4];
    switch (p >> 6) {
        case 0: word_test<1>(p, iters, s); break;
        case 1: word_test<2>(p, iters, s); break;
        case 2: word_test<3>(p, iters, s); break;
        default: word_test<4>(p, iters, s); break;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) res[(size_t)blockIdx.x * 4 + j] = s[j];
}

cudaError_t launch_word(const SmallJob* jobs, int njobs, uint64_t* res, cudaStream_t st) {
    ll_word<<<njobs, 1, 0, st>>>(jobs, res);
    return cudaGetLastError();
}

template <int LOG_M, int LE>
static size_t small_smem_bytes() {
    using G = SmallGeo<LOG_M, LE>;
    size_t b = sizeof(double2) * (G::M + G::M / G::E);
    b += sizeof(double2) * twiddle_table_len<G>();
    b += 2 * sizeof(double) * G::E + sizeof(int) * (G::E + (G::E & 1 ? 1 : 0) + 2);
    b += sizeof(double) * G::W * G::E + 2 * sizeof(unsigned long long);
    b += sizeof(unsigned short) * G::E * G::T;  // partner slots of the real-FFT split
    if (G::TWM == TW_PASS) b += sizeof(unsigned short) * (G::E / G::RLAST) * G::T;  // its twiddles
    return b;
}

template <int LOG_M, int LE>
static cudaError_t launch_small_le(const SmallJob* jobs, int njobs, const double2* qtw,
                                   int64_t* digits, SmallResult* results, float* errlog,
                                   double abort_err, cudaStream_t st) {
    using G = SmallGeo<LOG_M, LE>;
    const size_t smem = small_smem_bytes<LOG_M, LE>();
    static PerDeviceOnce configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(ll_small_fp64<LOG_M, LE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ll_small_fp64<LOG_M, LE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     kWholeTestCarveout);
        if (e != cudaSuccess) return e;
        configured.mark();
    }
    ll_small_fp64<LOG_M, LE><<<njobs, G::T, smem, st>>>(jobs, qtw, digits, results, errlog, abort_err);
    return cudaGetLastError();
}

int small_fp64_log_e(int log_n, int njobs) {
    return njobs <= device_sms() ? small_log_e_alone(log_n - 1) : small_log_e_batch(log_n - 1);
}
bool small_fp64_pass_table(int log_e) { return small_tw_layout(log_e) == TW_PASS; }

template <int LOG_M>
static cudaError_t launch_small_t(int log_e, const SmallJob* jobs, int njobs, const double2* qtw,
                                  int64_t* digits, SmallResult* results, float* errlog,
                                  double abort_err, cudaStream_t st) {
    if (log_e == small_log_e_alone(LOG_M))
        return launch_small_le<LOG_M, small_log_e_alone(LOG_M)>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
    if (log_e == small_log_e_batch(LOG_M))
        return launch_small_le<LOG_M, small_log_e_batch(LOG_M)>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_small_fp64(int log_n, int log_e, const SmallJob* jobs, int njobs, const double2* qtw,
                              int64_t* digits, SmallResult* results, float* errlog,
                              double abort_err, cudaStream_t st) {
    switch (log_n - 1) {
        case 4: return launch_small_t<4>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 5: return launch_small_t<5>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 6: return launch_small_t<6>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 7: return launch_small_t<7>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 8: return launch_small_t<8>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 9: return launch_small_t<9>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 10: return launch_small_t<10>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 11: return launch_small_t<11>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 12: return launch_small_t<12>(log_e, jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace llg
