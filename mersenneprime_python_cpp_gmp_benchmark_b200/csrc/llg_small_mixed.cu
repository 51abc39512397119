// Whole-test-on-chip FP64 IBDWT Lucas-Lehmer kernel for the non-power-of-two lengths
// N = 2 R0 L, R0 in {3, 5}, L = 2^LOG_L (N = 3072, 5120, 6144, 10240, 12288): the reference's
// {3, 5} x 2^k transform lengths (lucaslehmer.cpp:244-254), which hold the same exponent with up to
// 37.5% fewer points than the next power of two.
//
// Same structure as the power-of-two kernel (llg_small.cu): one block per exponent, the M = R0 L
// packed complex values u_m = y_2m + i y_2m+1 stay on chip for all p - 2 squarings. The M-point
// transform is split as R0 x L (decimation in frequency, m = n + L r, k = R0 k' + k0):
//   X[R0 k' + k0] = sum_n w_L^{n k'} w_M^{n k0} sum_r u[n + L r] w_R0^{r k0}
// so a squaring is: the radix-R0 step with the twiddle w_M^{n k0}; R0 independent L-point FFTs (the
// power-of-two radix passes, one segment of L/8 or L/16 threads each, named barriers per segment); the
// real-FFT split and square on the pair (k, M - k), which pairs segment k0 with segment R0 - k0; the
// inverse L-point FFTs; the conjugate twiddle and the inverse radix-R0 step; then unweight, round,
// carry and weight in registers.
//
// Between squarings, and for the radix-R0 steps and the carry, thread t < TA = L / NPT holds
// x[c] = u[t + TA c], c < CA = NPT R0: the NPT columns n = t + TA i of every segment r
// (c = i + NPT r). The radix-R0 DFT of column n is then in one thread's registers; one store and one
// load per value move it to and from the segment-major order of the L-point FFTs (thread (seg, tl)
// holds z[seg][tl + TL i]). The digit order m = t + TA c runs across the lanes, then to the next
// column, as in the power-of-two kernel, so the carry is that kernel's with TA threads and CA
// columns; it wraps from the last digit to digit 0 (2^p == 1). The FFTs' R0 segments take at least
// TA threads.
//
// Twiddles are read where they are used: the passes' in pass order (TW_PASS), w_M^{n k0} as a table
// of R0 - 1 rows over n, the radix-R0 constants as immediates. Against quarter-wave tables with a fold
// and factored products, us a squaring: N = 3072 5.65 -> 4.2 for one test, 28.9 -> 26.3 for 1184; 5120
// 7.2 -> 6.0, 50.3 -> 43.9; 6144 10.2 -> 7.7, 32.1 -> 29.2 (592 tests); 10240 and 12288, which had read R0
// values from shared memory for every output of a radix-R0 step, 16.5 -> 12.5 and 17.4 -> 15.3, 33.3
// -> 25.3 and 35.1 -> 31.1 (296 tests). Fewer FP64 instructions and no integer fold; barriers and the
// latency of the shared-memory exchanges bound it now.

#include <cuda_runtime.h>

#include <cstdint>

#include "llg_device.cuh"
#include "llg_fft.cuh"
#include "llg_internal.h"

namespace llg {

// LE: log2 of the values per FFT thread; MINB: blocks per SM the kernel is built for (mixed_form)
template <int R0_, int LOG_L, int LE_, int MINB_>
struct MixedGeom {
    static constexpr int LE = LE_, MINB = MINB_;
    using GL = SmallG<LOG_L, LE, TW_PASS, true>;
    static constexpr int R0 = R0_;
    static constexpr int L = GL::M, TL = GL::T, E = GL::E;
    static constexpr int M = R0 * L, N = 2 * M;
    static constexpr int NPT = (R0 == 5 ? 2 : 4) << (LE - 3);  // columns n per digit thread
    static constexpr int TA = L / NPT, CA = NPT * R0, WA = TA / 32;
    static constexpr int T = R0 * TL;
    static constexpr int PADL = L + L / E;                       // exchange slots of one segment
    static constexpr int QL = (int)twiddle_table_len<GL>();      // pass twiddles of the L-point FFT
    static constexpr int NB = E / GL::RLAST;                     // split twiddles a thread reads
    static_assert(TA <= T && TA % 32 == 0 && TL % 32 == 0, "digit threads are whole warps of the FFT threads");
    static size_t smem() {
        return sizeof(double2) * ((size_t)R0 * PADL + QL + (R0 - 1) * L) + sizeof(double) * (2 * CA + WA * CA) +
               sizeof(int) * CA + 2 * sizeof(unsigned long long) + sizeof(unsigned short) * (E + NB) * T;
    }
};

// R0-point DFT in registers. The terms of r and R0 - r pair up as (x_r + x_{R0-r}) cos + i (x_r -
// x_{R0-r}) sin, and X[R0 - k] differs from X[k] only in the sign of the sine half.
template <int R0, bool INV>
__device__ __forceinline__ void dft_r0(double2 (&x)[R0]) {
    constexpr int H = (R0 - 1) / 2;
    // cos and sin of 2 pi j / R0
    constexpr double cs[5] = {1.0, R0 == 3 ? -0.5 : 0.30901699437494742410, R0 == 3 ? -0.5 : -0.80901699437494742410,
                              -0.80901699437494742410, 0.30901699437494742410};
    constexpr double sn[5] = {0.0, R0 == 3 ? 0.86602540378443864676 : 0.95105651629515357212,
                              R0 == 3 ? -0.86602540378443864676 : 0.58778525229247312917, -0.58778525229247312917,
                              -0.95105651629515357212};
    double2 sm[H], df[H];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
        sm[r - 1] = cadd(x[r], x[R0 - r]);
        df[r - 1] = csub(x[r], x[R0 - r]);
    }
    double2 x0 = x[0];
#pragma unroll
    for (int r = 0; r < H; ++r) x0 = cadd(x0, sm[r]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        double2 a = x[0], b = make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 1; r <= H; ++r) {
            const double c = cs[(k * r) % R0], s = INV ? sn[(k * r) % R0] : -sn[(k * r) % R0];
            a = make_double2(fma(sm[r - 1].x, c, a.x), fma(sm[r - 1].y, c, a.y));
            b = make_double2(fma(-df[r - 1].y, s, b.x), fma(df[r - 1].x, s, b.y));
        }
        x[k] = cadd(a, b);
        x[R0 - k] = csub(a, b);
    }
    x[0] = x0;
}

template <int R0, int LOG_L, int LE, int MINB>
__global__ void __launch_bounds__(MixedGeom<R0, LOG_L, LE, MINB>::T, MINB)
    ll_small_fp64_mixed(const SmallJob* __restrict__ jobs, const double2* __restrict__ qtw_g,
                        int64_t* __restrict__ digits_out, SmallResult* __restrict__ results,
                        float* __restrict__ errlog, double abort_err) {
    using MG = MixedGeom<R0, LOG_L, LE, MINB>;
    using GL = typename MG::GL;
    constexpr int L = MG::L, TL = MG::TL, E = MG::E, M = MG::M, N = MG::N, T = MG::T, TA = MG::TA,
                  CA = MG::CA, WA = MG::WA, NPT = MG::NPT, PADL = MG::PADL, QL = MG::QL, PL = LE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* bufs = reinterpret_cast<double2*>(smem_raw);  // R0 segment buffers of PADL slots
    double2* qtwL = bufs + R0 * PADL;                        // pass twiddles of the L-point FFT
    double2* tabM = qtwL + QL;                               // [k0 - 1][n] w_M^{n k0}
    double* wB = reinterpret_cast<double*>(tabM + (R0 - 1) * L);  // CA column weights
    double* iwB = wB + CA;
    double* cbuf = iwB + CA;                                 // WA * CA carry-outs of last lanes
    int* sB = reinterpret_cast<int*>(cbuf + WA * CA);
    unsigned long long* serr = reinterpret_cast<unsigned long long*>(sB + CA);  // 2 (8-aligned: CA even)
    static_assert(CA % 2 == 0, "8-byte alignment of serr");
    // slot of the partner U_{M-k} of position tl E + j of this thread's segment, [j][t]: fixed for
    // the whole test, read in the real-FFT split instead of two digit reversals a value
    unsigned short* pslot = reinterpret_cast<unsigned short*>(serr + 2);  // E * T
    unsigned short* kslot = pslot + E * T;  // [h][t]: the split's twiddles (split_code)
    constexpr int NB = MG::NB;

    const int t = threadIdx.x;
    const bool holds = t < TA;  // a digit thread (whole warps)
    const int seg = t / TL, tl = t % TL;
    const int lane = t & 31, warp = t >> 5;
    unsigned long long t_start = 0;
    if (t == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    const SmallJob job = jobs[blockIdx.x];
    const uint64_t p = job.p;
    const uint64_t iters = job.iters;
    const int q = (int)(p / (uint64_t)N);
    const int rem = (int)(p % (uint64_t)N);

    for (int k = t; k < QL + (R0 - 1) * L; k += T) qtwL[k] = qtw_g[k];
    for (int c = t; c < CA; c += T) {
        // digit j = 2m + e with m = t + TA c: s_j = (sA(t, e) + sB(c)) mod N
        const uint64_t s = ((uint64_t)N - ((uint64_t)2 * TA * c * p) % (uint64_t)N) % (uint64_t)N;
        sB[c] = (int)s;
        wB[c] = exp2((double)s / (double)N);
        iwB[c] = exp2(-(double)s / (double)N) / (4.0 * (double)M);
    }
    if (t < 2) serr[t] = 0ull;
    {
        const int sg = t / TL, tq = t % TL, sgp = (sg == 0) ? 0 : R0 - sg;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int kk = freq_of_pos<GL>(tq * E + j);
            const int kp = (sg == 0) ? ((L - kk) & (L - 1)) : (L - 1 - kk);
            pslot[j * T + t] = (unsigned short)(sgp * PADL + physp<PL>(pos_of_freq<GL>(kp)));
        }
#pragma unroll
        for (int h = 0; h < NB; ++h) kslot[h * T + t] = split_code<M, L>(R0 * freq_rev<GL>(tq * NB + h) + sg);
    }
    __syncthreads();

    const int sA0 = (int)(((uint64_t)N - ((uint64_t)(2 * t) * p) % (uint64_t)N) % (uint64_t)N);
    const int sA1 = (int)(((uint64_t)N - ((uint64_t)(2 * t + 1) * p) % (uint64_t)N) % (uint64_t)N);
    const double wA0 = exp2((double)sA0 / (double)N), wA1 = exp2((double)sA1 / (double)N);
    const double iwA0 = exp2(-(double)sA0 / (double)N), iwA1 = exp2(-(double)sA1 / (double)N);
    // kind of the two digits of column c, fixed for the whole test, 4 bits per column: bit 0 / 1:
    // digit 2m / 2m+1 has q + 1 bits; bit 2 / 3: its weight wrapped past N
    uint32_t kinds[(CA + 7) / 8];
#pragma unroll
    for (int w = 0; w < (CA + 7) / 8; ++w) kinds[w] = 0u;
#pragma unroll
    for (int c = 0; c < CA; ++c) {
        const int sb = sB[c];
        const bool o0 = sA0 + sb >= N, o1 = sA1 + sb >= N;
        const int s0 = o0 ? sA0 + sb - N : sA0 + sb;
        const int s1 = o1 ? sA1 + sb - N : sA1 + sb;
        const uint32_t kd = (uint32_t)(s0 < rem) | ((uint32_t)(s1 < rem) << 1) | ((uint32_t)o0 << 2) | ((uint32_t)o1 << 3);
        kinds[c / 8] |= kd << (4 * (c % 8));
    }
    const DigitBase dq(q);
    auto kind = [&](int c, int bit) { return kind_unit(kinds[c / 8], 4 * (c % 8) + bit); };
    // made opaque before each use: the weights and digit sizes derived from the kinds are then
    // formed where used, not hoisted into registers held across the transforms
    auto refresh_kinds = [&]() {
#pragma unroll
        for (int w = 0; w < (CA + 7) / 8; ++w) asm volatile("" : "+r"(kinds[w]));
    };

    // the digits between squarings, as integers (as doubles they spilled: N = 6144 28.7 -> 34.0 us a
    // squaring): s_0 = 4 (digit 0 has weight 1)
    int x0s[CA], x1s[CA];
#pragma unroll
    for (int c = 0; c < CA; ++c) x0s[c] = x1s[c] = 0;
    if (t == 0) x0s[0] = 4;

    const NamedSync gsync{1u + (unsigned)seg, (unsigned)TL};
    double2* mybuf = bufs + seg * PADL;
    double maxerr = 0.0;
    uint64_t it = 0;
    uint32_t status = LLG_ST_OK;

    for (;;) {
        // ---- weight, radix-R0 DFT of the thread's NPT columns n, twiddle w_M^{n k0}, to segment
        //      order (one column's R0 values live at a time) ----
        refresh_kinds();
        if (holds) {
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
                const int n = t + TA * i;
                double2 z[R0];
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int c = i + NPT * r;
                    const double w = wB[c];
                    z[r] = make_double2(i2d_shift(x0s[c]) * scale_down(wA0 * w, kind(c, 2)),
                                        i2d_shift(x1s[c]) * scale_down(wA1 * w, kind(c, 3)));
                }
                dft_r0<R0, false>(z);
                bufs[physp<PL>(n)] = z[0];
#pragma unroll
                for (int k0 = 1; k0 < R0; ++k0)
                    bufs[k0 * PADL + physp<PL>(n)] = cmul(z[k0], tabM[(k0 - 1) * L + n]);
            }
        }
        __syncthreads();
        double2 v[E];
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = mybuf[physp<PL>(tl + TL * i)];
        // the first pass stores after a segment barrier: the segment's loads above must be done
        radix_pass<GL, 0, false, true, NamedSync, 1, PL>(v, mybuf, qtwL, tl, gsync);
        gsync();
        forward_from<GL, 1, NamedSync, 1, PL>(v, mybuf, qtwL, tl, gsync);

        // ---- pair (k, M - k): real-FFT split + square (result scaled by 4, folded into iwB) ----
#pragma unroll
        for (int j = 0; j < E; ++j) mybuf[physp<PL>(tl * E + j)] = v[j];
        __syncthreads();
        {
            // w_M^{R0 kk + seg}: one table value per j / RL, times the exact rotation w_RL^(j % RL)
            constexpr int RL = GL::RLAST;
            double2 wk[NB];
#pragma unroll
            for (int h = 0; h < NB; ++h) wk[h] = split_twiddle(tabM, kslot[h * T + t]);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const double2 A = v[j], Bc = conj2(bufs[pslot[j * T + t]]);  // conj(U_{M-k})
                const double2 s = cadd(A, Bc), d = csub(A, Bc);
                const double2 a3 = make_double2(3.0 * A.x - Bc.x, 3.0 * A.y - Bc.y);
                const double2 d2 = make_double2((d.x - d.y) * (d.x + d.y), 2.0 * d.x * d.y);
                v[j] = csub(cmul(a3, s), cmul(wk[j / RL], rot_k<RL, false>(d2, j % RL)));
            }
        }
        __syncthreads();  // partner reads (other segments) done before any segment stores
        inverse_from<GL, GL::P - 1, false, NamedSync, 1, PL>(v, mybuf, qtwL, tl, gsync);
        if (seg > 0) {
#pragma unroll
            for (int i = 0; i < E; ++i) v[i] = cmulc(v[i], tabM[(seg - 1) * L + tl + TL * i]);
        }
        gsync();  // this segment's last inverse pass read its buffer
#pragma unroll
        for (int i = 0; i < E; ++i) mybuf[physp<PL>(tl + TL * i)] = v[i];
        __syncthreads();

        // ---- inverse radix-R0 DFT back to the thread's columns, then unweight, round and carry
        //      each column (the columns' carries are independent until the exchange below) ----
        ErrMax<2> err;
        refresh_kinds();
        if (holds) {
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
                const int n = t + TA * i;
                double2 z[R0];
#pragma unroll
                for (int k0 = 0; k0 < R0; ++k0) z[k0] = bufs[k0 * PADL + physp<PL>(n)];
                dft_r0<R0, true>(z);
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int c = i + NPT * r;
                    const double iw = iwB[c];
                    const double a = z[r].x * scale_up(iwA0 * iw, kind(c, 2));
                    const double b = z[r].y * scale_up(iwA1 * iw, kind(c, 3));
                    const double ra = round_shift(a), rb = round_shift(b);
                    err.add(a - ra, b - rb);
                    double cy;
                    double x0 = dsplit_k(ra, dq, kind(c, 0), cy);
                    const double x1 = dsplit_k(rb + cy, dq, kind(c, 1), cy);
                    const double cout = cy;
                    if (lane == 31) cbuf[warp * CA + c] = cout;
                    const double cin = __shfl_up_sync(0xffffffffu, cout, 1);
                    if (lane != 0) {
                        x0 = dsplit_k(x0 + cin, dq, kind(c, 0), cy);
                        x1s[c] = d2i_exact(x1 + cy);
                    } else {
                        x1s[c] = d2i_exact(x1);
                    }
                    x0s[c] = d2i_exact(x0);
                }
            }
        }
        const double lerr = err.value();
        maxerr = fmax(maxerr, lerr);
        if (errlog) atomicMax(&serr[it & 1], (unsigned long long)__double_as_longlong(lerr));
        const int bad = __syncthreads_or(lerr > abort_err);
        if (errlog && t == 0) {
            errlog[it] = (float)__longlong_as_double((long long)serr[it & 1]);
            serr[(it + 1) & 1] = 0ull;
        }
        refresh_kinds();
        if (holds && lane == 0) {
#pragma unroll
            for (int c = 0; c < CA; ++c) {
                // m - 1 of m = t + TA c: the previous warp's last lane, or the last warp's last lane
                // of column c - 1 (column CA - 1 at m = 0: the wrap-around, 2^p == 1)
                double cin = (warp > 0) ? cbuf[(warp - 1) * CA + c] : cbuf[(WA - 1) * CA + ((c + CA - 1) % CA)];
                if (t == 0 && c == 0) cin -= 2.0;  // the "- 2" of s^2 - 2
                double cy;
                x0s[c] = d2i_exact(dsplit_k(i2d_shift(x0s[c]) + cin, dq, kind(c, 0), cy));
                x1s[c] += d2i_exact(cy);
            }
        }
        ++it;
        if (bad) {
            status = LLG_ST_ROUNDOFF;
            break;
        }
        if (it >= iters) break;
    }

    if (holds && digits_out) {
        int64_t* out = digits_out + (size_t)blockIdx.x * N;
#pragma unroll
        for (int c = 0; c < CA; ++c) {
            const uint64_t m = (uint64_t)t + (uint64_t)TA * c;
            out[2 * m] = x0s[c];
            out[2 * m + 1] = x1s[c];
        }
    }
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

template <int R0, int LOG_L, int LE, int MINB>
static cudaError_t launch_mixed_t(const SmallJob* jobs, int njobs, const double2* qtw, int64_t* digits,
                                  SmallResult* results, float* errlog, double abort_err, cudaStream_t st) {
    using MG = MixedGeom<R0, LOG_L, LE, MINB>;
    const size_t smem = MG::smem();
    static PerDeviceOnce configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(ll_small_fp64_mixed<R0, LOG_L, LE, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ll_small_fp64_mixed<R0, LOG_L, LE, MINB>, cudaFuncAttributePreferredSharedMemoryCarveout, kWholeTestCarveout);
        if (e != cudaSuccess) return e;
        configured.mark();
    }
    ll_small_fp64_mixed<R0, LOG_L, LE, MINB><<<njobs, MG::T, smem, st>>>(jobs, qtw, digits, results, errlog, abort_err);
    return cudaGetLastError();
}

bool mixed_length_supported(uint32_t n, int* r0, int* log_l) {
    for (int r = 3; r <= 5; r += 2)
        for (int l = 9; l <= (r == 3 ? 11 : 10); ++l)
            if (n == 2u * (uint32_t)r << l) {
                if (r0) *r0 = r;
                if (log_l) *log_l = l;
                return true;
            }
    return false;
}

// Values a thread and blocks per SM, by length and whether each test has its SM to itself. Measured,
// us a squaring: one test, N = 3072 4.27 (8 values, one block per SM; 5.10 built for four, 8.0 with 16
// values), 5120 5.94 (6.20 for two, 8.5), 6144 7.79 (9.8, 9.8); more tests than SMs: N = 3072 13.1 (8
// values, four blocks; 592 tests; 17.5 with 16), 5120 22.1 (two blocks; 25.1), 6144 28.7 (16 values, two
// blocks; 32.5 with 8). One block fits an SM at 10240 and 12288: 16 values, 12.3 and 15.0 (8: 13.1, 17.2).
// (All with the round-off maximum in 20 bits; in full, 1 to 2% more with several tests an SM.)
int small_fp64_mixed_log_e(uint32_t n, int njobs) {
    int r0 = 0, l = 0;
    if (!mixed_length_supported(n, &r0, &l)) return 0;
    if (l == 9) return 3;
    return r0 == 3 && l == 10 && njobs <= device_sms() ? 3 : 4;
}

cudaError_t launch_small_fp64_mixed(uint32_t n, const SmallJob* jobs, int njobs, const double2* qtw,
                                    int64_t* digits, SmallResult* results, float* errlog,
                                    double abort_err, cudaStream_t st) {
    const bool alone = njobs <= device_sms();
    switch (n) {
        case 3072:
            return alone ? launch_mixed_t<3, 9, 3, 1>(jobs, njobs, qtw, digits, results, errlog, abort_err, st)
                         : launch_mixed_t<3, 9, 3, 4>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 5120:
            return alone ? launch_mixed_t<5, 9, 3, 1>(jobs, njobs, qtw, digits, results, errlog, abort_err, st)
                         : launch_mixed_t<5, 9, 3, 2>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 6144:
            return alone ? launch_mixed_t<3, 10, 3, 1>(jobs, njobs, qtw, digits, results, errlog, abort_err, st)
                         : launch_mixed_t<3, 10, 4, 2>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 10240: return launch_mixed_t<5, 10, 4, 1>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        case 12288: return launch_mixed_t<3, 11, 4, 1>(jobs, njobs, qtw, digits, results, errlog, abort_err, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace llg
