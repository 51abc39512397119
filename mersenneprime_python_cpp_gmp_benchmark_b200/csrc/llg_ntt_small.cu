// Whole-test-on-chip exact IBDWT over GF(2^64 - 2^32 + 1) for N = 64 .. 8192 (the Goldilocks NTT
// engine). One block per exponent, all squarings on chip. The reference's kernel for this
// (cuda/ll_ntt.cu:74-167) runs radix-2 stages with a barrier per stage and a carry loop that
// repeats until no carry is left; here:
//   * radix-8 passes in registers (internal twiddles are powers of 2, i.e. shifts), one exchange
//     through shared memory per pass, no bit reversal (the pointwise square ignores order);
//   * weights w^s with w an N-th root of 2 in the field (s = ceil(jp/N) N - jp), computed once per
//     test as w^sA * w^sB (digit m = t + T*i: sA from the thread, sB from i): the products in shared
//     memory up to N = 2048, formed in each squaring above (they would not fit beside the
//     exchange buffer of several blocks);
//   * the carry in four fixed hops: each digit's carry-out is taken from zero (independent of its
//     carry-in), the carry-in is absorbed with a renormalisation twice and the remainder (|r| < 2 in
//     practice) added to the next digit, so the result is exact and three exchanges suffice. From
//     the second hop on a digit and its carry fit 32 bits.
// Exactness: every convolution output is an integer below N 2^(2B-2) < q/2 for the lengths chosen
// by the host (B = bits of the largest digit), so the field value is the integer.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "llg_device.cuh"
#include "llg_fft.cuh"
#include "llg_internal.h"
#include "llg_ntt.cuh"

namespace llg {

// log2 of the values per thread: 4 values (radix-4 passes, twice the warps) up to N = 1024, where a
// test then spreads over the SM's four schedulers; 8 above. Measured, one test alone, us a
// squaring, 4 values against 8: N = 256 1.73 / 3.75, 512 2.09 / 4.58, 1024 3.62 / 5.49, 2048 7.23 / 6.69,
// 4096 16.4 / 14.4; 592 tests at once: N = 512 5.62 / 6.93, 1024 11.5 / 13.4, 2048 26.2 / 24.4. (The
// radix-16 kernel before: N = 512 31.8 alone, 31.4 with 592; N = 2048 35.3 and 70.2. With the twiddles in
// pass order now 2.07 and 5.42, 6.57 and 23.6.)
__host__ __device__ constexpr int small_ntt_log_e(int log_n) { return log_n <= 10 ? 2 : 3; }

template <int LOG_N>
struct SmallNtt {
    static constexpr int LE = small_ntt_log_e(LOG_N);
    using G = SmallG<LOG_N, LE>;
    static constexpr int N = G::M, E = G::E, T = G::T, W = G::W;
    static constexpr bool WT = LOG_N <= 11;  // whole weight tables in shared memory
    static constexpr int QL = gl::table_len<G>();
    static constexpr int NW = WT ? N : E;
    // blocks per SM the kernel is built for (64 registers a thread at 8 values)
    static constexpr int MINB = 1024 / T > 16 ? 16 : (1024 / T < 1 ? 1 : 1024 / T);
    static size_t smem() {
        return sizeof(uint64_t) * (G::PAD + QL + 2 * NW) + (sizeof(long long) + 2 * sizeof(int)) * W * E;
    }
};

// Carry exchange of one hop: c[i] = carry-out of element m - 1 (element m = t + T i); the last
// thread's carries go to thread 0 one column on. cb: W x E slots (several warps only).
template <int T, int W, int E, class C>
__device__ __forceinline__ void carry_exchange(C (&c)[E], C* cb, int t) {
    if constexpr (W == 1) {
        constexpr unsigned mask = (T >= 32) ? 0xffffffffu : ((1u << (T & 31)) - 1u);
#pragma unroll
        for (int i = 0; i < E; ++i) c[i] = __shfl_sync(mask, c[i], (t + T - 1) & (T - 1));
        const C last = c[E - 1];
#pragma unroll
        for (int i = E - 1; i > 0; --i) c[i] = (t == 0) ? c[i - 1] : c[i];
        c[0] = (t == 0) ? last : c[0];
    } else {
        const int lane = t & 31, warp = t >> 5;
        if (lane == 31) {
#pragma unroll
            for (int i = 0; i < E; ++i) cb[warp * E + i] = c[i];
        }
#pragma unroll
        for (int i = 0; i < E; ++i) c[i] = __shfl_up_sync(0xffffffffu, c[i], 1);
        __syncthreads();
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < E; ++i)
                c[i] = (warp > 0) ? cb[(warp - 1) * E + i] : cb[(W - 1) * E + ((i + E - 1) % E)];
        }
    }
}

template <int LOG_N>
__global__ void __launch_bounds__(SmallNtt<LOG_N>::T, SmallNtt<LOG_N>::MINB)
    ll_small_ntt(const SmallJob* __restrict__ jobs, const uint64_t* __restrict__ qtw_g, NttConst K,
                 int64_t* __restrict__ digits_out, SmallResult* __restrict__ results) {
    using SN = SmallNtt<LOG_N>;
    using G = typename SN::G;
    constexpr int N = G::M, E = G::E, T = G::T, W = G::W, QL = SN::QL;
    constexpr bool WT = SN::WT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* buf = reinterpret_cast<uint64_t*>(smem_raw);    // exchange buffer, PAD slots
    uint64_t* qtw = buf + G::PAD;                              // twiddles in pass order
    uint64_t* wT = qtw + QL;                                   // WT: w^s of digit m; else w^sB(i)
    uint64_t* iwT = wT + SN::NW;                               // WT: w^-s / N of digit m; else w^-sB(i) / N
    long long* cbuf = reinterpret_cast<long long*>(iwT + SN::NW);  // hop 1: W x E carry slots
    int* cbuf2 = reinterpret_cast<int*>(cbuf + W * E);          // hops 2 and 3: 2 x W x E

    const int t = threadIdx.x;
    unsigned long long t_start = 0;
    if (t == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    const SmallJob job = jobs[blockIdx.x];
    const uint64_t p = job.p, iters = job.iters;
    const int qp = (int)(p >> LOG_N);
    const int rem = (int)(p & (uint64_t)(N - 1));
    const unsigned wmask = (T >= 32) ? 0xffffffffu : ((1u << (T & 31)) - 1u);
    using Sync = typename std::conditional<(T > 32), CtaSync, WarpSync>::type;
    Sync sync;
    if constexpr (T <= 32) sync.mask = wmask;

    for (int k = t; k < QL; k += T) qtw[k] = qtw_g[k];
    // digit m = t + T i: s_m = (sA(t) + sB(i)) mod N, sB(i) = (-T i p) mod N; per value: bit i of
    // big: the digit has qp + 1 bits (s < p mod N), bit i of wrap: sA + sB >= N (the weight is the
    // product / 2)
    auto s_of = [&](uint64_t m) { return (int)((uint64_t)(N - (int)((m * p) & (uint64_t)(N - 1))) & (uint64_t)(N - 1)); };
    const int sA = s_of((uint64_t)t);
    const uint64_t wA = gl::pow(K.root2, (uint64_t)sA);
    const uint64_t iwA = gl::pow(K.inv_root2, (uint64_t)sA);
    uint32_t big = 0u, wrap = 0u;
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const int sB = s_of((uint64_t)T * i);
        const bool o = sA + sB >= N;
        const int s = o ? sA + sB - N : sA + sB;
        big |= (uint32_t)(s < rem) << i;
        wrap |= (uint32_t)o << i;
        if constexpr (WT) {
            wT[t + T * i] = gl::pow(K.root2, (uint64_t)s);
            iwT[t + T * i] = gl::mul(gl::pow(K.inv_root2, (uint64_t)s), K.invN);
        } else if (t == 0) {
            wT[i] = gl::pow(K.root2, (uint64_t)sB);
            iwT[i] = gl::mul(gl::pow(K.inv_root2, (uint64_t)sB), K.invN);
        }
    }
    sync();
    const uint64_t wAh = gl::mul(wA, gl::HALF), iwA2 = gl::add(iwA, iwA);
    auto weight = [&](int i) { return WT ? wT[t + T * i] : gl::mul((wrap >> i) & 1u ? wAh : wA, wT[i]); };
    // w^-s = w^-sA w^-sB, times w^N = 2 past N
    auto inv_weight = [&](int i) { return WT ? iwT[t + T * i] : gl::mul((wrap >> i) & 1u ? iwA2 : iwA, iwT[i]); };
    auto bits = [&](int i) { return qp + (int)((big >> i) & 1u); };

    uint64_t v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = 0ull;
    if (t == 0) v[0] = 4ull;  // s_0 = 4 at digit 0 (weight 1)
    int x[E];
    uint64_t it = 0;

    for (;;) {
        gl::forward_from<G, 0, Sync>(v, buf, qtw, t, sync);
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = gl::mul(v[j], v[j]);
        gl::inverse_from<G, G::P - 1, false, Sync>(v, buf, qtw, t, sync);
        // unweight (with 1/N and the square's 2^64), lift to signed, hop 1 from zero
        {
            long long c[E];
#pragma unroll
            for (int i = 0; i < E; ++i) x[i] = gl::balance64(gl::lift(gl::mul(v[i], inv_weight(i))), bits(i), c[i]);
            carry_exchange<T, W, E>(c, cbuf, t);
            if (t == 0) c[0] -= 2;  // the "- 2" of s^2 - 2 at digit 0
            // hop 2: absorb the neighbour's carry
#pragma unroll
            for (int i = 0; i < E; ++i) x[i] = gl::balance64((long long)x[i] + c[i], bits(i), c[i]);
            int c2[E];
#pragma unroll
            for (int i = 0; i < E; ++i) c2[i] = (int)c[i];
            carry_exchange<T, W, E>(c2, cbuf2, t);
            // hop 3: absorb the (small) second carry, renormalise once more
#pragma unroll
            for (int i = 0; i < E; ++i) x[i] = gl::balance32(x[i] + c2[i], bits(i), c2[i]);
            carry_exchange<T, W, E>(c2, cbuf2 + W * E, t);
            // hop 4: the remainder (|c| <= 1 in practice) stays in the digit
#pragma unroll
            for (int i = 0; i < E; ++i) x[i] += c2[i];
        }
        ++it;
        if (it >= iters) break;
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = gl::mul(gl::from_int(x[i]), weight(i));
    }

    if (digits_out) {
        int64_t* out = digits_out + (size_t)blockIdx.x * N;
#pragma unroll
        for (int i = 0; i < E; ++i) out[t + T * i] = x[i];
    }
    if (t == 0) {
        SmallResult r;
        r.max_err = 0.0;
        r.iters_done = it;
        r.status = LLG_ST_OK;
        unsigned long long t_end;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
        r.ns = t_end - t_start;
        results[blockIdx.x] = r;
    }
}

template <int LOG_N>
static cudaError_t launch_small_ntt_t(const SmallJob* jobs, int njobs, const uint64_t* qtw, NttConst K,
                                      int64_t* digits, SmallResult* results, cudaStream_t st) {
    using SN = SmallNtt<LOG_N>;
    const size_t smem = SN::smem();
    static PerDeviceOnce configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(ll_small_ntt<LOG_N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ll_small_ntt<LOG_N>, cudaFuncAttributePreferredSharedMemoryCarveout, kWholeTestCarveout);
        if (e != cudaSuccess) return e;
        configured.mark();
    }
    ll_small_ntt<LOG_N><<<njobs, SN::T, smem, st>>>(jobs, qtw, K, digits, results);
    return cudaGetLastError();
}

int small_ntt_values(int log_n) { return small_ntt_log_e(log_n); }

cudaError_t launch_small_ntt(int log_n, const SmallJob* jobs, int njobs, const uint64_t* qtw, NttConst K,
                             int64_t* digits, SmallResult* results, cudaStream_t st) {
    switch (log_n) {
        case 6: return launch_small_ntt_t<6>(jobs, njobs, qtw, K, digits, results, st);
        case 7: return launch_small_ntt_t<7>(jobs, njobs, qtw, K, digits, results, st);
        case 8: return launch_small_ntt_t<8>(jobs, njobs, qtw, K, digits, results, st);
        case 9: return launch_small_ntt_t<9>(jobs, njobs, qtw, K, digits, results, st);
        case 10: return launch_small_ntt_t<10>(jobs, njobs, qtw, K, digits, results, st);
        case 11: return launch_small_ntt_t<11>(jobs, njobs, qtw, K, digits, results, st);
        case 12: return launch_small_ntt_t<12>(jobs, njobs, qtw, K, digits, results, st);
        case 13: return launch_small_ntt_t<13>(jobs, njobs, qtw, K, digits, results, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace llg
