// Two-pass exact IBDWT over GF(2^64 - 2^32 + 1) for N = 2^14 .. 2^23, the residue resident in HBM
// as N field elements (8N bytes, the same footprint as the FP64 engine's N/2 complex values).
//
// Same four-step structure and tile layout as the FP64 two-pass engine (llg_large.cu), with one
// digit per element instead of two (no real-FFT packing, so the column pass needs no partner
// column: one block per column, pointwise square):
//   row pass (a tile of kNttRowG consecutive rows a, all C columns):  inverse C-point NTT, unweight
//       (and 1/N), signed lift, carry, "- 2", weight, forward C-point NTT;
//   column pass (one column c):  twiddle w_N^{ac}, forward R-point NTT, square, inverse, w_N^{-ac}.
// A row tile interleaves its rows across the lanes of every warp (thread t: row t % G, NTT thread
// t / G): loads and stores go straight between memory and registers, and the carries between the
// rows of a tile are lane shuffles.
// Carry: digit j = a + R b, so the chain runs down the rows of each column. Each row's carry-out
// is taken from zero (independent of its carry-in); the carry-in is absorbed with two
// renormalisations (hops 2, 3) whose own carries move one row further down, and the last, tiny
// remainder is added without renormalising (hop 4). A tile's last row therefore publishes three
// carries, all computable without the previous tile (a tile has >= 3 rows); tile k+1 reads them
// after a bounded wait on tile k's flag (tickets in launch order keep tile k resident). The
// wrap-around carry into row 0 (2^p == 1) comes from row R-1: the first ticket is a separate job
// that runs the last tile's rows through the inverse NTT and the hops and publishes their
// carries, one column on, in the slot tile 0 reads; the last tile waits (bounded) for that job
// before overwriting those rows.
//
// Both passes are bound by the integer ALU (the arithmetic of llg_ntt.cuh). Measured, us a squaring
// replayed from graphs, against radix-16 passes of one row per warp group with the 128-bit
// reduction: N = 2^16 55.5 -> 17.7, 2^18 67.3 -> 23.2, 2^21 176.8 -> 106.9, 2^23 654 -> 431. At 2^21 the
// row pass issued 37.2 M warp instructions (47.3 M before) at 57% of the ALU's rate (39%), the
// column pass 31.1 M at 67% (58%); neither waits for instruction fetch any more (5.5 cycles per
// issued instruction before). Kinds from a table and pass-ordered twiddles then took the row pass at
// 2^21 from 71 to 66.5 us.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "llg_device.cuh"
#include "llg_fft.cuh"
#include "llg_internal.h"
#include "llg_ntt.cuh"

namespace llg {

namespace {

constexpr int kNttRowG = 4;

__device__ __forceinline__ uint64_t twiddle_N(const NttLargeArgs& A, uint32_t x) {
    return gl::mul(__ldg(A.tw1 + (x & ((1u << A.tw_shift) - 1u))), __ldg(A.tw2 + (x >> A.tw_shift)));
}

}  // namespace

template <int LOG_C>
using NttRowG = SmallG<LOG_C, gl::kLogE>;
template <int LOG_R>
using NttColG = SmallG<LOG_R, gl::kLogE>;

// exchange-buffer slots of a tile: its rows of C + C/8 padded slots
template <int LOG_C>
__host__ __device__ constexpr int ntt_row_slots() { return kNttRowG * ((1 << LOG_C) + ((1 << LOG_C) >> gl::kLogE)); }

template <int LOG_C, int MODE>
__global__ void __launch_bounds__(kNttRowG * NttRowG<LOG_C>::T, 1024 / (kNttRowG * NttRowG<LOG_C>::T) > 8 ? 8 : 1024 / (kNttRowG * NttRowG<LOG_C>::T))
    ntt_row(const NttLargeArgs A) {
    using GC = NttRowG<LOG_C>;
    constexpr int C = GC::M, TR = GC::T, E = GC::E, G = kNttRowG, T = G * TR, PL = gl::kLogE;
    constexpr int QL = gl::table_len<GC>();
    constexpr unsigned FULL = 0xffffffffu;
    static_assert(T % 32 == 0 && 32 % G == 0 && G >= 4 && C % T == 0, "whole warps of whole row groups");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* xbuf = reinterpret_cast<uint64_t*>(smem_raw);  // exchange: slot physp(x) * G + row
    uint64_t* qtw = xbuf + ntt_row_slots<LOG_C>();            // twiddles in pass order
    uint64_t* swB = qtw + QL;                                 // C column weights
    uint64_t* siwB = swB + C;                                 // C inverse column weights
    __shared__ int s_job;
    __shared__ unsigned s_epoch;

    const int t = threadIdx.x, ra = t % G, tr = t / G;
    uint64_t* buf = xbuf + ra;
    const int R = A.R;
    const CtaSync sync;

    // the next pass may launch once every block of this one has started (or, pdl_late, is near its
    // end); constant tables first, nothing the previous pass writes before the wait
    if (!A.pdl_late) pdl_launch_dependents();
    for (int k = t; k < QL; k += T) cp_async<8>(qtw + k, A.qtwC + k);
    for (int k = t; k < C; k += T) {
        cp_async<8>(swB + k, A.wB + k);
        if (MODE != LARGE_INIT) cp_async<8>(siwB + k, A.iwB + k);
    }
    pdl_wait_previous();
    if (t == 0) {
        const unsigned ep = *reinterpret_cast<volatile unsigned*>(&A.ctl->epoch);
        s_epoch = ep;
        if (MODE == LARGE_INIT) {
            s_job = blockIdx.x;
        } else {
            // tickets in launch order: ticket 0 is the wrap-around job, ticket k tile k - 1
            const int tk = (int)atomicAdd(&A.ctl->ticket[ep & 1], 1u);
            if (tk == A.nblocks) {
                // every block of this launch holds its ticket: both counters can be reset
                A.ctl->ticket[(ep + 1) & 1] = 0u;
                A.ctl->ticket[ep & 1] = 0u;
            }
            s_job = tk - 1;
        }
    }
    __syncthreads();
    const int job = s_job;  // -1: the wrap-around job (rows R-G .. R-1), else the tile
    const unsigned ep = s_epoch;
    const bool wrap_job = job < 0;
    const int a = (wrap_job ? R - G : job * G) + ra;  // this thread's row

    uint64_t v[E];
    int x[E];
    // bit i of big: the digit has q + 1 bits; of wrap: sA + sB >= N (fill_ntt_kinds)
    const uint32_t kw = __ldg(A.kinds + (size_t)(a / G) * T + t);
    const uint32_t big = kw & 0xffu, wrap = kw >> 8;
    auto bits = [&](int i) { return A.q + (int)((big >> i) & 1u); };

    if constexpr (MODE == LARGE_INIT) {
#pragma unroll
        for (int i = 0; i < E; ++i) x[i] = A.digits[(size_t)a + (size_t)R * (tr + TR * i)];
        cp_async_wait_all();
        __syncthreads();  // the tables are in shared memory
    } else {
        {
            const uint64_t* lp = A.V + (size_t)(tr * E) * R + a;
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = __ldcg(lp + (size_t)j * R);
        }
        cp_async_wait_all();
        __syncthreads();  // the tables are in shared memory
        gl::inverse_from<GC, GC::P - 1, false, CtaSync, G, PL>(v, buf, qtw, tr, sync);

        // ---- unweight, lift, hop 1 of every row; hops 2 to 4 of the rows whose carry-in comes from
        //      inside the tile. Row G-1 publishes its three carry-outs (the wrap job: one column on).
        const int slot = job + 1;
        const uint64_t ia = __ldg(A.iwA + a), ia2 = gl::add(ia, ia);
        int c3r[E];  // hop-3 carry-outs (row 1's, which row 2 needs, are formed after the wait)
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int b = tr + TR * i;
            const int nb = bits(i);
            // w^-s = w^-sA w^-sB, times w^N = 2 past N
            const uint64_t z = gl::mul(v[i], gl::mul((wrap >> i) & 1u ? ia2 : ia, siwB[b]));
            long long c1, c;
            int y = gl::balance64(gl::lift(z), nb, c1);
            c = c1;
            const long long in1 = __shfl_up_sync(FULL, c1, 1, G);
            int c2 = 0, c3 = 0;
            if (ra > 0) {
                y = gl::balance64((long long)y + in1, nb, c);
                c2 = (int)c;
            }
            const int in2 = __shfl_up_sync(FULL, c2, 1, G);
            if (ra > 1) y = gl::balance32(y + in2, nb, c3);
            const int in3 = __shfl_up_sync(FULL, c3, 1, G);
            if (ra > 2) y += in3;
            if (ra == G - 1) {
                const size_t o = (size_t)slot * C + (wrap_job ? ((b + 1) & (C - 1)) : b);
                A.c1[o] = c1;
                A.c2[o] = c2;
                A.c3[o] = c3;
            }
            x[i] = y;
        }
        if (ra == G - 1) __threadfence();  // each publisher orders its carry stores before the flag
        __syncthreads();
        if (t == 0) *reinterpret_cast<volatile unsigned*>(&A.flags[slot]) = ep + 1u;
        if (wrap_job) return;
        // ---- the tile's first row: hops 2 to 4 from the previous tile's last row (or the wrap). The
        //      row passes through the exchange buffer, so that every thread takes C / T of its
        //      columns rather than one lane in G all of them. ----
        int* row0 = reinterpret_cast<int*>(xbuf);  // C digits of row 0
        int* h2 = row0 + C;                        // its hop-2 and hop-3 carry-outs
        int* h3 = h2 + C;
        if (ra == 0) {
#pragma unroll
            for (int i = 0; i < E; ++i) row0[tr + TR * i] = x[i];
        }
        if (t == 0) wait_flag(&A.flags[job], ep + 1u, A.ctl, kSpinLimit);
        __syncthreads();
        {
            const size_t o = (size_t)job * C;
#pragma unroll
            for (int k = 0; k < C / T; ++k) {
                const int b = t + T * k;
                // row 0's thread t % TR, value t / TR + G k
                const int nb = A.q + (int)((__ldg(A.kinds + (size_t)job * T + (t % TR) * G) >> (t / TR + G * k)) & 1u);
                long long cin = __ldcg(A.c1 + o + b), c;
                if (job == 0 && b == 0) cin -= 2;  // the "- 2" of s^2 - 2 (digit 0)
                int y = gl::balance64((long long)row0[b] + cin, nb, c), c3;
                h2[b] = (int)c;
                y = gl::balance32(y + __ldcg(A.c2 + o + b), nb, c3);
                h3[b] = c3;
                row0[b] = y + __ldcg(A.c3 + o + b);
            }
        }
        __syncthreads();
        // row 1: hops 3 and 4 from row 0; row 2: hop 4 from row 1
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int b = tr + TR * i;
            c3r[i] = 0;
            if (ra == 0) x[i] = row0[b];
            else if (ra == 1) x[i] = gl::balance32(x[i] + h2[b], bits(i), c3r[i]) + h3[b];
            const int in3 = __shfl_up_sync(FULL, c3r[i], 1, G);
            if (ra == 2) x[i] += in3;
        }
        if (MODE == LARGE_FINAL || A.dump) {
#pragma unroll
            for (int i = 0; i < E; ++i) A.digits[(size_t)a + (size_t)R * (tr + TR * i)] = x[i];
        }
        if constexpr (MODE == LARGE_FINAL) return;
    }

    // ---- weight, forward row NTT, store ----
    const uint64_t wa = __ldg(A.wA + a), wah = gl::mul(wa, gl::HALF);
#pragma unroll
    for (int i = 0; i < E; ++i)
        v[i] = gl::mul(gl::from_int(x[i]), gl::mul((wrap >> i) & 1u ? wah : wa, swB[tr + TR * i]));
    // the first forward pass stores after a barrier: the first row's carries may still be read from
    // the exchange buffer
    gl::radix_pass<GC, 0, false, true, CtaSync, G, PL>(v, buf, qtw, tr, sync);
    static_assert(GC::P > 1, "at least two row passes");
    sync();
    gl::forward_from<GC, 1, CtaSync, G, PL>(v, buf, qtw, tr, sync);
    if (MODE == LARGE_ITER && job == A.nblocks - 1) {
        // rows R-G .. R-1 are the wrap job's input: wait (bounded) until it has read them
        if (t == 0) wait_flag(&A.flags[0], ep + 1u, A.ctl, kSpinLimit);
        __syncthreads();
    }
    if (A.pdl_late) pdl_launch_dependents();
    uint64_t* vp = A.V + (size_t)(tr * E) * R + a;
#pragma unroll
    for (int j = 0; j < E; ++j) __stcg(vp + (size_t)j * R, v[j]);
}

// Each block runs columns blockIdx.x, + gridDim.x, ...: its twiddle tables are read once.
template <int LOG_R>
__global__ void __launch_bounds__(NttColG<LOG_R>::T, 1024 / NttColG<LOG_R>::T > 16 ? 16 : 1024 / NttColG<LOG_R>::T)
    ntt_col(const NttLargeArgs A) {
    using GR = NttColG<LOG_R>;
    constexpr int R = GR::M, TC = GR::T, E = GR::E;
    constexpr int QL = gl::table_len<GR>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* buf = reinterpret_cast<uint64_t*>(smem_raw);
    uint64_t* qtw = buf + GR::PAD;
    uint64_t* ptabs = qtw + QL;  // two columns' tables in turn: E forward, E inverse
    const int tc = threadIdx.x;
    const int N = 1 << A.logN;
    if (!A.pdl_late) pdl_launch_dependents();  // as in ntt_row
    for (int k = tc; k < QL; k += TC) cp_async<8>(qtw + k, A.qtwR + k);
    bool first = true;
    for (int c = blockIdx.x; c < A.C; c += gridDim.x) {
        uint64_t* ptab = ptabs + (c / (int)gridDim.x & 1) * 2 * E;
        // four-step twiddle w_N^{a c}, a = tc + TC i: w_N^{c tc} * w_N^{c TC i}
        for (int i = tc; i < E; i += TC) {
            const uint32_t xi = (uint32_t)(((uint64_t)c * TC * i) & (uint64_t)(N - 1));
            ptab[i] = twiddle_N(A, xi);
            ptab[E + i] = twiddle_N(A, (uint32_t)((N - xi) & (N - 1)));
        }
        const uint32_t xq = (uint32_t)(((uint64_t)c * tc) & (uint64_t)(N - 1));
        uint64_t* col = A.V + (size_t)__ldg(A.pos_of_c + c) * R;
        const uint64_t q = twiddle_N(A, xq);
        if (first) pdl_wait_previous();
        uint64_t v[E];
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = __ldcg(col + tc + TC * i);
        if (first) cp_async_wait_all();
        first = false;
        __syncthreads();  // ptab, and the tables
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = gl::mul(v[i], gl::mul(q, ptab[i]));
        gl::forward_from<GR, 0>(v, buf, qtw, tc);
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = gl::mul(v[j], v[j]);
        gl::inverse_from<GR, GR::P - 1, false>(v, buf, qtw, tc);
        const uint64_t qi = twiddle_N(A, (uint32_t)((N - xq) & (N - 1)));
#pragma unroll
        for (int i = 0; i < E; ++i) col[tc + TC * i] = gl::mul(v[i], gl::mul(qi, ptab[E + i]));
        // the next column's first stores to buf are to slots this thread read itself
    }
    if (A.pdl_late) pdl_launch_dependents();
    if (blockIdx.x == 0 && tc == 0) atomicAdd(&A.ctl->epoch, 1u);
}

// NttLargeArgs::kinds: word t of tile k holds the kinds of thread t's values (row t % G of the tile,
// columns t / G + TR i): bit i: the digit has q + 1 bits (s < p mod N, s = (sA(a) + sB(b)) mod N);
// bit 8 + i: sA + sB >= N.
__global__ void fill_ntt_kinds(uint32_t* kinds, const int* __restrict__ sA, const int* __restrict__ sB, int N, int rem,
                               int C, int words) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words) return;
    constexpr int E = 1 << gl::kLogE;
    const int TR = C / E, T = kNttRowG * TR, t = w % T;
    const int sa = sA[w / T * kNttRowG + t % kNttRowG];
    uint32_t k = 0u;
    for (int i = 0; i < E; ++i) {
        const int sb = sB[t / kNttRowG + TR * i];
        const bool o = sa + sb >= N;
        const int s = o ? sa + sb - N : sa + sb;
        k |= ((uint32_t)(s < rem) << i) | ((uint32_t)o << (8 + i));
    }
    kinds[w] = k;
}
cudaError_t launch_fill_ntt_kinds(uint32_t* kinds, const int* sA, const int* sB, int N, int rem, int C, int R, cudaStream_t st) {
    const int words = (int)((long long)R * C >> gl::kLogE);
    fill_ntt_kinds<<<(words + 255) / 256, 256, 0, st>>>(kinds, sA, sB, N, rem, C, words);
    return cudaGetLastError();
}

template <int LOG_C>
static size_t ntt_row_smem() {
    constexpr int C = 1 << LOG_C;
    return sizeof(uint64_t) * (ntt_row_slots<LOG_C>() + gl::table_len<NttRowG<LOG_C>>() + 2 * C);
}

template <int LOG_R>
static size_t ntt_col_smem() {
    using GR = NttColG<LOG_R>;
    return sizeof(uint64_t) * (GR::PAD + gl::table_len<GR>() + 4 * GR::E);
}

// Programmatic stream serialisation, as the FP64 passes.
template <class... KArgs>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st,
                              const NttLargeArgs& a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int LOG_C, int MODE>
static cudaError_t ntt_row_attr() {
    cudaError_t e = cudaFuncSetAttribute(ntt_row<LOG_C, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ntt_row_smem<LOG_C>());
    return e;
}

// INIT: one block per tile. ITER / FINAL: one block more, for the wrap-around job.
template <int LOG_C, int MODE>
static cudaError_t ntt_row_t(const NttLargeArgs& a, cudaStream_t st) {
    return launch_pdl(ntt_row<LOG_C, MODE>, a.nblocks + (MODE == LARGE_INIT ? 0 : 1), kNttRowG * NttRowG<LOG_C>::T,
                      ntt_row_smem<LOG_C>(), st, a);
}

template <int LOG_R>
static cudaError_t ntt_col_t(const NttLargeArgs& a, cudaStream_t st) {
    // one resident wave of blocks where a single block fits an SM (N = 2^23: 224 us a pass against 234);
    // a block per column elsewhere (R = 2^11: 49 against 55)
    const int most = LOG_R >= 13 ? device_sms() : a.C;
    return launch_pdl(ntt_col<LOG_R>, a.C < most ? a.C : most, NttColG<LOG_R>::T, ntt_col_smem<LOG_R>(), st, a);
}

template <int LOG_R>
static cudaError_t ntt_col_attr() {
    cudaError_t e = cudaFuncSetAttribute(ntt_col<LOG_R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ntt_col_smem<LOG_R>());
    return e;
}

template <int LOG_C>
static cudaError_t ntt_row_attrs() {
    cudaError_t e = ntt_row_attr<LOG_C, LARGE_INIT>();
    if (!e) e = ntt_row_attr<LOG_C, LARGE_ITER>();
    if (!e) e = ntt_row_attr<LOG_C, LARGE_FINAL>();
    return e;
}

cudaError_t configure_ntt_large(int log_c, int log_r) {
    cudaError_t e;
    switch (log_c) {
        case 7: e = ntt_row_attrs<7>(); break;
        case 8: e = ntt_row_attrs<8>(); break;
        case 9: e = ntt_row_attrs<9>(); break;
        case 10: e = ntt_row_attrs<10>(); break;
        default: return cudaErrorInvalidValue;
    }
    if (e) return e;
    switch (log_r) {
        case 7: return ntt_col_attr<7>();
        case 8: return ntt_col_attr<8>();
        case 9: return ntt_col_attr<9>();
        case 10: return ntt_col_attr<10>();
        case 11: return ntt_col_attr<11>();
        case 12: return ntt_col_attr<12>();
        case 13: return ntt_col_attr<13>();
        default: return cudaErrorInvalidValue;
    }
}

template <int MODE>
static cudaError_t ntt_row_mode(int log_c, const NttLargeArgs& a, cudaStream_t st) {
    switch (log_c) {
        case 7: return ntt_row_t<7, MODE>(a, st);
        case 8: return ntt_row_t<8, MODE>(a, st);
        case 9: return ntt_row_t<9, MODE>(a, st);
        case 10: return ntt_row_t<10, MODE>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_ntt_row(int log_c, int mode, const NttLargeArgs& a, cudaStream_t st) {
    switch (mode) {
        case LARGE_INIT: return ntt_row_mode<LARGE_INIT>(log_c, a, st);
        case LARGE_ITER: return ntt_row_mode<LARGE_ITER>(log_c, a, st);
        case LARGE_FINAL: return ntt_row_mode<LARGE_FINAL>(log_c, a, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_ntt_col(int log_r, const NttLargeArgs& a, cudaStream_t st) {
    switch (log_r) {
        case 7: return ntt_col_t<7>(a, st);
        case 8: return ntt_col_t<8>(a, st);
        case 9: return ntt_col_t<9>(a, st);
        case 10: return ntt_col_t<10>(a, st);
        case 11: return ntt_col_t<11>(a, st);
        case 12: return ntt_col_t<12>(a, st);
        case 13: return ntt_col_t<13>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace llg
