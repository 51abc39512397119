// Internal declarations shared by the kernels and the C-ABI layer (not part of the public ABI).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace llg {

// Per-device record of a one-time kernel setup (cudaFuncSetAttribute applies to the current device
// only): done() for the current device, mark() after the setup succeeded there. Devices 0..63; the
// race between two first launches is benign (the setup is idempotent).
struct PerDeviceOnce {
    std::atomic<unsigned long long> bits{0};
    static int current() {
        int d = 0;
        return cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < 64 ? d : -1;
    }
    bool done() const {
        const int d = current();
        return d >= 0 && ((bits.load() >> d) & 1ull);
    }
    void mark() {
        const int d = current();
        if (d >= 0) bits.fetch_or(1ull << d);
    }
};

// SM count of the current device (148 when it cannot be asked).
inline int device_sms() {
    static std::atomic<int> sms[64];
    const int d = PerDeviceOnce::current();
    if (d < 0) return 148;
    int n = sms[d].load();
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || n <= 0) n = 148;
        sms[d].store(n);
    }
    return n;
}

// Shared-memory carve-out of the whole-test kernels: all of it. The blocks of a launch are resident
// for the whole test, so a carve-out that holds fewer of them than the registers would leaves tests
// waiting for a full test's time; the default carve-out did so in some launches (1184 tests at
// N = 512, eight an SM: 11.4 us a squaring by default, 6.4 with all of it).
constexpr int kWholeTestCarveout = 100;

enum : uint32_t {
    LLG_ST_OK = 0,
    LLG_ST_ROUNDOFF = 1,  // a round-off distance exceeded the abort threshold
};

struct SmallJob {
    uint64_t p;
    uint64_t iters;  // squarings to run (>= 1)
};

struct SmallResult {
    double max_err;
    uint64_t iters_done;
    uint64_t ns;  // device time of the test (%globaltimer)
    uint32_t status;
    uint32_t pad;
};

// FP64 whole-test kernel, N = 2^log_n with 5 <= log_n <= 13, in the form with 2^log_e values a
// thread that small_fp64_log_e gives for this many tests; qtw: the table of M = N / 2 points, in the
// form's own pass order (pass_twiddle_table) or the spread quarter table (spread_quarter_table).
// digits: njobs * N int64 (may be null).
int small_fp64_log_e(int log_n, int njobs);
bool small_fp64_pass_table(int log_e);
cudaError_t launch_small_fp64(int log_n, int log_e, const SmallJob* jobs, int njobs, const double2* qtw,
                              int64_t* digits, SmallResult* results, float* errlog,
                              double abort_err, cudaStream_t st);

// FP64 whole-test kernel for N = 2 R0 2^l (R0 = 3: l = 9..11; R0 = 5: l = 9..10); qtw: the twiddles
// mixed_twiddle_table builds for the form's values a thread.
bool mixed_length_supported(uint32_t n, int* r0, int* log_l);
int small_fp64_mixed_log_e(uint32_t n, int njobs);  // log2 of the values a thread for that many tests
cudaError_t launch_small_fp64_mixed(uint32_t n, const SmallJob* jobs, int njobs, const double2* qtw,
                                    int64_t* digits, SmallResult* results, float* errlog,
                                    double abort_err, cudaStream_t st);

// p < 256: exact multi-limb word arithmetic, one block per exponent (4 limbs out per exponent).
cudaError_t launch_word(const SmallJob* jobs, int njobs, uint64_t* res, cudaStream_t st);

// Goldilocks constants of one NTT length N (mod q): an N-th root of 2 and its inverse in Montgomery
// form (x 2^64), and 2^128 / N (1 / N in Montgomery form, times the 2^64 that the pointwise
// Montgomery square takes out).
struct NttConst {
    uint64_t root2, inv_root2, invN;
};

// Exact NTT whole-test kernel, N = 2^log_n with 6 <= log_n <= 13 (qtw: ntt_pass_table of the form's
// values a thread).
int small_ntt_values(int log_n);  // log2 of the values a thread
cudaError_t launch_small_ntt(int log_n, const SmallJob* jobs, int njobs, const uint64_t* qtw, NttConst K,
                             int64_t* digits, SmallResult* results, cudaStream_t st);

// cudaMallocAsync from the library's own pool of the current device (cudaFreeAsync frees).
cudaError_t pool_malloc(void** out, size_t bytes, cudaStream_t st);

// Adds `bytes` to the library's host-to-device copy count (llg_h2d_bytes).
void count_h2d(size_t bytes);

// Digits (int32, natural order, within one of balanced) at length n of the residue s in d_words
// (ceil(p/64) little-endian limbs, s < 2^p), formed on the GPU; enqueued on st. n <= p, digits of
// at most 30 bits.
cudaError_t digits_from_words(uint64_t p, uint64_t n, const uint64_t* d_words, int32_t* d_digits, cudaStream_t st);

// Exact residues of a whole-test batch on the GPU: cnt exponents (d_jobs[i].p <= pmax), n int64
// digits each (d_digits, natural order). Per exponent: d_res64[i], d_flags[i] (bit 0: residue zero,
// bit 1: failure) and, when d_words is non-null, the ceil(p/64) words at d_word_off[i]. Enqueued
// on st.
cudaError_t rebuild_batch(const int64_t* d_digits, const SmallJob* d_jobs, int cnt, uint32_t n, uint64_t pmax,
                          uint64_t* d_res64, int32_t* d_flags, uint64_t* d_words, const uint64_t* d_word_off,
                          cudaStream_t st);

// ---- two-pass engine (N = 2^14 .. 2^23): state resident in HBM ------------------------------

// Row-pass tiles of g rows of 2^log_c complex values that have kernels (LLG_ROW_SHAPES lists
// them as X(log_c, g)): g * 2^log_c / (values per thread) threads, a multiple of 32 up to 512,
// and at most ~180 KB of shared memory. large_rows_per_block is the default g of a row length.
#define LLG_ROW_SHAPES(X) \
    X(6, 4) X(6, 8) X(7, 2) X(7, 4) X(7, 8) X(8, 2) X(8, 4) X(8, 8) X(9, 2) X(9, 4) X(9, 8) X(10, 2) \
    X(10, 4) X(10, 8) X(11, 2) X(11, 4)
constexpr bool large_rows_supported(int log_c, int g) {
    return (log_c >= 6 && log_c <= 11) && (g == 2 || g == 4 || g == 8) && !(log_c == 6 && g == 2) &&
           !(log_c == 11 && g == 8);
}
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int large_rows_per_block(int log_c) { return log_c >= 11 ? 2 : 4; }
constexpr unsigned long long kSpinLimit = 1ull << 22;  // x ~64 ns sleeps: ~0.3 s, then give up + flag
// log2 of the complex values per thread in the row pass of g rows of 2^log_c complex: 16 for rows
// longer than 2^9, 8 up to there (two or more blocks per SM), 4 in the tiles of the shortest lengths,
// whose passes are a few blocks of a few warps (N = 2^14 7.2 -> 6.2 us a squaring, 2^16 7.6 -> 7.0, 2^18 9.6
// -> 8.9; rows of 2^8 by 4, which the longer lengths use, were slower: 2^20 18.3 -> 21.0)
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int large_row_log_e(int log_c, int g) {
    return log_c > 9 ? 4 : ((log_c <= 7 && g <= 4) || (log_c == 8 && g == 2)) ? 2 : 3;
}

// Whether the row pass reads its twiddles in pass order (pass_twiddle_table), as below 16 values a
// thread, or from the full padded table with factored products: at 16 values fifteen reads a pass
// were no faster than six and nine products (N = 2^23 138.7 against 138.0), at 8 they were (5 x 2^18 26.6
// against 27.3).
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr bool large_row_pass_table(int log_c, int g) { return large_row_log_e(log_c, g) < 4; }

struct LargeCtl {
    unsigned long long tickets;      // FP64 row-pass tickets taken since the start
    unsigned int epoch;              // squarings whose column pass has finished; +1 per column pass. The
                                     // NTT row pass reads it; an FP64 one counts by its tickets
    unsigned int ticket[2];          // NTT row-pass block tickets, alternating by epoch parity
    unsigned int timeout;            // set when a bounded wait gave up (the result is then invalid)
    unsigned long long err_max;      // bits of the max round-off over the run (double, >= 0)
    unsigned long long err_since;    // same, since the host last cleared it
};

enum { LARGE_INIT = 0, LARGE_ITER = 1, LARGE_FINAL = 2 };

#ifdef __CUDACC__
// Bounded wait until *f >= target. On giving up it sets ctl->timeout (the run's result is then
// reported invalid) and returns, so a kernel never spins forever.
__device__ __forceinline__ void wait_flag(unsigned int* f, unsigned int target, LargeCtl* ctl,
                                          unsigned long long limit) {
    volatile unsigned int* vf = f;
    unsigned long long spins = 0;
    while (*vf < target) {
        if (++spins > limit) {
            atomicExch(&ctl->timeout, 1u);
            break;
        }
        __nanosleep(64);
    }
    __threadfence();
}
#endif

// One column's carry-outs of a row tile's last row, published and read as one 16-byte access: the
// tag says whose they are, so a reader needs no separate flag (and the writer no fence).
struct __align__(16) LargeCarry {
    double c1;      // hop-1 carry-out (an integer)
    int c2;         // hop-2 carry-out (an integer of a few units)
    unsigned tag;   // epoch + 1 of the squaring they belong to
};

struct LargeArgs {
    double2* V;               // state: element (row a, column slot pos) at pos * R + a
    const double2* qtwC;      // twiddles of the C-point row FFT (large_row_pass_table)
    const double2* qtwR;      // quarter table of the R-point column FFT (spread layout for a
                              // power-of-two R, padded for R = R0 L)
    const double2* qtwL;      // R = R0 L: padded quarter table of the L-point column sub-FFTs
    const double2* tw1;       // e^{-2 pi i x / M}, x < 2^tw_shift
    const double2* tw2;       // e^{-2 pi i y 2^tw_shift / M}
    const int* pos_of_c;      // column slot of row-FFT frequency c
    const double* wA;         // [2R] 2^(sA/N) of digit 2a+e
    const double* iwA;        // [2R] 2^(-sA/N)
    const double* wB;         // [C] 2^(sB/N)
    const double* iwB;        // [C] 2^(-sB/N) / (4M)
    const uint32_t* kinds;    // digit kinds by tile and thread (fill_kinds)
    LargeCarry* carry;        // [nblocks + 1][C] carry-outs of a tile's last row: slot 0 the
                              // wrap-around job's (row R-1, one column on), k + 1 tile k's
    LargeCtl* ctl;
    unsigned int* wrap_read;  // epoch + 1 once the wrap-around job has read its rows
    unsigned long long spin_limit;  // bound of every wait on a flag (x ~64 ns sleeps)
    int* digits;              // N int32, natural order (INIT input; dump / FINAL output)
    float* errlog;            // per-epoch max round-off ring (may be null)
    int errlog_len;
    int dump;                 // ITER: also write the digits
    int pdl_late;             // where the passes let the next one launch: at their end, or at their start
    int tw_shift;
    int C, R, nblocks;
    int q;                    // p / N
};

constexpr size_t large_kind_words(size_t rc, int log_e) { return rc >> (log_e < 3 ? log_e : 3); }
// Fills LargeArgs::kinds for tiles of g rows with 2^log_e values a thread from the weight exponents sA
// ([2R] (-(2a+e) p) mod N) and sB ([C] (-2Rb p) mod N); large_kind_words of them.
cudaError_t launch_fill_kinds(uint32_t* kinds, const int* sA, const int* sB, int N, int rem, int C, int R, int g, int log_e,
                              cudaStream_t st);
// Row pass; grid > 0 overrides the block count (nblocks, + 1 for the wrap-around job unless INIT).
cudaError_t launch_large_row(int log_c, int g, int mode, const LargeArgs& a, cudaStream_t st, int grid = 0);
// Column-length code of the two-pass engine: log2 R for a power of two, 100 R0 + log2 L for the
// column length R = R0 L (launch_large_col and configure_large take it).
constexpr int large_col_code(int r0, int log_l) { return r0 == 1 ? log_l : 100 * r0 + log_l; }
cudaError_t launch_large_col(int log_r, const LargeArgs& a, cudaStream_t st);

// ---- two-pass exact NTT engine (N = 2^14 .. 2^23): N field elements in HBM ------------------

struct NttLargeArgs {
    uint64_t* V;              // state: element (row a, column slot pos) at pos * R + a
    // every constant in Montgomery form (llg_ntt.cuh)
    const uint64_t* qtwC;     // twiddles of the C-point row NTT in pass order (ntt_pass_table)
    const uint64_t* qtwR;     // twiddles of the R-point column NTT
    const uint64_t* tw1;      // w_N^x, x < 2^tw_shift
    const uint64_t* tw2;      // w_N^(y 2^tw_shift)
    const int* pos_of_c;      // column slot of row-NTT frequency c
    const uint64_t* wA;       // [R] w^sA(a), w an N-th root of 2
    const uint64_t* iwA;      // [R] w^-sA(a)
    const uint64_t* wB;       // [C] w^sB(b)
    const uint64_t* iwB;      // [C] w^-sB(b) / N, times the square's 2^64
    const uint32_t* kinds;    // digit kinds by tile and thread (fill_ntt_kinds): N / 8 words
    long long* c1;            // [nblocks + 1][C] hop-1 carry-outs of a tile's last row: slot 0 the
                              // wrap-around job's (row R-1, one column on), k + 1 tile k's
    int* c2;                  // [nblocks + 1][C] hop-2 carry-outs
    int* c3;                  // [nblocks + 1][C] hop-3 carry-outs
    LargeCtl* ctl;
    unsigned int* flags;      // [nblocks + 1] epoch + 1 once the job of that slot published its carries
    int* digits;              // N int32, natural order (INIT input; dump / FINAL output)
    int dump;
    int pdl_late;             // as LargeArgs::pdl_late
    int tw_shift;
    int C, R, nblocks;
    int q;
    int logN;
};

cudaError_t launch_fill_ntt_kinds(uint32_t* kinds, const int* sA, const int* sB, int N, int rem, int C, int R, cudaStream_t st);
cudaError_t launch_ntt_row(int log_c, int mode, const NttLargeArgs& a, cudaStream_t st);
cudaError_t launch_ntt_col(int log_r, const NttLargeArgs& a, cudaStream_t st);
cudaError_t configure_ntt_large(int log_c, int log_r);

}  // namespace llg
