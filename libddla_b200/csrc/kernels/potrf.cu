// Blocked right-looking Cholesky with look-ahead (ddla::ppotrf / ddla::potrf on
// a 1x1 grid).
//
// Replaces the vendor call the reference makes at src/Cholesky/potrf.cpp:106-113
// (cusolverDn?potrf).  Per block column k of width NB:
//   1. the NB x NB diagonal block: real types on the FP64 tensor cores
//      (k_potrf_diag_dmma, panel.cu), complex types in shared memory in 32-wide
//      steps (k_potrf_diag, diag_factor.cuh); info detected in-kernel;
//   2. L21 = A21 * L11^{-H}: real types on the FP64 tensor cores
//      (k_trsm_panel_dmma, panel.cu); complex types by k_trsm_panel, warps own
//      rows, lanes own columns, each solved entry broadcast with a warp shuffle;
//   3. trailing update -- C -= L21 * L21^H on lower tiles (FP64 DMMA for double and
//                        lower complex double, syrk.cu; packed FP32 FMAs for float,
//                        sgemm.cu; register-tiled SIMT for the rest).
// Look-ahead: the update of block column k+1 plus the diagonal block and panel
// of k+1 run on a high-priority internal stream while the update of the rest
// of the trailing matrix runs on the caller's stream; events order the two so
// that no tile is touched by both at once.
// info follows LAPACK ?potrf: the order of the first leading minor that is not
// positive definite (diagonal value <= 0 or NaN), 0 on success.  Every kernel
// returns immediately once info is set, so the first failure is the one kept.
#include <climits>
#include <mutex>
#include <type_traits>

#include <ddla_kernels.h>

#include "common.cuh"
#include "ddla_kernels_internal.h"
#include "diag_factor.cuh"
#include "profile.h"
#include "tc_common.cuh"

namespace ddlak {

// ---------------------------------------------------------------------------
// 1. diagonal block
// ---------------------------------------------------------------------------
// (one CTA runs: the bound lets it use the registers.  Without, the compiler stopped at 147 for
// single complex: 112 / 121 us for a lower / upper 128 x 128 block against 92 / 99.)
template <class T, bool UP>
__global__ void __launch_bounds__(256, 1) k_potrf_diag(T* __restrict__ A, long long lda, int k0, int nbk,
                                                    int* __restrict__ info)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* s = reinterpret_cast<T*>(smem_raw);
    const int ld = diag_block_ld(nbk);
    if (*(volatile int*)info != 0) return;
    load_lview_block<T, UP>(s, ld, A, lda, k0, k0, nbk, nbk, nbk, nbk, true);
    const int fail = factor_block_smem<T>(s, ld, nbk);
    if (nbk == 128) {  // the full block: index arithmetic by shifts
        for (int idx = threadIdx.x; idx < 128 * 128; idx += blockDim.x) {
            const int i = UP ? idx >> 7 : idx & 127, j = UP ? idx & 127 : idx >> 7;
            if (i >= j) lview_st<T, UP>(A, lda, k0 + i, k0 + j, s[i + j * ld]);
        }
    } else {
        for (int idx = threadIdx.x; idx < nbk * nbk; idx += blockDim.x) {
            const int i = idx % nbk, j = idx / nbk;
            if (i >= j) lview_st<T, UP>(A, lda, k0 + i, k0 + j, s[i + j * ld]);
        }
    }
    if (fail && threadIdx.x == 0) *info = k0 + fail;
}

// ---------------------------------------------------------------------------
// 2. panel: X * L11^H = A21 for the rows below the diagonal block.
//    Each warp owns PR rows; lane l owns columns l, l+32, ... of those rows.
// ---------------------------------------------------------------------------
template <class T, bool UP, int NQ, int PR>
__global__ void __launch_bounds__(256) k_trsm_panel(T* __restrict__ A, long long lda, int k0, int nbk, int n,
                                                    const int* __restrict__ info)
{
    using R = real_t<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* l11 = reinterpret_cast<T*>(smem_raw);  // [c + j*ldl], c,j < NQ*32, zero outside nbk
    const int ldl = NQ * 32 + 1;
    __shared__ R s_rinv[NQ * 32];
    if (*(volatile int*)info != 0) return;

    load_lview_block<T, UP>(l11, ldl, A, lda, k0, k0, nbk, nbk, NQ * 32, NQ * 32, true);
    // multiply by reciprocal pivots, as reference BLAS ?trsm does for side 'R'
    for (int j = threadIdx.x; j < NQ * 32; j += blockDim.x) s_rinv[j] = j < nbk ? R(1) / re(l11[j + j * ldl]) : R(0);
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // persistent over row groups of 8 warps x PR rows: L11 is loaded once per CTA
    const long long ngroups = ceil_div((long long)n - k0 - nbk, 8LL * PR);
    for (long long grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const long long row0 = (long long)k0 + nbk + (grp * (blockDim.x >> 5) + warp) * PR;
        if (row0 >= n) continue;
        T p[PR][NQ];
#pragma unroll
        for (int r = 0; r < PR; ++r)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const long long i = row0 + r;
                const int c = q * 32 + lane;
                p[r][q] = (i < n && c < nbk) ? lview_ld<T, UP>(A, lda, i, k0 + c) : zero<T>();
            }

#pragma unroll
        for (int qj = 0; qj < NQ; ++qj) {
            for (int jj = 0; jj < 32; ++jj) {
                const int j = qj * 32 + jj;
                if (j >= nbk) break;
                const R rjj = s_rinv[j];
                T x[PR];
#pragma unroll
                for (int r = 0; r < PR; ++r) {
                    const T v = scal(p[r][qj], rjj);
                    if (lane == jj) p[r][qj] = v;
                    x[r] = shfl(v, jj);
                }
#pragma unroll
                for (int q = qj; q < NQ; ++q) {
                    const int c = q * 32 + lane;
                    if (c > j) {
                        const T lcj = cj(l11[c + j * ldl]);
#pragma unroll
                        for (int r = 0; r < PR; ++r) p[r][q] = fms(p[r][q], x[r], lcj);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < PR; ++r)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const long long i = row0 + r;
                const int c = q * 32 + lane;
                if (i < n && c < nbk) lview_st<T, UP>(A, lda, i, k0 + c, p[r][q]);
            }
    }
}

// Grid of the panel solve: every row group once, at most as many CTAs as fit on
// the device at once (the kernel loops over row groups).
template <class K>
long long trsm_grid(K* kernel, size_t smem, long long groups)
{
    static std::mutex mu;
    static int cap[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return groups;
    std::lock_guard<std::mutex> lk(mu);
    if (cap[dev] == 0) {
        int sms = 148, per = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, smem);
        cap[dev] = sms * (per > 0 ? per : 1);
    }
    return groups < cap[dev] ? groups : cap[dev];
}

// ---------------------------------------------------------------------------
// 3. generic trailing update (SIMT; the complex types).  64x64 tiles, 16-wide k
//    chunks through shared memory, 4x4 per thread.  Region: rows [t0, n) and
//    columns [t0, n) (cols == 0, lower triangle of tiles) or [t0, t0+cols).
// ---------------------------------------------------------------------------
template <class T, bool UP>
__global__ void __launch_bounds__(256) k_syrk_simt(T* __restrict__ A, long long lda, int k0, int nbk, int n,
                                                   long long t0, int cols, const int* __restrict__ info)
{
    constexpr int BT = 64, BK = 16;
    __shared__ T As[BK][BT + 1];
    __shared__ T Bs[BK][BT + 1];
    if (*(volatile int*)info != 0) return;
    int I, J;
    if (cols == 0) {
        tile_of_tri(blockIdx.x, I, J);
    } else {
        const int nct = (cols + BT - 1) / BT;
        J = blockIdx.x % nct;
        I = blockIdx.x / nct;
        if (I < J) return;
    }
    const long long cend = cols == 0 ? (long long)n : t0 + cols;
    const long long ri = t0 + (long long)I * BT, rj = t0 + (long long)J * BT;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = zero<T>();

    for (int kc = 0; kc < nbk; kc += BK) {
        for (int idx = threadIdx.x; idx < BT * BK; idx += 256) {
            int i, k;
            if (UP) { k = idx % BK; i = idx / BK; } else { i = idx % BT; k = idx / BT; }
            const bool kin = kc + k < nbk;
            As[k][i] = (kin && ri + i < n) ? lview_ld<T, UP>(A, lda, ri + i, k0 + kc + k) : zero<T>();
            Bs[k][i] = (kin && rj + i < cend) ? lview_ld<T, UP>(A, lda, rj + i, k0 + kc + k) : zero<T>();
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            T av[4], bv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) av[a] = As[k][tx + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) bv[b] = cj(Bs[k][ty + 16 * b]);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma_(acc[a][b], av[a], bv[b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const long long i = ri + tx + 16 * a, j = rj + ty + 16 * b;
            if (i < n && j < cend && i >= j) {
                T c = lview_ld<T, UP>(A, lda, i, j);
                lview_st<T, UP>(A, lda, i, j, sub(c, acc[a][b]));
            }
        }
}

template <class T, bool UP>
cudaError_t trailing_update_simt(T* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                                 cudaStream_t st)
{
    const long long m = (long long)n - t0;
    if (m <= 0) return cudaSuccess;
    const long long t = ceil_div(m, 64);
    const long long grid = cols == 0 ? t * (t + 1) / 2 : t * ceil_div(cols, 64);
    k_syrk_simt<T, UP><<<(unsigned)grid, 256, 0, st>>>(A, lda, k0, nbk, n, t0, cols, dinfo);
    return cudaGetLastError();
}

#define DDLAK_INST_SIMT(T, UP)                                                                                      \
    template cudaError_t trailing_update_simt<T, UP>(T*, long long, int, int, int, long long, int, const int*,     \
                                                     cudaStream_t);
DDLAK_INST_SIMT(cf32, false)
DDLAK_INST_SIMT(cf32, true)
DDLAK_INST_SIMT(cf64, false)
DDLAK_INST_SIMT(cf64, true)
#undef DDLAK_INST_SIMT

// ---------------------------------------------------------------------------
// host-side enqueue of the whole factorization
// ---------------------------------------------------------------------------
template <class T> constexpr int potrf_nb() { return sizeof(T) == 16 ? 64 : 128; }

// The diagonal block: real types on the FP64 tensor cores (panel.cu), complex types
// in shared memory.
template <class T, bool UP>
static cudaError_t diag_block(T* A, long long lda, int k0, int nbk, int* dinfo, cudaStream_t s)
{
    const double cf = Traits<T>::cplx ? 4.0 : 1.0, b = nbk;
    ProfScope ps(PK_POTRF_DIAG, s, cf * b * b * b / 3.0, sizeof(T) * b * (b + 1));
    if constexpr (!Traits<T>::cplx) {
        return launch_potrf_diag<T, UP>(A, lda, 0, 1, k0, nbk, dinfo, s);
    } else {
        k_potrf_diag<T, UP><<<1, 256, (size_t)nbk * diag_block_ld(nbk) * sizeof(T), s>>>(A, lda, k0, nbk, dinfo);
        note_launches(1);
        return cudaGetLastError();
    }
}

// X L11^H = A21 for the rows below it
template <class T, bool UP>
static cudaError_t panel_solve(T* A, long long lda, int k0, int nbk, int n, const int* dinfo, cudaStream_t s)
{
    if constexpr (!Traits<T>::cplx) {
        return launch_trsm_panel_dmma<T, UP>(A, lda, 0, 1, k0, nbk, n, dinfo, s);
    } else {
        constexpr int NQ = potrf_nb<T>() / 32;
        constexpr int PR = sizeof(T) >= 16 ? 4 : 8;
        const size_t panel_smem = (size_t)(NQ * 32) * (NQ * 32 + 1) * sizeof(T);
        const long long m = (long long)n - k0 - nbk;
        if (m <= 0) return cudaSuccess;
        const double md = (double)m, b = nbk;
        ProfScope ps(PK_TRSM_PANEL, s, 4.0 * md * b * b, sizeof(T) * (2.0 * md * b + b * (b + 1) / 2));
        const long long grid = trsm_grid(k_trsm_panel<T, UP, NQ, PR>, panel_smem, ceil_div(m, 8 * PR));
        k_trsm_panel<T, UP, NQ, PR><<<(unsigned)grid, 256, panel_smem, s>>>(A, lda, k0, nbk, n, dinfo);
        note_launches(1);
        return cudaGetLastError();
    }
}

namespace {
struct LookaheadRes {
    cudaStream_t hi = nullptr;
    cudaEvent_t start = nullptr, panel = nullptr, rest = nullptr;
};
LookaheadRes& lookahead_res()
{
    static thread_local LookaheadRes res[64];
    int dev = 0;
    cudaGetDevice(&dev);
    LookaheadRes& r = res[dev & 63];
    if (r.hi == nullptr) {
        int least = 0, greatest = 0;
        cudaDeviceGetStreamPriorityRange(&least, &greatest);
        cudaStreamCreateWithPriority(&r.hi, cudaStreamNonBlocking, greatest);
        cudaEventCreateWithFlags(&r.start, cudaEventDisableTiming);
        cudaEventCreateWithFlags(&r.panel, cudaEventDisableTiming);
        cudaEventCreateWithFlags(&r.rest, cudaEventDisableTiming);
    }
    return r;
}
}  // namespace

template <class T, bool UP>
static cudaError_t potrf_enqueue(T* A, long long lda, int n, int G, int* dinfo, cudaStream_t st)
{
    constexpr int NB = potrf_nb<T>();
    if constexpr (Traits<T>::cplx) {
        constexpr int NQ = NB / 32;
        constexpr int PR = sizeof(T) >= 16 ? 4 : 8;
        const size_t diag_smem = (size_t)NB * diag_block_ld(NB) * sizeof(T);
        const size_t panel_smem = (size_t)(NQ * 32) * (NQ * 32 + 1) * sizeof(T);
        if (cudaError_t e = smem_optin(k_potrf_diag<T, UP>, diag_smem); e != cudaSuccess) return e;
        if (cudaError_t e = smem_optin(k_trsm_panel<T, UP, NQ, PR>, panel_smem); e != cudaSuccess) return e;
    }
    const double cf = Traits<T>::cplx ? 4.0 : 1.0;  // real flops per multiply-add relative to a real one
    LookaheadRes& L = lookahead_res();
    cudaStream_t hi = L.hi;

    cudaError_t panel_err = cudaSuccess;
    auto diag_and_panel = [&](int k0, cudaStream_t s) {
        const int nbk = n - k0 < NB ? n - k0 : NB;
        cudaError_t pe = diag_block<T, UP>(A, lda, k0, nbk, dinfo, s);
        if (pe == cudaSuccess) pe = panel_solve<T, UP>(A, lda, k0, nbk, n, dinfo, s);
        if (pe != cudaSuccess && panel_err == cudaSuccess) panel_err = pe;
    };
    // C -= L(:, k0 : k0 + kw) L(:, k0 : k0 + kw)^H on the region from row / column t0
    auto update = [&](int k0, int kw, long long t0, int cols, cudaStream_t s) -> cudaError_t {
        const double md = (double)(n - t0), b = kw;
        const double cw = cols ? (double)cols : md;
        const double fl = cols ? cf * 2.0 * b * (md * cw - cw * (cw - 1) / 2) : cf * md * (md + 1) * b;
        ProfScope ps(PK_SYRK_UPDATE, s, fl, sizeof(T) * ((cols ? 2.0 * md * cw : md * (md + 1)) + md * b));
        const cudaError_t e = trailing_update<T, UP>(A, lda, k0, kw, n, t0, cols, dinfo, s);
        note_launches(1);
        return e;
    };

    // Super-steps of G block columns: the chain on the high-priority stream factors
    // them one after the other (block g first takes the left-looking update from
    // blocks 0..g-1 of the super-step), then updates the next super-step's G block
    // columns (look-ahead); the caller's stream updates everything to their right
    // with K = G NB in one pass, so the trailing matrix is read and written once
    // per G block columns.  The caller's stream waits for the super-step's panels;
    // the chain waits for the previous trailing update before its look-ahead; the
    // two touch disjoint tiles.
    const long long SW = (long long)G * NB;
    cudaEventRecord(L.start, st);
    cudaStreamWaitEvent(hi, L.start, 0);
    bool have_rest = false;
    cudaError_t e = cudaSuccess;
    for (long long k0 = 0; k0 < n; k0 += SW) {
        for (int g = 0; g < G; ++g) {
            const long long kg = k0 + (long long)g * NB;
            if (kg >= n) break;
            if (g > 0) {
                const int cols = (long long)n - kg < NB ? (int)(n - kg) : NB;
                if ((e = update((int)k0, g * NB, kg, cols, hi)) != cudaSuccess) return e;
            }
            diag_and_panel((int)kg, hi);
        }
        const long long t0 = k0 + SW;
        if (t0 >= n) break;
        cudaEventRecord(L.panel, hi);
        if (have_rest) cudaStreamWaitEvent(hi, L.rest, 0);
        const int la_cols = (long long)n - t0 < SW ? (int)(n - t0) : (int)SW;
        if ((e = update((int)k0, (int)SW, t0, la_cols, hi)) != cudaSuccess) return e;
        have_rest = false;
        if (t0 + SW < n) {
            cudaStreamWaitEvent(st, L.panel, 0);
            if ((e = update((int)k0, (int)SW, t0 + SW, 0, st)) != cudaSuccess) return e;
            cudaEventRecord(L.rest, st);
            have_rest = true;
        }
    }
    // join
    cudaEventRecord(L.panel, hi);
    cudaStreamWaitEvent(st, L.panel, 0);
    if (panel_err != cudaSuccess) return panel_err;
    return cudaGetLastError();
}

// Block columns per super-step.  A wide super-step reads and writes the trailing matrix
// less often, but its left-looking updates (K up to 128 (G - 1) on one block column)
// lie on the chain, which is all of the time at small orders.  The orders from which 2, 4
// and 8 are the faster, by type, triangle and, for FP32, whether the update's tiles
// come by TMA (the cp.async form gains more from a long K).  ms with G = 1 / 2 / 4 / 8, leading dimension n, on both sides of the lines:
//   d L      3584  1.56 / 1.60 / 1.79 / 2.08    4096  1.98 / 1.98 / 2.18 / 2.65    6144  5.00 / 4.42 / 4.48 / 4.96
//            7168  7.42 / 6.32 / 6.11 / 6.71    10240 - / 16.2 / 14.7 / 14.7       12288 - / 26.6 / 23.7 / 23.2
//   d U      1536  .650 / .649 / .709 / .803    4096  2.77 / 2.51 / 2.54 / 2.96    4608  3.64 / 3.23 / 3.13 / 3.43
//            7168  12.0 / 8.70 / 7.53 / 7.66    8192  17.4 / 12.3 / 10.3 / 10.1    16384 - / 88.8 / 66.6 / 57.4
//   s L TMA  7168  5.56 / 5.70 / 6.63 / 8.45    8192  7.24 / 7.21 / 8.28 / 10.4    24576 - / 111.8 / 112.1 / 117.2
//   s U TMA  5120  3.85 / 3.90 / 4.53 / 5.98    6144  5.83 / 5.49 / 6.12 / 7.80    7168  9.00 / 7.84 / 8.07 / 10.0
//            8192  13.4 / 11.0 / 10.6 / 12.7    12288 44.7 / 33.4 / 28.9 / 29.3    14336 70.2 / 51.6 / 43.9 / 42.5
//   s L odd  2047  1.62 / 1.62 / 1.79 / 2.20    4001  4.38 / 3.98 / 4.10 / 4.89    5003  6.82 / 5.82 / 5.74 / 6.75
//            10001 36.9 / 23.7 / 18.5 / 18.8    12287 67.9 / 41.4 / 29.8 / 28.2
//   s U odd  2047  1.39 / 1.48 / 1.72 / 2.20    3001  2.47 / 2.42 / 2.79 / 3.45    6001  8.16 / 6.52 / 6.66 / 8.11
//            7003  11.9 / 9.19 / 8.90 / 10.6    10001 35.4 / 23.8 / 19.5 / 19.7    12287 64.3 / 41.9 / 32.6 / 30.8
//   c L      8192  24.7 / 25.1 / 26.7 / 29.8    10240 44.0 / 43.5 / 45.2 / 49.4    16384 159.1 / 153.4 / 153.6 / 159.5
//            24576 - / 495.0 / 494.5 / 511.3
//   c U      6144  15.5 / 15.7 / 16.7 / 19.2    7168  21.9 / 21.1 / 22.6 / 25.5    10240 55.5 / 51.0 / 51.1 / 55.3
//            12288 91.0 / 82.6 / 80.7 / 85.7    24576 - / 600.6 / 586.0 / 604.6
//   z L      4608  9.26 / 9.46 / 9.92 / 11.5    5120  11.4 / 11.0 / 12.0 / 13.7    7168  24.1 / 22.6 / 22.6 / 25.4
//            14336 - / 140.1 / 134.2 / 134.3    20480 - / 392.3 / 373.9 / 368.5
//   z U      4096  9.23 / 9.38 / 10.4 / 12.4    4608  12.2 / 12.0 / 13.0 / 15.5    7168  34.7 / 31.8 / 32.3 / 35.9
//            8192  50.3 / 45.0 / 44.2 / 48.2    20480 - / 604.9 / 577.0 / 584.9
// (odd leading dimensions of d lie at the same lines: L 6001 4.83 / 4.82, U 4001 2.87 / 2.89 for 2 / 4.)
static int potrf_group(char type, char uplo, int n, bool tma)
{
    constexpr int never = INT_MAX;
    const bool up = uplo == 'U';
    struct Lines { int two, four, eight; };
    const Lines l = type == 'd'   ? (up ? Lines{1536, 4352, 7680} : Lines{4096, 6400, 10240})
                    : type == 'c' ? (up ? Lines{6400, 11264, never} : Lines{9728, 16384, never})
                    : type == 'z' ? (up ? Lines{4352, 7680, never} : Lines{4864, 7168, 14848})
                    : tma         ? (up ? Lines{5376, 7680, 13312} : Lines{7936, never, never})
                                  : (up ? Lines{2560, 6400, 11008} : Lines{2048, 4608, 11008});
    return n >= l.eight ? 8 : n >= l.four ? 4 : n >= l.two ? 2 : 1;
}

template <class T>
static cudaError_t potrf_typed(char uplo, int n, int G, void* A, long long lda, int* dinfo, cudaStream_t st)
{
    if (uplo == 'U') return potrf_enqueue<T, true>(static_cast<T*>(A), lda, n, G, dinfo, st);
    return potrf_enqueue<T, false>(static_cast<T*>(A), lda, n, G, dinfo, st);
}

}  // namespace ddlak

// ---------------------------------------------------------------------------
// L L^T x = b for a batch of factored equal-order FP64 matrices (lower, order
// <= 1024, one right-hand side each), one CTA per matrix with x in shared
// memory; log det = 2 sum log l_ii on the way.  Forward, by 32-row blocks: warp
// 0 solves the block (lane i owns row i; x_j times 1 / l_jj, then broadcast),
// every thread updates its rows below with the block's 32 columns (coalesced
// column reads, a row's 32 in flight together).  Backward, by 32-row blocks from
// the end: each warp forms four of the block's dot products with the solved x
// below (coalesced, their loads in flight together, warp sums), then warp 0 solves
// the transposed block from a shared copy.  A matrix with info != 0 keeps b and
// gets log det = NaN.  What bounds it: load latency over its 64 block steps.
// ---------------------------------------------------------------------------
constexpr int PB_NT = 256, PB_NMAX = 1024;

__global__ void __launch_bounds__(PB_NT) k_potrs_batched_f64(int n, const double* __restrict__ Lg, long long lda,
                                                             long long astride, double* __restrict__ Bg,
                                                             long long bstride, const int* __restrict__ info,
                                                             double* __restrict__ logdet)
{
    __shared__ double x[PB_NMAX];
    __shared__ double blk[32][33];
    __shared__ double s_ld;
    const int m = blockIdx.x, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (info[m] != 0) {
        if (t == 0 && logdet) logdet[m] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    const double* L = Lg + (long long)m * astride;
    double* B = Bg + (long long)m * bstride;
    for (int i = t; i < n; i += PB_NT) x[i] = B[i];
    double ld = 0.0;  // warp 0: sum of log l_ii over the rows its lanes own
    __syncthreads();
    for (int b0 = 0; b0 < n; b0 += 32) {
        const int w = n - b0 < 32 ? n - b0 : 32;
        // the block's lower triangle into shared memory first (all warps, coalesced), so that
        // warp 0's chain reads no global memory
        for (int e = t; e < 32 * 32; e += PB_NT) {
            const int r = e & 31, c = e >> 5;
            blk[r][c] = (r < w && c <= r) ? L[(b0 + r) + (long long)(b0 + c) * lda] : 0.0;
        }
        __syncthreads();
        if (warp == 0) {
            double xi = lane < w ? x[b0 + lane] : 0.0;
            const double dl = lane < w ? blk[lane][lane] : 1.0, ri = 1.0 / dl;
            ld += log(dl);
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {  // columns at or past w are zero
                if (lane == j) xi *= ri;
                const double xj = __shfl_sync(0xffffffffu, xi, j);
                if (lane > j) xi = fma(-blk[lane][j], xj, xi);
            }
            if (lane < w) x[b0 + lane] = xi;
        }
        __syncthreads();
        for (int r = b0 + 32 + t; r < n; r += PB_NT) {  // only below a full block (w = 32)
            double acc = x[r];
            const double* lr = L + r + (long long)b0 * lda;
            double l[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) l[j] = lr[(long long)j * lda];
#pragma unroll
            for (int j = 0; j < 32; ++j) acc = fma(-l[j], x[b0 + j], acc);
            x[r] = acc;
        }
        __syncthreads();
    }
    if (warp == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if (lane == 0) s_ld = 2.0 * ld;
    }
    for (int b0 = ((n - 1) / 32) * 32; b0 >= 0; b0 -= 32) {
        const int w = n - b0 < 32 ? n - b0 : 32;
        // x_i -= sum_{r >= b0 + 32} l(r, b0 + i) x_r for the block's columns i (w = 32 when there is such r)
        if (b0 + 32 < n) {
            constexpr int CW = 32 / (PB_NT / 32);
            const double* lc = L + (long long)(b0 + CW * warp) * lda;
            double acc[CW];
#pragma unroll
            for (int c = 0; c < CW; ++c) acc[c] = 0.0;
#pragma unroll 4
            for (int r = b0 + 32 + lane; r < n; r += 32) {
                const double xr = x[r];
#pragma unroll
                for (int c = 0; c < CW; ++c) acc[c] = fma(lc[r + c * lda], xr, acc[c]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < CW; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < CW; ++c) x[b0 + CW * warp + c] -= acc[c];
        }
        for (int e = t; e < 32 * 32; e += PB_NT) {  // the block itself, for the transposed solve
            const int r = e & 31, c = e >> 5;
            blk[r][c] = (r < w && c <= r) ? L[(b0 + r) + (long long)(b0 + c) * lda] : 0.0;
        }
        __syncthreads();
        if (warp == 0) {
            double xi = lane < w ? x[b0 + lane] : 0.0;
            const double ri = lane < w ? 1.0 / blk[lane][lane] : 0.0;
#pragma unroll 8
            for (int j = 31; j >= 0; --j) {  // rows at or past w are zero
                if (lane == j) xi *= ri;
                const double xj = __shfl_sync(0xffffffffu, xi, j);
                if (lane < j) xi = fma(-blk[j][lane], xj, xi);
            }
            if (lane < w) x[b0 + lane] = xi;
        }
        __syncthreads();
    }
    for (int i = t; i < n; i += PB_NT) B[i] = x[i];
    if (t == 0 && logdet) logdet[m] = s_ld;
}

// A batch of equal-order FP64 matrices (lower), right-looking by super-steps of
// G block columns of 128, each step one launch per kernel over the whole batch:
// the diagonal blocks (one CTA per matrix), the panels (16-row strips, grid.y = matrix;
// both panel.cu) and the updates (TMA DMMA tiles, grid.y = matrix).  In a
// super-step, block column g first takes the update of its own 128 columns by
// block columns 0 .. g-1 (K = 128 g), and the rest of the trailing matrix is
// updated once with K = 128 G, so the trailing matrix is read and written once
// per 128 G columns and the update tiles run long K.
#ifndef BATCHED_POTRF_GROUP
#define BATCHED_POTRF_GROUP 4
#endif
extern "C" int ddlak_potrf_batched_f64(int batch, int n, void* A_, long long lda, long long astride, int* dinfo,
                                       void* stream)
{
    using namespace ddlak;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* A = static_cast<double*>(A_);
    if (batch < 0 || n < 0 || (batch > 0 && (!A || !dinfo || lda < n || astride < lda * (long long)n)))
        return (int)cudaErrorInvalidValue;
    if (batch == 0) return 0;
    if (batch > 65535 || (lda & 1) || (astride & 1) || (reinterpret_cast<uintptr_t>(A) & 15))
        return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(dinfo, 0, sizeof(int) * (size_t)batch, st);
    if (e != cudaSuccess || n == 0) return (int)e;
    constexpr int NB = 128, G = BATCHED_POTRF_GROUP;
    const double nb3 = (double)batch;
    auto diag_and_panel = [&](int k0) -> cudaError_t {
        const int nbk = n - k0 < NB ? n - k0 : NB;
        const double b = nbk;
        {
            ProfScope ps(PK_POTRF_DIAG, st, nb3 * b * b * b / 3.0, nb3 * 8.0 * b * (b + 1));
            if (cudaError_t de = launch_potrf_diag<double, false>(A, lda, astride, batch, k0, nbk, dinfo, st);
                de != cudaSuccess)
                return de;
        }
        return launch_trsm_panel_dmma<double, false>(A, lda, astride, batch, k0, nbk, n, dinfo, st);
    };
    // C -= L(:, k0 : k0 + kw) L(:, k0 : k0 + kw)^T on the region from t0 (all of it, or cols columns)
    auto update = [&](int k0, int kw, long long t0, int cols) -> cudaError_t {
        const double md = (double)(n - t0), b = kw;
        const double cw = cols ? (double)cols : md;
        const double fl = cols ? 2.0 * b * (md * cw - cw * (cw - 1) / 2) : md * (md + 1) * b;
        ProfScope ps(PK_SYRK_UPDATE, st, nb3 * fl, nb3 * 8.0 * ((cols ? 2.0 * md * cw : md * (md + 1)) + md * b));
        const cudaError_t ue = launch_syrk_batched(A, lda, astride, batch, k0, kw, n, t0, cols, dinfo, st);
        note_launches(1);
        return ue;
    };
    for (int k0 = 0; k0 < n; k0 += G * NB) {
        if ((e = diag_and_panel(k0)) != cudaSuccess) return (int)e;
        // block column g of the super-step: the update of its own columns by block columns
        // 0 .. g-1 of the super-step (left-looking, K = 128 g), then its factor
        for (int g = 1; g < G; ++g) {
            const int kg = k0 + g * NB;
            if (kg >= n) break;
            const int cg = n - kg < NB ? n - kg : NB;
            if ((e = update(k0, g * NB, kg, cg)) != cudaSuccess) return (int)e;
            if ((e = diag_and_panel(kg)) != cudaSuccess) return (int)e;
        }
        const long long t0 = (long long)k0 + G * NB;
        if (t0 >= n) break;
        if ((e = update(k0, G * NB, t0, 0)) != cudaSuccess) return (int)e;
    }
    return (int)cudaGetLastError();
}

extern "C" int ddlak_potrs_batched_f64(int batch, int n, const void* L, long long lda, long long astride, void* B,
                                       long long bstride, const int* dinfo, double* logdet, void* stream)
{
    using namespace ddlak;
    if (batch < 0 || n < 0 || n > PB_NMAX) return (int)cudaErrorInvalidValue;
    if (batch == 0 || n == 0) return 0;
    if (!L || !B || !dinfo || lda < n || astride < lda * (long long)n || bstride < n)
        return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const double nn = n;
    ProfScope ps(PK_POTRS_FUSED, st, 2.0 * batch * nn * nn, 8.0 * batch * nn * (nn + 1));
    k_potrs_batched_f64<<<(unsigned)batch, PB_NT, 0, st>>>(n, static_cast<const double*>(L), lda, astride,
                                                         static_cast<double*>(B), bstride, dinfo, logdet);
    note_launches(1);
    return (int)cudaGetLastError();
}

extern "C" int ddlak_potrf_grouped(char type, char uplo, int group, int n, void* A, long long lda, int* dinfo,
                                   void* stream)
{
    using namespace ddlak;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (group < 1 || group > DDLAK_POTRF_MAX_GROUP) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(dinfo, 0, sizeof(int), st);
    if (e != cudaSuccess) return (int)e;
    if (n <= 0) return 0;
    switch (type) {
    case 's': e = potrf_typed<float>(uplo, n, group, A, lda, dinfo, st); break;
    case 'd': e = potrf_typed<double>(uplo, n, group, A, lda, dinfo, st); break;
    case 'c': e = potrf_typed<cf32>(uplo, n, group, A, lda, dinfo, st); break;
    case 'z': e = potrf_typed<cf64>(uplo, n, group, A, lda, dinfo, st); break;
    default: return (int)cudaErrorInvalidValue;
    }
    return (int)e;
}

extern "C" int ddlak_potrf(char type, char uplo, int n, void* A, long long lda, int* dinfo, void* stream)
{
    const bool tma = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;  // as sg::encode for FP32
    return ddlak_potrf_grouped(type, uplo, ddlak::potrf_group(type, uplo, n, tma), n, A, lda, dinfo, stream);
}
