// Trailing update of the blocked Cholesky: C -= L21 * L21^H on lower tiles.
//
// This is the work the reference hands to cuSOLVER inside ?potrf
// (src/Cholesky/potrf.cpp:111) and, on multi-rank grids, to herk/gemm
// (src/Cholesky/ppotrf.cpp:212-238).  For double it runs on the FP64 tensor
// cores: mma.sync m16n8k4 f64 (DMMA).  Complex double (lower) runs as two real
// DMMA products per fragment; float runs on packed FP32 FMAs (sgemm.cu), the other
// complex forms on the SIMT kernel in potrf.cu.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "ddla_kernels_internal.h"
#include "profile.h"
#include "tc_common.cuh"

namespace ddlak {

namespace {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
// one arrival on the mbarrier once the cp.async copies this thread has issued so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// D += A B over k = 4 on the FP64 tensor cores, for two 8-row blocks at once
// (mma.sync m16n8k4 f64): lane (g = lane / 4, q = lane % 4) supplies A(g, q) and
// A(g + 8, q) -- the rows of its upper and lower 8-row block -- and B(q, g), and
// holds D(g, 2q + e) in u[e] and D(g + 8, 2q + e) in v[e].  The same fragments as
// two m8n8k4 products on the two blocks, in half the instructions.
__device__ __forceinline__ void dmma2(double (&u)[2], double (&v)[2], double a_up, double a_lo, double b)
{
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(u[0]), "+d"(u[1]), "+d"(v[0]), "+d"(v[1])
                 : "d"(a_up), "d"(a_lo), "d"(b));
}

// ---------------------------------------------------------------------------
// FP64 on the tensor cores (m16n8k4 DMMA), either triangle.  A CTA owns one
// BM x BN lower tile of the region: RW x CW warps hold the accumulators; 32-column
// slices of the panel rows [ri, ri + BM) and [rj, rj + BN) come through a ring of NS
// stages with a `full` and an `empty` mbarrier each.  Every warp releases a stage by
// itself and the stage of slice c - 1 is refilled after slice c, so the warps drift
// and the DMMA pipe is not drained once per slice.
//
// Shared slices, in doubles (both keep the 8-byte fragment reads conflict free):
//   'L' storage: [32 k][rows + 4]     'U' storage (k contiguous): [rows][36]
// Two ways in:
//   TMA  thread 0, one box per operand (4 extra rows or columns pad the slice); base
//        16-byte aligned and even lda
//   CP   16-byte cp.async by all threads for any lda and any 8-byte aligned base: a line (a column of 'L', a row of 'U') that starts on an odd 8-byte
//        word is copied from one word earlier and lands one word later in its
//        slice.  The parity alternates with the line when lda is odd, and a lane's
//        fragments always come from lines of one parity, so the readers just add
//        a per-lane offset.  Words past the limits are zero-filled, not read.
// What bounds it: the DMMA pipe (FP64 tensor, 35.5 TFLOP/s by cuBLAS DGEMM); odd leading
// dimensions take some 15 % longer (a whole factorization 57.0 ms at n = 16383, 49.6 at 16384;
// the 16-byte copies of a slice are some 17 per thread against 256 DMMAs per warp).
// Every wait is bounded: if one gives up, the CTA records it in g_dmma_status,
// writes NaN into its tile (the factorization then stops at that column block with
// a failed pivot) and waits, bounded, for its copies still in flight.
// ---------------------------------------------------------------------------
constexpr int SY_BK = 32;

template <int BM_, int BN_, int RW_, int CW_, int NS_, int PER_SM_>
struct SyCfg {
    static constexpr int BM = BM_, BN = BN_, RW = RW_, CW = CW_, NS = NS_, PER_SM = PER_SM_;
    static constexpr int WM = BM / RW, WN = BN / CW;  // a warp's tile
    static constexpr int FM = WM / 8, FN = WN / 8;    // its 8 x 8 fragments
    static constexpr int WARPS = RW * CW, THREADS = 32 * WARPS;
};
using SyBig = SyCfg<128, 128, 2, 4, 3, 1>;
using SySmall = SyCfg<64, 64, 2, 2, 3, 2>;

template <bool UP>
__host__ __device__ constexpr int sy_ld(int rows) { return UP ? SY_BK + 4 : rows + 4; }
template <bool UP>
__host__ __device__ constexpr int sy_box(int rows) { return UP ? rows * sy_ld<UP>(rows) : SY_BK * sy_ld<UP>(rows); }
template <class Cfg, bool UP>
constexpr size_t sy_smem() { return (size_t)Cfg::NS * (sy_box<UP>(Cfg::BM) + sy_box<UP>(Cfg::BN)) * 8 + 128; }

__device__ int g_dmma_status;  // for a debugger: the caller sees the failed pivot

// Where the shared copy of a line starts relative to its slice row: 1 when the line's
// first word (A + start + line * lda) is not 16-byte aligned.
__device__ __forceinline__ int sy_shift(const double* A, long long lda, long long line, long long start)
{
    return (int)(((reinterpret_cast<uintptr_t>(A) >> 3) + (uintptr_t)(line * lda + start)) & 1);
}

// The CP copies of thread `t` of `nt`: `lines` lines of `len` words starting at word `start` (valid below
// wlim; lines valid below llim), line l at A + (line0 + l) * lda, into dst + l * ld.
__device__ __forceinline__ void sy_copy(double* dst, int ld, const double* A, long long lda, long long line0, int lines,
                                        long long llim, long long start, int len, long long wlim, int t,
                                        int nt)
{
    const int units = (len + 2) / 2;  // 16-byte units of a shifted line
    for (int x = t; x < lines * units; x += nt) {
        const int l = x / units, u = x - l * units;
        const long long line = line0 + l;
        const int sh = sy_shift(A, lda, line, start);
        const long long w = start - sh + 2 * u;
        const int bytes = line < llim && w < wlim ? (w + 1 < wlim ? 16 : 8) : 0;
        cp_async16(dst + l * ld + 2 * u, bytes ? A + line * lda + w : A - ((reinterpret_cast<uintptr_t>(A) >> 3) & 1),
                   bytes);
    }
}

template <class Cfg, bool UP, bool TMA, bool BATCH>  // BATCH: blockIdx.y is the matrix of a batch (3-D maps)
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::PER_SM)
    k_syrk_dmma(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
                double* __restrict__ A, long long lda, long long astride, int k0, int nbk, int n, long long t0,
                int cols, const int* __restrict__ info)
{
    constexpr int BM = Cfg::BM, BN = Cfg::BN, NS = Cfg::NS, FM = Cfg::FM, FN = Cfg::FN;
    constexpr int LDA_S = sy_ld<UP>(BM), LDB_S = sy_ld<UP>(BN), ABOX = sy_box<UP>(BM), BBOX = sy_box<UP>(BN);
    extern __shared__ __align__(128) unsigned char sy_raw[];
    __shared__ __align__(8) uint64_t full[NS], empty[NS];
    const int z = BATCH ? (int)blockIdx.y : 0;
    A += (long long)z * astride;
    info += z;
    if (*(volatile const int*)info != 0) return;
    int I, J;  // tile row and column, the tile's last row at or below its first column
    const int nct = cols == 0 ? 0 : (cols + BN - 1) / BN;
    if (cols == 0) {
        static_assert(BM == BN, "square tiles");
        tile_of_tri(blockIdx.x, I, J);
    } else {
        J = blockIdx.x % nct;
        I = blockIdx.x / nct;
        if (I < J) return;
    }
    const long long cend = cols == 0 ? (long long)n : t0 + cols;
    const long long ri = t0 + (long long)I * BM, rj = t0 + (long long)J * BN;
    double* sm = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(sy_raw) + 127) & ~uintptr_t(127));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nchunks = nbk / SY_BK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            tc::mbar_init(&full[s], TMA ? 1 : Cfg::THREADS);
            tc::mbar_init(&empty[s], Cfg::WARPS);  // one arrival per warp
        }
        tc::mbar_fence_init();
    }
    auto issue = [&](int c) {  // slice c into its stage: thread 0 (TMA) or every thread
        const int s = c % NS;
        double* st = sm + (size_t)s * (ABOX + BBOX);
        const int kc = k0 + c * SY_BK;
        if constexpr (TMA) {
            tc::mbar_expect_tx(&full[s], (ABOX + BBOX) * 8u);
            const int xa = UP ? kc : (int)ri, ya = UP ? (int)ri : kc;
            const int xb = UP ? kc : (int)rj, yb = UP ? (int)rj : kc;
            if (BATCH) {
                tc::tma_load_3d(st, &amap, &full[s], xa, ya, z);
                tc::tma_load_3d(st + ABOX, &bmap, &full[s], xb, yb, z);
            } else {
                tc::tma_load_2d(st, &amap, &full[s], xa, ya);
                tc::tma_load_2d(st + ABOX, &bmap, &full[s], xb, yb);
            }
        } else {
            const int t = threadIdx.x, nt = Cfg::THREADS;
            if (UP) {
                sy_copy(st, LDA_S, A, lda, ri, BM, n, kc, SY_BK, kc + SY_BK, t, nt);
                sy_copy(st + ABOX, LDB_S, A, lda, rj, BN, cend, kc, SY_BK, kc + SY_BK, t, nt);
            } else {
                sy_copy(st, LDA_S, A, lda, kc, SY_BK, kc + SY_BK, ri, BM, n, t, nt);
                sy_copy(st + ABOX, LDB_S, A, lda, kc, SY_BK, kc + SY_BK, rj, BN, cend, t, nt);
            }
            cp_async_arrive(&full[s]);
        }
    };
    const bool issuer = !TMA || threadIdx.x == 0;
    if (TMA && issuer) {  // the barriers are this thread's own: no need to wait for the others
        tc::prefetch_tmap(&amap);
        tc::prefetch_tmap(&bmap);
        for (int c = 0; c < NS && c < nchunks; ++c) issue(c);
    }
    __syncthreads();
    if (!TMA)
        for (int c = 0; c < NS && c < nchunks; ++c) issue(c);

    const int wm = (warp / Cfg::CW) * Cfg::WM, wn = (warp % Cfg::CW) * Cfg::WN;
    const int g = lane >> 2, q = lane & 3;
    double acc[FM][FN][2];
#pragma unroll
    for (int a = 0; a < FM; ++a)
#pragma unroll
        for (int b = 0; b < FN; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    // this lane's fragment words: row (wm + 8 a + g), k = kk + q
    const int sha = TMA ? 0 : (UP ? sy_shift(A, lda, ri + g, k0) : sy_shift(A, lda, k0 + q, ri));
    const int shb = TMA ? 0 : (UP ? sy_shift(A, lda, rj + g, k0) : sy_shift(A, lda, k0 + q, rj));
    const int fa = (UP ? (wm + g) * LDA_S + q : q * LDA_S + wm + g) + sha;
    const int fb = (UP ? (wn + g) * LDB_S + q : q * LDB_S + wn + g) + shb;
    bool ok = true;
    int consumed = 0, issued = nchunks < NS ? nchunks : NS;
    for (int c = 0; c < nchunks; ++c) {
        const int s = c % NS;
        if (!tc::mbar_wait(&full[s], (uint32_t)((c / NS) & 1), &g_dmma_status, 0x41)) {
            ok = false;
            break;
        }
        consumed = c + 1;
        const double* As = sm + (size_t)s * (ABOX + BBOX) + fa;
        const double* Bs = sm + (size_t)s * (ABOX + BBOX) + ABOX + fb;
#pragma unroll
        for (int kk = 0; kk < SY_BK; kk += 4) {
            double af[FM], bf[FN];
#pragma unroll
            for (int a = 0; a < FM; ++a) af[a] = As[UP ? 8 * a * LDA_S + kk : kk * LDA_S + 8 * a];
#pragma unroll
            for (int b = 0; b < FN; ++b) bf[b] = Bs[UP ? 8 * b * LDB_S + kk : kk * LDB_S + 8 * b];
#pragma unroll
            for (int a = 0; a < FM; a += 2)
#pragma unroll
                for (int b = 0; b < FN; ++b) dmma2(acc[a][b], acc[a + 1][b], af[a], af[a + 1], bf[b]);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);  // this warp is done with stage s
        if (issuer && c >= 1 && c - 1 + NS < nchunks) {
            const int cp = c - 1;  // refill slice cp's stage with slice cp + NS
            if (!tc::mbar_wait(&empty[cp % NS], (uint32_t)((cp / NS) & 1), &g_dmma_status, 0x44)) {
                ok = false;
                break;
            }
            issue(cp + NS);
            issued = cp + NS + 1;
        }
    }
    if (!TMA) cp_wait_all();
    ok = __syncthreads_and(ok);
    if (TMA && !ok) {  // copies issued for slices consumed .. issued - 1 may still be in flight
        if (threadIdx.x == 0)
            for (int c = consumed; c < issued; ++c)
                (void)tc::mbar_wait(&full[c % NS], (uint32_t)((c / NS) & 1), &g_dmma_status, 0x42);
        __syncthreads();
    }
    if (!ok) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
        for (int a = 0; a < FM; ++a)
#pragma unroll
            for (int b = 0; b < FN; ++b) acc[a][b][0] = acc[a][b][1] = nan;
    }

    // C -= acc on the lower part of the region; the C values of two fragment rows are loaded
    // together before any store, so the loads overlap instead of serialising behind the stores
#pragma unroll
    for (int a2 = 0; a2 < FM; a2 += 2) {
        double cv[2][FN][2];
        bool in[2][FN][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int b = 0; b < FN; ++b)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const long long i = ri + wm + (a2 + h) * 8 + g;
                    const long long jj = rj + wn + b * 8 + 2 * q + e;
                    in[h][b][e] = i < n && jj < cend && i >= jj;
                    cv[h][b][e] = in[h][b][e] ? __ldcg(UP ? A + jj + i * lda : A + i + jj * lda) : 0.0;
                }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int b = 0; b < FN; ++b)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (!in[h][b][e]) continue;
                    const long long i = ri + wm + (a2 + h) * 8 + g;
                    const long long jj = rj + wn + b * 8 + 2 * q + e;
                    *(UP ? A + jj + i * lda : A + i + jj * lda) = cv[h][b][e] - acc[a2 + h][b][e];
                }
    }
}

template <class Cfg, bool UP, bool BATCH>
cudaError_t launch_syrk(double* A, long long lda, long long astride, int batch, int k0, int nbk, int n, long long t0,
                        int cols, const int* dinfo, cudaStream_t st)
{
    const long long tr = ceil_div((long long)n - t0, Cfg::BM);
    const dim3 grid((unsigned)(cols == 0 ? tr * (tr + 1) / 2 : tr * ceil_div(cols, Cfg::BN)), (unsigned)batch);
    constexpr size_t smem = sy_smem<Cfg, UP>();
    CUtensorMap amap{}, bmap{};
    auto encode = [&](CUtensorMap* map, int rows) {
        const int bx = UP ? sy_ld<UP>(rows) : rows + 4, by = UP ? rows : SY_BK;
        if (BATCH)
            return tc::encode_colmajor_3d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, n, n, lda, batch, astride, bx, by);
        return tc::encode_colmajor_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, n, n, lda, bx, by,
                                      CU_TENSOR_MAP_SWIZZLE_NONE);
    };
    cudaError_t e = cudaSuccess;
    if (!(t0 & 1) && encode(&amap, Cfg::BM) && encode(&bmap, Cfg::BN)) {
        auto* k = k_syrk_dmma<Cfg, UP, true, BATCH>;
        if ((e = smem_optin(k, smem)) != cudaSuccess) return e;
        k<<<grid, Cfg::THREADS, smem, st>>>(amap, bmap, A, lda, astride, k0, nbk, n, t0, cols, dinfo);
    } else if constexpr (BATCH) {
        return cudaErrorInvalidValue;  // its one caller takes even leading dimensions and aligned bases only
    } else {
        auto* k = k_syrk_dmma<Cfg, UP, false, false>;
        if ((e = smem_optin(k, smem)) != cudaSuccess) return e;
        k<<<grid, Cfg::THREADS, smem, st>>>(amap, bmap, A, lda, astride, k0, nbk, n, t0, cols, dinfo);
    }
    return cudaGetLastError();
}

}  // namespace

// Fewest 128 x 128 tiles for which they are used.  A region with fewer leaves SMs idle
// (one such CTA per SM), and 64 x 64 tiles, two per SM, spread it.  ms of a whole factorization,
// nothing else changed, with 128 x 128 tiles always / from 148 / never:
//   lower  n = 1024 .466 / .351 / .351   2048 .974 / .756 / .750   5003 3.82 / 3.33 / 3.25
//          8192 9.27 / 8.24 / 8.04       16384 51.6 / 49.6 / 50.5
//   upper  2048 1.22 / .945 / .945       5003 5.09 / 4.21 / 4.13   16384 58.7 / 57.3 / 55.6
// Lines at 74, 148 and 296 tiles are within 3 % of one another at every order.
constexpr long long kSyrkBigTiles = 148;

// The FP64 update of a batch of equal-order matrices (batch 1: one matrix, astride unused),
// nbk a multiple of 32.
template <bool UP, bool BATCH>
static cudaError_t syrk_dmma(double* A, long long lda, long long astride, int batch, int k0, int nbk, int n,
                             long long t0, int cols, const int* dinfo, cudaStream_t st)
{
    const long long m = (long long)n - t0;
    if (m <= 0) return cudaSuccess;
    if (nbk <= 0 || nbk % SY_BK != 0) return cudaErrorInvalidValue;
    const long long t = ceil_div(m, 128);
    const long long tiles = (cols == 0 ? t * (t + 1) / 2 : t * ceil_div(cols, 128)) * batch;
    if (tiles < kSyrkBigTiles)
        return launch_syrk<SySmall, UP, BATCH>(A, lda, astride, batch, k0, nbk, n, t0, cols, dinfo, st);
    return launch_syrk<SyBig, UP, BATCH>(A, lda, astride, batch, k0, nbk, n, t0, cols, dinfo, st);
}

cudaError_t launch_syrk_batched(double* A, long long lda, long long astride, int batch, int k0, int nbk, int n,
                                long long t0, int cols, const int* dinfo, cudaStream_t st)
{
    if (batch < 1 || batch > 65535) return cudaErrorInvalidValue;
    return syrk_dmma<false, true>(A, lda, astride, batch, k0, nbk, n, t0, cols, dinfo, st);
}

namespace {

// ---------------------------------------------------------------------------
// Complex double (lower storage) on the FP64 tensor cores.  With K interleaved
// as k' = 2k + c (c = real, imaginary part) and b the conjugated operand,
//   Re C -= sum_k' A'(i, k') B'(k', j),  A'(i, 2k + c) = part c of a(i, k)
//   Im C -= sum_k' A''(i, k') B'(k', j), A''(i, 2k) = Im a(i, k), A''(i, 2k+1) = -Re a(i, k)
// with B'(2k + c, j) = part c of b(j, k): two real DMMA products per fragment
// pair, and one 16-byte shared load of a(i, k) gives a lane both its A' and A''
// values.  Tiles of 64 x 64 complex, 4 warps of 32 x 32, 16 complex k per stage
// by TMA over the matrix seen as 2n x n doubles (rows 2 ri .. 2 ri + 135: the 4
// extra complex rows pad the shared tile), 3 stages, bounded waits as above.
// ---------------------------------------------------------------------------
constexpr int ZT_BM = 64, ZT_BK = 16, ZT_LDS = 2 * (ZT_BM + 4), ZT_NS = 3;  // ZT_LDS in doubles (136)
constexpr int ZT_BOX = ZT_BK * ZT_LDS;
constexpr unsigned ZT_BOX_BYTES = ZT_BOX * 8u;                   // 17408
constexpr size_t ZT_SMEM = (size_t)ZT_NS * 2 * ZT_BOX_BYTES + 128;

__global__ void __launch_bounds__(128) k_herk_zmma_tma(const __grid_constant__ CUtensorMap amap,
                                                       cf64* __restrict__ A, long long lda, int k0, int nbk, int n,
                                                       long long t0, int cols, const int* __restrict__ info)
{
    extern __shared__ __align__(128) unsigned char zt_raw[];
    __shared__ __align__(8) uint64_t full[ZT_NS];
    if (*(volatile const int*)info != 0) return;
    int I, J;
    if (cols == 0) {
        tile_of_tri(blockIdx.x, I, J);
    } else {
        const int nct = (cols + ZT_BM - 1) / ZT_BM;
        J = blockIdx.x % nct;
        I = blockIdx.x / nct;
        if (I < J) return;
    }
    const long long cend = cols == 0 ? (long long)n : t0 + cols;
    const long long ri = t0 + (long long)I * ZT_BM, rj = t0 + (long long)J * ZT_BM;
    double* sm = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(zt_raw) + 127) & ~uintptr_t(127));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp >> 1, wn = warp & 1;  // 2 x 2 warps of 32 x 32
    const int g = lane >> 2, q = lane & 3;
    const int nchunks = nbk / ZT_BK;

    auto issue = [&](int c) {
        const int s = c % ZT_NS;
        double* st = sm + (size_t)s * 2 * ZT_BOX;
        tc::mbar_expect_tx(&full[s], 2 * ZT_BOX_BYTES);
        tc::tma_load_2d(st, &amap, &full[s], (int)(2 * ri), k0 + c * ZT_BK);
        tc::tma_load_2d(st + ZT_BOX, &amap, &full[s], (int)(2 * rj), k0 + c * ZT_BK);
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < ZT_NS; ++s) tc::mbar_init(&full[s], 1);
        tc::mbar_fence_init();
        tc::prefetch_tmap(&amap);
        for (int c = 0; c < ZT_NS && c < nchunks; ++c) issue(c);
    }
    __syncthreads();

    double re[4][4][2], im[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = 0.0;

    bool ok = true;
    int consumed = 0;
    const int part = q & 1;
    for (int c = 0; c < nchunks; ++c) {
        const int s = c % ZT_NS;
        ok = __syncthreads_and(tc::mbar_wait(&full[s], (uint32_t)((c / ZT_NS) & 1), &g_dmma_status, 0x43));
        if (!ok) break;
        consumed = c + 1;
        const double* As = sm + (size_t)s * 2 * ZT_BOX;
        const double* Bs = As + ZT_BOX;
#pragma unroll
        for (int kk = 0; kk < 2 * ZT_BK; kk += 4) {  // real k' = kk + q, complex k = kk/2 + q/2
            const int kc = kk / 2 + (q >> 1);
            double a1[4], a2[4], bf[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double2 v = *reinterpret_cast<const double2*>(&As[kc * ZT_LDS + 2 * (wm * 32 + a * 8 + g)]);
                a1[a] = part ? v.y : v.x;   // A'
                a2[a] = part ? -v.x : v.y;  // A''
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const double2 v = *reinterpret_cast<const double2*>(&Bs[kc * ZT_LDS + 2 * (wn * 32 + b * 8 + g)]);
                bf[b] = part ? v.y : v.x;
            }
#pragma unroll
            for (int a = 0; a < 4; a += 2)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    dmma2(re[a][b], re[a + 1][b], a1[a], a1[a + 1], bf[b]);
                    dmma2(im[a][b], im[a + 1][b], a2[a], a2[a + 1], bf[b]);
                }
        }
        __syncthreads();
        if (threadIdx.x == 0 && c + ZT_NS < nchunks) issue(c + ZT_NS);
    }
    if (!ok) {
        if (threadIdx.x == 0) {
            for (int c = consumed; c < nchunks && c < consumed + ZT_NS; ++c)
                (void)tc::mbar_wait(&full[c % ZT_NS], (uint32_t)((c / ZT_NS) & 1), &g_dmma_status, 0x44);
        }
        __syncthreads();
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = nan;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        cf64 cv[4][2];
        bool in[4][2];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const long long i = ri + wm * 32 + a * 8 + g;
                const long long jj = rj + wn * 32 + b * 8 + 2 * q + e;
                in[b][e] = i < n && jj < cend && i >= jj;
                if (in[b][e]) {
                    const double2 v = __ldcg(reinterpret_cast<const double2*>(A + i + jj * lda));
                    cv[b][e] = {v.x, v.y};
                } else {
                    cv[b][e] = {0.0, 0.0};
                }
            }
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (!in[b][e]) continue;
                const long long i = ri + wm * 32 + a * 8 + g;
                const long long jj = rj + wn * 32 + b * 8 + 2 * q + e;
                A[i + jj * lda] = cf64{cv[b][e].x - re[a][b][e], cv[b][e].y - im[a][b][e]};
            }
    }
}

bool launch_zmma_tma(cf64* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                     cudaStream_t st, cudaError_t* err)
{
    if ((reinterpret_cast<uintptr_t>(A) & 15) || nbk % ZT_BK != 0 || nbk <= 0) return false;
    const long long m = (long long)n - t0;
    if (m <= 0) {
        *err = cudaSuccess;
        return true;
    }
    CUtensorMap amap;  // the complex matrix as 2n x n doubles, columns 2 lda doubles apart
    if (!tc::encode_colmajor_2d(&amap, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, 2LL * n, n, 2 * lda, ZT_LDS, ZT_BK,
                                CU_TENSOR_MAP_SWIZZLE_NONE))
        return false;
    if ((*err = smem_optin(k_herk_zmma_tma, ZT_SMEM)) != cudaSuccess) return true;
    const long long t = ceil_div(m, ZT_BM);
    const long long grid = cols == 0 ? t * (t + 1) / 2 : t * ceil_div(cols, ZT_BM);
    k_herk_zmma_tma<<<(unsigned)grid, 128, ZT_SMEM, st>>>(amap, A, lda, k0, nbk, n, t0, cols, dinfo);
    *err = cudaGetLastError();
    return true;
}

}  // namespace

template <class T, bool UP>
cudaError_t trailing_update(T* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                            cudaStream_t st)
{
    if constexpr (std::is_same<T, double>::value) {
        return syrk_dmma<UP, false>(A, lda, 0, 1, k0, nbk, n, t0, cols, dinfo, st);
    }
    if constexpr (std::is_same<T, float>::value) return syrk_f32<UP>(A, lda, k0, nbk, n, t0, cols, dinfo, st);
    if constexpr (std::is_same<T, cf64>::value && !UP) {
        cudaError_t e = cudaSuccess;
        if (launch_zmma_tma(A, lda, k0, nbk, n, t0, cols, dinfo, st, &e)) return e;
    }
    if constexpr (Traits<T>::cplx) return trailing_update_simt<T, UP>(A, lda, k0, nbk, n, t0, cols, dinfo, st);
    return cudaErrorInvalidValue;
}

#define DDLAK_INST_TU(T, UP)                                                                                        \
    template cudaError_t trailing_update<T, UP>(T*, long long, int, int, int, long long, int, const int*, cudaStream_t);
DDLAK_INST_TU(float, false)
DDLAK_INST_TU(float, true)
DDLAK_INST_TU(double, false)
DDLAK_INST_TU(double, true)
DDLAK_INST_TU(cf32, false)
DDLAK_INST_TU(cf32, true)
DDLAK_INST_TU(cf64, false)
DDLAK_INST_TU(cf64, true)
#undef DDLAK_INST_TU

}  // namespace ddlak
