// The panel chain of the blocked Cholesky for real types: the 128 x 128
// diagonal block and the rows below it, both on the FP64 tensor cores
// (mma.sync m16n8k4 f64), arithmetic in FP64 for FP64 and FP32 storage.
// Both kernels work on 16-row strips held in registers as 8-column DMMA
// accumulator tiles and walk the block's 8-column steps from the left:
//
//   step j:  X = C_j Inv_j^T        Inv_j = L_jj^-1, the 8 x 8 diagonal tile's inverse
//            C_l -= X L_lj^T        for the strip's tiles l > j
//
// An accumulator fragment holds columns 2q and 2q + 1 of its row; read as the
// two k = 4 operands of the next product it supplies columns {0, 2, 4, 6} and
// {1, 3, 5, 7}, and since the sum over k has no order the B fragments are simply
// read in the same order, (2q, 2q + 1) as one 16-byte load: no shuffle.  The
// product's destination tile is the next lower one (C_(l-1) = C_l - ...), so the
// strip moves down one tile per step and the step loop stays rolled and its code in
// the instruction cache.
#include <type_traits>

#include <ddla_kernels.h>

#include "common.cuh"
#include "ddla_kernels_internal.h"
#include "profile.h"
#include "tile8.cuh"

namespace ddlak {

namespace {

constexpr int PN_NB = 128;           // block order
constexpr int PN_TILES = PN_NB / 8;  // 8-column steps

// d = c + a b, fragments as above (u: row g, v: row g + 8, columns 2q + e).  Not volatile:
// the two products of a tile depend on each other, and only if the compiler may put other
// tiles' between them is their latency (25 clocks) hidden.
__device__ __forceinline__ void dmma4(double (&d)[4], const double (&c)[4], double a_up, double a_lo, double b)
{
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
                 : "=d"(d[0]), "=d"(d[1]), "=d"(d[2]), "=d"(d[3])
                 : "d"(a_up), "d"(a_lo), "d"(b), "d"(c[0]), "d"(c[1]), "d"(c[2]), "d"(c[3]));
}

// X = C Inv^T for one tile of a strip (Inv row-major)
__device__ __forceinline__ void tile_solve(double (&X)[4], const double (&C)[4], const double* Inv, int g, int q)
{
    const double2 b = *reinterpret_cast<const double2*>(&Inv[g * 8 + 2 * q]);
    const double z[4] = {0.0, 0.0, 0.0, 0.0};
    double Y[4];
    dmma4(Y, z, C[0], C[2], b.x);
    dmma4(X, Y, C[1], C[3], b.y);
}
// the same where C holds NaN or infinities
__device__ __forceinline__ void tile_solve_rows(double (&X)[4], const double (&C)[4], const double* Inv, int lane)
{
    const double2 u = tri_row(C[0], C[1], Inv, 1, 8, true, lane), v = tri_row(C[2], C[3], Inv, 1, 8, true, lane);
    X[0] = u.x, X[1] = u.y, X[2] = v.x, X[3] = v.y;
}

// C_(l-1) = C_l - X B_l^T for the strip's tiles L0 <= l < L0 + G, as straight-line code: all the
// operand loads, then the first products, then the second ones, so that neither the loads'
// nor the products' latency is exposed (with a branch per tile a product took 59 clocks).
// tile(l) gives this lane's operand pair of tile l; it is called past the last tile too.
template <int L0, int G, class Tile>
__device__ __forceinline__ void strip_update(double (&C)[PN_TILES][4], const double (&X)[4], Tile tile)
{
    double2 b[G];
    double Y[G][4];
#pragma unroll
    for (int i = 0; i < G; ++i) b[i] = tile(L0 + i);
#pragma unroll
    for (int i = 0; i < G; ++i) dmma4(Y[i], C[L0 + i], -X[0], -X[2], b[i].x);
#pragma unroll
    for (int i = 0; i < G; ++i) dmma4(C[L0 + i - 1], Y[i], -X[1], -X[3], b[i].y);
}

template <bool UP>
__device__ __forceinline__ long long lpos(long long lda, long long i, long long j)
{
    return UP ? j + i * lda : i + j * lda;
}

// Named barriers of the diagonal kernel.
constexpr int DG_WORKERS = 8, DG_THREADS = 32 * (DG_WORKERS + 1);
template <int ID, int COUNT>
__device__ __forceinline__ void bar_sync()
{
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(COUNT) : "memory");
}
template <int ID, int COUNT>
__device__ __forceinline__ void bar_arrive()
{
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(COUNT) : "memory");
}

}  // namespace

// ---------------------------------------------------------------------------
// The diagonal block [k0, k0 + nbk)^2, nbk <= 128 (padded with the identity).
// Nine warps: warp 0 factors the 8 x 8 diagonal tile of each step, the other
// eight hold the block's 16-row strips.  Per step the strip that owns the
// diagonal tile hands it to warp 0 through shared memory; every lane of warp 0
// factors it redundantly in registers (no shuffles: a column costs one
// reciprocal square root, a multiply and a multiply-add) and lane c carries
// column c of the tile's inverse along; the strips then form X, publish it and
// update.  Warp 0's scheduler (warp id mod 4) gets only the two strips with the
// fewest tiles, so the chain does not queue behind the strips' DMMAs.
// info as LAPACK ?potrf: the first pivot that is not positive; the columns
// before it are final, it keeps its updated value.
// What bounds it: the chain of 128 dependent pivots, 16 steps of some 1900 clocks (the tile
// 1150, the hand-overs and the next tile's update the rest).  Measured on one B200: 16 us a
// block, against 36 us for 32-column panels with one warp's shared-memory column chain.
// ---------------------------------------------------------------------------
template <class S, bool UP>
__global__ void __launch_bounds__(DG_THREADS, 1) k_potrf_diag_dmma(S* __restrict__ A, long long lda, long long astride,
                                                                   int k0, int nbk, int* __restrict__ info)
{
    __shared__ __align__(16) double T[64];        // the diagonal tile, row-major
    __shared__ __align__(16) double Inv[64];      // its inverse, row-major
    __shared__ __align__(16) double Lt[64];       // its factor, row-major (warp 0's own)
    __shared__ __align__(16) double Xs[PN_NB * 8];  // the step's X, row-major
    __shared__ int s_fail;                        // 0, or 1 + the failed column of the current tile
    A += (long long)blockIdx.x * astride;  // blockIdx.x: the matrix of a batch
    info += blockIdx.x;
    if (*(volatile const int*)info != 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int steps = (nbk + 7) >> 3;
    S* Ab = A + lpos<UP>(lda, k0, k0);

    if (warp == 0) {
        for (int j = 0; j < steps; ++j) {
            bar_sync<1, 64>();  // T is in
            const int good = factor_tile8(T, Inv, Lt, nullptr, 8, lane);
            if (lane == 0) s_fail = good == 8 ? 0 : good + 1;
            bar_sync<2, DG_THREADS>();
            // the tile itself, two entries a lane
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int e = lane + 32 * x, r = UP ? e >> 3 : e & 7, c = UP ? e & 7 : e >> 3;
                if (c <= r && 8 * j + r < nbk) Ab[lpos<UP>(lda, 8 * j + r, 8 * j + c)] = (S)Lt[r * 8 + c];
            }
            __syncwarp();
            if (good < 8) {
                if (lane == 0) *info = k0 + 8 * j + good + 1;
                return;
            }
        }
        return;
    }

    // strips: the two lightest (rows 0.. and 16..) share warp 0's scheduler
    const int w = warp == 1 ? 7 : warp == 2 ? 6 : warp == 3 ? 5 : warp == 4 ? 0 : warp == 5 ? 2 : warp == 6 ? 3
                  : warp == 7 ? 4 : 1;
    const int r_up = 16 * w + g, r_lo = r_up + 8;
    double C[PN_TILES][4];
#pragma unroll
    for (int l = 0; l < PN_TILES; ++l) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = h ? r_lo : r_up, c = 8 * l + 2 * q + e;
                C[l][2 * h + e] = r == c && r >= nbk ? 1.0 : 0.0;
                if (c <= r && r < nbk) C[l][2 * h + e] = (double)Ab[lpos<UP>(lda, r, c)];
            }
    }
    // rows below step j's diagonal tile, the tile's first `good` columns
    auto store = [&](int j, const double (&X)[4], int good) {
        if (2 * w + 1 < j) return;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = h ? r_lo : r_up, c = 2 * q + e;
                if (r >= 8 * (j + 1) && r < nbk && c < good) Ab[lpos<UP>(lda, r, 8 * j + c)] = (S)X[2 * h + e];
            }
    };
    const bool odd = any_nonfinite(C);
    double X[4] = {0.0, 0.0, 0.0, 0.0};
    int fail = 0;
#pragma unroll 1
    for (int j = 0; j < steps; ++j) {
        const int cnt = 2 * w + 1 - j;  // tiles of this strip after tile j
        if (w == (j >> 1)) {
            if (j & 1) *reinterpret_cast<double2*>(&T[g * 8 + 2 * q]) = make_double2(C[0][2], C[0][3]);
            else *reinterpret_cast<double2*>(&T[g * 8 + 2 * q]) = make_double2(C[0][0], C[0][1]);
            bar_arrive<1, 64>();
        }
        if (j > 0) store(j - 1, X, 8);  // once the tile is handed over: off the chain
        bar_sync<2, DG_THREADS>();      // Inv and s_fail are in
        fail = s_fail;
        if (cnt >= 0) {
            tile_solve(X, C[0], Inv, g, q);
            // (a failed pivot may have put NaN in its column of every row)
            if (odd || fail) tile_solve_rows(X, C[0], Inv, lane);
            *reinterpret_cast<double2*>(&Xs[r_up * 8 + 2 * q]) = make_double2(X[0], X[1]);
            *reinterpret_cast<double2*>(&Xs[r_lo * 8 + 2 * q]) = make_double2(X[2], X[3]);
        }
        bar_sync<3, 32 * DG_WORKERS>();
        if (fail) {  // uniform over the workers
            store(j, X, fail - 1);
            return;
        }
        // (a branch per tile: the owner of the next diagonal tile, on the chain, has one or two)
#pragma unroll
        for (int l = 1; l < PN_TILES; ++l) {
            if (l > cnt) break;
            const double2 b = *reinterpret_cast<const double2*>(&Xs[(8 * (j + l) + g) * 8 + 2 * q]);
            double Y[4];
            dmma4(Y, C[l], -X[0], -X[2], b.x);
            dmma4(C[l - 1], Y, -X[1], -X[3], b.y);
        }
    }
    store(steps - 1, X, 8);
}

template <class S, bool UP>
cudaError_t launch_potrf_diag(S* A, long long lda, long long astride, int batch, int k0, int nbk, int* dinfo,
                              cudaStream_t st)
{
    k_potrf_diag_dmma<S, UP><<<(unsigned)batch, DG_THREADS, 0, st>>>(A, lda, astride, k0, nbk, dinfo);
    note_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// X L11^H = A21 for the rows below the diagonal block.  One warp per 16-row
// strip, four per CTA; L11's lower 8 x 8 tiles in shared memory (row-major, the
// 16-byte units of a row rotated by half the row index so that fragment loads
// and the column-wise fill are spread over the banks), the diagonal tiles'
// inverses formed by 128 threads (one column each) on the way.
// What bounds it: 272 DMMAs per strip (34 clocks each on a scheduler's FP64 pipe, 4.9 us),
// after L11's load and the inverses.  Measured: 13 us for the panels of n = 2048 (load 2.6,
// inverses 0.7, steps 9.4), against 33 us for one thread per row.  No alignment is asked of
// A, so there is one form for all.
// ---------------------------------------------------------------------------
namespace {
constexpr int TR_NT = 128, TR_ROWS = 64;
constexpr int TR_LTILES = PN_TILES * (PN_TILES + 1) / 2;
constexpr size_t TR_SMEM = (size_t)(TR_LTILES + PN_TILES) * 64 * sizeof(double);

// element (g, m) of tile (l, j), l >= j
__device__ __forceinline__ int tr_tile(int l, int j) { return (l * (l + 1) / 2 + j) * 64; }
__device__ __forceinline__ int tr_elem(int g, int m) { return g * 8 + (((m >> 1) ^ (g >> 1)) << 1) + (m & 1); }
}  // namespace

template <class S, bool UP>
__global__ void __launch_bounds__(TR_NT) k_trsm_panel_dmma(S* __restrict__ A, long long lda, long long astride, int k0,
                                                           int nbk, int n, const int* __restrict__ info)
{
    extern __shared__ __align__(16) double tr_smem[];
    __shared__ double Rp[PN_NB];
    double* Lt = tr_smem;
    double* Inv = tr_smem + TR_LTILES * 64;  // row-major 8 x 8 tiles
    A += (long long)blockIdx.y * astride;    // blockIdx.y: the matrix of a batch
    info += blockIdx.y;
    if (*(volatile const int*)info != 0) return;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int g = lane >> 2, q = lane & 3;
    const S* Ad = A + lpos<UP>(lda, k0, k0);
    // L11's tiles: a thread takes every other tile of line t and the others of line 127 - t ('L': a
    // line is a row, its tiles to the left of the diagonal; 'U': a column, its tiles below), so
    // that all threads copy about as much; consecutive threads on consecutive words
    auto fill = [&](int line, int par) {
        const int lt = line >> 3, li = line & 7;
        int off[8];  // word of the line's m-th entry in a tile
#pragma unroll
        for (int m = 0; m < 8; ++m) off[m] = UP ? tr_elem(m, li) : tr_elem(li, m);
        for (int o = (UP ? lt : 0) + par; o < (UP ? PN_TILES : lt + 1); o += 2) {
            double* dst = Lt + (UP ? tr_tile(o, lt) : tr_tile(lt, o));
            const S* src = Ad + lpos<UP>(lda, UP ? 8 * o : line, UP ? line : 8 * o);
            const long long step = lda;  // the next entry of the line
            S v[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const int r = UP ? 8 * o + m : line, c = UP ? line : 8 * o + m;
                const bool in = c <= r && r < nbk;
                if constexpr (std::is_same<S, double>::value) {
                    cp_async_elem<8>(dst + off[m], in ? src + m * step : Ad, in);
                } else {
                    v[m] = *(in ? src + m * step : Ad);
                    if (!in) v[m] = S(0);
                }
            }
            if constexpr (!std::is_same<S, double>::value) {
#pragma unroll
                for (int m = 0; m < 8; ++m) dst[off[m]] = (double)v[m];
            }
        }
    };
    fill(t, 0);
    fill(PN_NB - 1 - t, 1);
    if constexpr (std::is_same<S, double>::value) cp_group_commit();
    // this warp's strip (its loads overlap the fill above)
    const long long row0 = (long long)k0 + nbk + (long long)blockIdx.x * TR_ROWS + warp * 16;
    const long long r_up = row0 + g, r_lo = r_up + 8;
    double C[PN_TILES][4];
    if (nbk == PN_NB && row0 + 16 <= n) {  // whole strip: plain loads, in flight until the loop needs them
        const S* in = A + lpos<UP>(lda, r_up, k0 + 2 * q);
        const long long e_col = UP ? 1 : lda, e_row = UP ? 8 * lda : 8;
#pragma unroll
        for (int l = 0; l < PN_TILES; ++l)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) C[l][2 * h + e] = (double)in[(8 * l + e) * e_col + h * e_row];
    } else {
#pragma unroll
        for (int l = 0; l < PN_TILES; ++l)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const long long r = h ? r_lo : r_up;
                    const int c = 8 * l + 2 * q + e;
                    C[l][2 * h + e] = r < n && c < nbk ? (double)A[lpos<UP>(lda, r, k0 + c)] : 0.0;
                }
    }
    if constexpr (std::is_same<S, double>::value) cp_group_wait<0>();
    __syncthreads();
    // the reciprocal pivots, one a thread (rows at or past nbk: the identity)
    {
        const double l = t < nbk ? Lt[tr_tile(t >> 3, t >> 3) + tr_elem(t & 7, t & 7)] : 1.0;
        Rp[t] = isinf(l) ? 0.0 : recip_pivot(l);  // (the square root of a positive double is normal)
    }
    __syncthreads();
    {
        // column c of tile b's inverse: L y = e_c
        const int b = t >> 3, c = t & 7;
        const double* tile = Lt + tr_tile(b, b);
        double l[8][8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
            for (int k = 0; k < i; ++k) l[i][k] = tile[tr_elem(i, k)];
            l[i][i] = Rp[8 * b + i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            double s = i == c ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < i; ++k) s = fma(-l[i][k], y[k], s);
            y[i] = s * l[i][i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) Inv[b * 64 + i * 8 + c] = y[i];
    }
    __syncthreads();
    if (row0 >= n) return;
    const int steps = (nbk + 7) >> 3;
    const int unit = ((q ^ (g >> 1)) << 1) + g * 8;
    S* out = A + lpos<UP>(lda, r_up, k0 + 2 * q);  // this lane's entries of the step's columns
    const long long e_col = UP ? 1 : lda, e_row = UP ? 8 * lda : 8, e_step = UP ? 8 : 8 * lda;
    auto run = [&](auto odd) {
#pragma unroll 1
        for (int j = 0; j < steps; ++j) {
            double X[4];
            if constexpr (decltype(odd)::value) tile_solve_rows(X, C[0], Inv + j * 64, lane);
            else tile_solve(X, C[0], Inv + j * 64, g, q);
            const int cnt = steps - 1 - j;
            auto tile = [&](int l) {
                const int r = j + l < PN_TILES ? j + l : PN_TILES - 1;
                return *reinterpret_cast<const double2*>(&Lt[tr_tile(r, j) + unit]);
            };
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (8 * j + 2 * q + e < nbk) {
                    if (r_up < n) out[e * e_col] = (S)X[e];
                    if (r_lo < n) out[e * e_col + e_row] = (S)X[2 + e];
                }
            }
            out += e_step;
            if (cnt >= 1) strip_update<1, 5>(C, X, tile);
            if (cnt >= 6) strip_update<6, 5>(C, X, tile);
            if (cnt >= 11) strip_update<11, 5>(C, X, tile);
        }
    };
    // (two loops: with the choice in the loop the panels of n = 2048 took 2 us longer each)
    if (any_nonfinite(C)) run(std::true_type{});
    else run(std::false_type{});
}

template <class S, bool UP>
cudaError_t launch_trsm_panel_dmma(S* A, long long lda, long long astride, int batch, int k0, int nbk, int n,
                                   const int* dinfo, cudaStream_t st)
{
    const long long m = (long long)n - k0 - nbk;
    if (m <= 0) return cudaSuccess;
    if (cudaError_t e = smem_optin(k_trsm_panel_dmma<S, UP>, TR_SMEM); e != cudaSuccess) return e;
    const double md = (double)m, b = nbk, nm = batch;
    ProfScope ps(PK_TRSM_PANEL, st, nm * md * b * b, nm * sizeof(S) * (2.0 * md * b + b * (b + 1) / 2));
    const dim3 grid((unsigned)ceil_div(m, TR_ROWS), (unsigned)batch);
    k_trsm_panel_dmma<S, UP><<<grid, TR_NT, TR_SMEM, st>>>(A, lda, astride, k0, nbk, n, dinfo);
    note_launches(1);
    return cudaGetLastError();
}

#define DDLAK_INST_PANEL(S, UP)                                                                                   \
    template cudaError_t launch_potrf_diag<S, UP>(S*, long long, long long, int, int, int, int*, cudaStream_t);   \
    template cudaError_t launch_trsm_panel_dmma<S, UP>(S*, long long, long long, int, int, int, int, const int*, \
                                                       cudaStream_t);
DDLAK_INST_PANEL(float, false)
DDLAK_INST_PANEL(float, true)
DDLAK_INST_PANEL(double, false)
DDLAK_INST_PANEL(double, true)
#undef DDLAK_INST_PANEL

}  // namespace ddlak
