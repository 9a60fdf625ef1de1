// Batched uneven Cholesky: factor, solve and log-determinant of thousands of
// independent Hermitian positive-definite matrices of different orders in ONE
// persistent launch (no reference counterpart; the per-matrix equivalent is
// ppotrf + ppotrs + diag_logdet, src/Cholesky/ppotrf.cpp:326-349,
// ppotrs.cpp:65-85, diag_logdet.cpp:42-55).
//
// Scheduling: grid = SMs x resident CTAs.  Each CTA takes the next matrix from
// a device work list (sorted by decreasing order, so the largest start first:
// longest-processing-time order) with one atomicAdd, processes it alone, and
// takes the next.  The last CTA to leave resets the two counters, so the same
// launch can be replayed (it is captured in a CUDA graph by the host).
//
// Per matrix (order n <= NMAX, lower storage, lda >= n), 256 threads, on the FP64
// tensor cores (mma.sync m16n8k4 f64; FP64 arithmetic for both storages):
//   left-looking by block columns of width W (a tuned choice per matrix, see
//   ddlak_vbatched_variants), rows in rounds of 128: warp w holds the 16-row strip w
//   of the round as W / 8 accumulator tiles, subtracts L(rows, 0:J) L(J:J+W, 0:J)^T
//   with 16-column slices of both staged in shared memory (16-byte cp.async for any
//   lda, see vb_copy), then
//     * round 0 is the diagonal block, factored in 8-column steps as panel.cu does: the
//       owner of the 8 x 8 diagonal tile hands it to a warp that holds no strip (the
//       tile and a strip together would not fit the registers), which factors it with
//       its inverse; the strips form X = C Inv^T, publish it and update;
//     * every other strip is solved against the published block.
//   The right-hand side is row n of the matrix: its forward substitution is the same
//   arithmetic.  The backward one runs after it in steps of 32 rows.  log det A is
//   -2 sum log(1 / l_jj).
// What bounds it: at small orders the chain of pivots (two CTAs per SM cover each
// other's), at large ones the DMMA pipe.  Measured, time of a CTA per matrix at full
// residency (FP64, solve included, W = 64): n = 64 30 us, 256 237 us, 512 1.04 ms; 4096
// matrices of 16 .. 512: FP64 9.4 -> 4.4 ms, FP32 6.4 -> 4.3 ms against block columns in
// registers on the FP64 / FP32 pipes.  At two CTAs per SM 28 (FP32) to 48 (FP64) bytes spill.
// info follows LAPACK ?potrf (order of the first non-positive leading minor);
// a failed matrix keeps its right-hand side and gets logdet NaN.
#include <cuda_runtime.h>

#include <type_traits>

#include <ddla_kernels.h>

#include "common.cuh"
#include "tile8.cuh"
#include "profile.h"

namespace ddlak {
namespace {

constexpr int VB_NT = 256;   // threads per CTA
constexpr int VB_KC = 16;    // columns per staged slice
constexpr int VB_ROWS = 128; // rows per round
constexpr int VB_BW = 32;    // rows per backward-substitution step
constexpr int VB_MAXW = 64;
constexpr int VB_FACTOR = VB_NT / 32 - 1;  // the warp that factors the diagonal tiles

// the two block-column widths a launch can use per matrix
struct VbWidths { static constexpr int w0 = 32, w1 = 64; };

template <class T>
__device__ __forceinline__ T wshfl(T v, int src)
{
    return __shfl_sync(0xffffffffu, v, src);
}

// d += a b, fragments as in panel.cu
__device__ __forceinline__ void vb_mma(double (&d)[4], double a_up, double a_lo, double b)
{
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a_up), "d"(a_lo), "d"(b));
}

// Shared memory: two stages of [KC][rows + pad] slices of the round's rows (A) and of the
// block column's rows (B), the block's published X per 8-column step, the diagonal tiles'
// inverses, and per matrix the right-hand side and the reciprocal pivots.
template <class T, int NMAX>
struct VbSmem {
    // 4 (FP64) / 8 (FP32) words past a multiple of 128: fragment reads of four lines fall in
    // different banks, and a shifted line (vb_copy) fits
    static constexpr int LDA = VB_ROWS + (sizeof(T) == 8 ? 4 : 8), LDB = VB_MAXW + (sizeof(T) == 8 ? 4 : 8);
    static constexpr size_t stage = (size_t)VB_KC * (LDA + LDB) * sizeof(T);
    static constexpr size_t xs = (size_t)(VB_MAXW / 8) * VB_MAXW * 8 * sizeof(double);
    static constexpr size_t inv = (size_t)(VB_MAXW / 8) * 64 * sizeof(double);
    static constexpr size_t bytes = 2 * stage + xs + inv + (2 * NMAX + 128) * sizeof(double);
};

// Words by which column `line` of a slice starting at row `start` is shifted: 16-byte
// copies need 16-byte aligned sources, so a column whose first word is not aligned is
// copied from the boundary before it.  The shift depends on the column only modulo
// 16 / sizeof(T) <= 4, so a lane's fragments (columns k0 + kk + q, kk a multiple of 4)
// always find the same one.
template <class T>
__device__ __forceinline__ int vb_shift(const T* A, long long lda, long long line, int start)
{
    constexpr int E = 16 / sizeof(T);
    return (int)((reinterpret_cast<uintptr_t>(A) / sizeof(T) + (uintptr_t)(line * lda + start)) & (E - 1));
}
// KC columns from k0, rows [start, start + ROWS) below n (the rest zero): line l at dst + l * ld,
// shifted.  Rows before `start` may be copied along (start >= 32 whenever this is called).
template <class T, int ROWS>
__device__ __forceinline__ void vb_copy(T* dst, int ld, const T* __restrict__ A, long long lda, int k0, int start, int n)
{
    constexpr int E = 16 / sizeof(T);
    constexpr int units = ROWS / E + 1;
    for (int x = threadIdx.x; x < VB_KC * units; x += VB_NT) {
        const int l = x / units, u = x - l * units;
        const int sh = vb_shift(A, lda, k0 + l, start);
        const int w = start - sh + E * u;
        const int left = n - w, bytes = (left < 0 ? 0 : left > E ? E : left) * (int)sizeof(T);
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + l * ld + E * u);
        const T* src = bytes ? A + w + (long long)(k0 + l) * lda
                             : reinterpret_cast<const T*>(reinterpret_cast<uintptr_t>(A) & ~uintptr_t(15));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    }
}

template <class T, int NMAX, int W>
__device__ void vb_matrix(int n, T* __restrict__ A, long long lda, T* __restrict__ b, double* logdet_out,
                          int* info_out, unsigned char* smem, int* s_flag, double* s_red)
{
    using S = VbSmem<T, NMAX>;
    constexpr int RT = W / 8, DW = W / 16;  // tiles of a strip, strips (warps) of the diagonal block
    static_assert(W % VB_KC == 0 && W <= VB_MAXW && VB_ROWS == 16 * (VB_NT / 32), "block shape");
    double* Xs = reinterpret_cast<double*>(smem + 2 * S::stage);
    double* Inv = Xs + S::xs / sizeof(double);
    double* T8 = Inv + S::inv / sizeof(double);
    double* Lt = T8 + 64;
    double* bs = Lt + 64;
    double* rinv = bs + NMAX;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, q = lane & 3;
    const bool solve = b != nullptr;
    const int nrow = n + (solve ? 1 : 0);  // row n: the right-hand side
    if (solve)
        for (int i = t; i < n; i += VB_NT) bs[i] = (double)b[i];
    if (t == 0) s_flag[0] = 0;
    __syncthreads();
    int info = 0;

    for (int J = 0; J < n; J += W) {
        const int nw = min(W, n - J), steps = (nw + 7) >> 3;
        // round 0: the diagonal block's rows; then the rows below, 128 at a time
        for (int row0 = J; row0 < nrow; row0 += row0 == J ? W : VB_ROWS) {
            const int r_up = row0 + 16 * warp + g, r_lo = r_up + 8;
            const bool first = row0 == J;
            const int rows = first ? W : VB_ROWS;
            const bool active = 16 * warp < rows && row0 + 16 * warp < nrow;  // uniform over the warp
            const bool has_rhs = solve && n >= row0 && n < row0 + rows;
            double C[RT][4];
            // unconditional loads (of A(0, 0) where there is nothing to load), so that all are in flight
            // at once: as branches they took their latencies one after the other
#pragma unroll
            for (int l = 0; l < RT; ++l)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int r = h ? r_lo : r_up, c = J + 8 * l + 2 * q + e;
                        const bool in = active && r < n && c <= r;
                        const double v = (double)A[in ? r + (long long)c * lda : 0];
                        C[l][2 * h + e] = in ? v : 0.0;
                    }
            if (has_rhs && (n - row0) >> 4 == warp) {  // this strip holds row n
#pragma unroll
                for (int l = 0; l < RT; ++l)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int r = h ? r_lo : r_up, c = J + 8 * l + 2 * q + e;
                            if (r == n && c < n) C[l][2 * h + e] = bs[c];
                        }
            }
            // C -= L(rows, 0:J) L(J:J+W, 0:J)^T
            const int nch = J / VB_KC;
            auto stage = [&](int ch) {
                T* st = reinterpret_cast<T*>(smem + (ch & 1) * S::stage);
                if (first) vb_copy<T, W>(st, S::LDA, A, lda, ch * VB_KC, row0, n);
                else vb_copy<T, VB_ROWS>(st, S::LDA, A, lda, ch * VB_KC, row0, n);
                if (!first) vb_copy<T, W>(st + VB_KC * S::LDA, S::LDB, A, lda, ch * VB_KC, J, n);
            };
            if (nch > 0) stage(0);
            cp_group_commit();
            const int sha = vb_shift(A, lda, q, row0), shb = vb_shift(A, lda, q, J);
            const int ldb = first ? S::LDA : S::LDB;
            for (int ch = 0; ch < nch; ++ch) {
                if (ch + 1 < nch) stage(ch + 1);
                cp_group_commit();
                cp_group_wait<1>();
                __syncthreads();
                T* st = reinterpret_cast<T*>(smem + (ch & 1) * S::stage);
                if (has_rhs) {  // row n of the slice: the solved part of the right-hand side
                    if (t < VB_KC)
                        st[t * S::LDA + n - row0 + vb_shift(A, lda, t, row0)] = (T)bs[ch * VB_KC + t];
                    __syncthreads();
                }
                if (active) {
                    const T* as = st + q * S::LDA + 16 * warp + g + sha;
                    const T* bp = (first ? st : st + VB_KC * S::LDA) + q * ldb + g + shb;
#pragma unroll
                    for (int kk = 0; kk < VB_KC; kk += 4) {
                        const double a_up = -(double)as[kk * S::LDA], a_lo = -(double)as[kk * S::LDA + 8];
#pragma unroll
                        for (int l = 0; l < RT; ++l) vb_mma(C[l], a_up, a_lo, (double)bp[kk * ldb + 8 * l]);
                    }
                }
                __syncthreads();
            }
            cp_group_wait<0>();

            // one step of a strip: X = C_0 Inv^T, its columns before `good` stored; then the update
            auto solve_step = [&](int j, auto odd, double (&X)[4]) {
                const double2 v = *reinterpret_cast<const double2*>(&Inv[j * 64 + g * 8 + 2 * q]);
                X[0] = X[1] = X[2] = X[3] = 0.0;
                vb_mma(X, C[0][0], C[0][2], v.x);
                vb_mma(X, C[0][1], C[0][3], v.y);
                if (odd) {
                    const double2 u = tri_row(C[0][0], C[0][1], Inv + j * 64, 1, 8, true, lane);
                    const double2 l = tri_row(C[0][2], C[0][3], Inv + j * 64, 1, 8, true, lane);
                    X[0] = u.x, X[1] = u.y, X[2] = l.x, X[3] = l.y;
                }
            };
            auto store = [&](int j, const double (&X)[4], int rmin, int good) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int r = h ? r_lo : r_up, c = 2 * q + e;
                        if (r >= rmin && c < good) {
                            if (r < n) A[r + (long long)(J + 8 * j + c) * lda] = (T)X[2 * h + e];
                            else if (r < nrow) bs[J + 8 * j + c] = X[2 * h + e];
                        }
                    }
            };
            auto update = [&](int j, int cnt, const double (&X)[4]) {
#pragma unroll
                for (int l = 1; l < RT; ++l) {
                    if (l > cnt) break;
                    const double2 v = *reinterpret_cast<const double2*>(&Xs[(j * W + 8 * (j + l) + g) * 8 + 2 * q]);
                    double D[4] = {C[l][0], C[l][1], C[l][2], C[l][3]};
                    vb_mma(D, -X[0], -X[2], v.x);
                    vb_mma(D, -X[1], -X[3], v.y);
#pragma unroll
                    for (int e = 0; e < 4; ++e) C[l - 1][e] = D[e];
                }
            };
            if (first) {
                if (warp == VB_FACTOR) {
#pragma unroll 1
                    for (int j = 0; j < steps; ++j) {
                        const int kv = min(8, nw - 8 * j);
                        asm volatile("bar.sync 1, 64;" ::: "memory");  // the tile is in T8
                        const int good = factor_tile8(T8, Inv + j * 64, Lt, rinv + J + 8 * j, kv, lane);
                        if (lane == 0 && good < kv) s_flag[0] = J + 8 * j + good + 1;
                        asm volatile("bar.sync 2, %0;" ::"n"(32 * (DW + 1)) : "memory");
                        // the tile itself (with the failed column's updated values) and, if row n
                        // crosses it, that part of the right-hand side
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const int r = (lane + 32 * x) >> 3, c = lane & 7, R = J + 8 * j + r;
                            if (c < kv && R < n && c <= r) A[R + (long long)(J + 8 * j + c) * lda] = (T)Lt[r * 8 + c];
                            else if (c < kv && R == n && solve) bs[J + 8 * j + c] = Lt[r * 8 + c];
                        }
                        if (good < kv) break;
                        __syncwarp();
                    }
                } else if (warp < DW) {
                    const bool odd = any_nonfinite(C);
#pragma unroll 1
                    for (int j = 0; j < steps; ++j) {
                        const int kv = min(8, nw - 8 * j);
                        if (warp == (j >> 1)) {
                            *reinterpret_cast<double2*>(&T8[g * 8 + 2 * q]) =
                                (j & 1) ? make_double2(C[0][2], C[0][3]) : make_double2(C[0][0], C[0][1]);
                            asm volatile("bar.arrive 1, 64;" ::: "memory");
                        }
                        asm volatile("bar.sync 2, %0;" ::"n"(32 * (DW + 1)) : "memory");
                        const int fl = s_flag[0];
                        double X[4];
                        solve_step(j, odd || fl != 0, X);
                        *reinterpret_cast<double2*>(&Xs[(j * W + r_up - J) * 8 + 2 * q]) = make_double2(X[0], X[1]);
                        *reinterpret_cast<double2*>(&Xs[(j * W + r_lo - J) * 8 + 2 * q]) = make_double2(X[2], X[3]);
                        asm volatile("bar.sync 4, %0;" ::"n"(32 * DW) : "memory");
                        if (!fl) update(j, 2 * warp + 1 - j, X);
                        store(j, X, J + 8 * (j + 1), fl ? fl - 1 - J - 8 * j : kv);
                        if (fl) break;
                    }
                }
                __syncthreads();  // the block, its inverses and the flag are published
                info = s_flag[0];
            } else if (active) {
                auto run = [&](auto odd) {
#pragma unroll 1
                    for (int j = 0; j < steps; ++j) {
                        const int good = info ? info - 1 - J - 8 * j : nw - 8 * j;  // final columns from here
                        if (good <= 0) break;
                        double X[4];
                        solve_step(j, odd, X);
                        store(j, X, 0, min(good, 8));
                        if (info && good < 8) break;
                        update(j, RT - 1 - j, X);
                    }
                };
                // (a failed pivot may have put NaN in its column of every row)
                run(info || any_nonfinite(C));
            }
        }
        __syncthreads();  // the block column is in A
        if (info) break;
    }

    if (info == 0) {
        double lsum = 0.0;
        for (int i = t; i < n; i += VB_NT) lsum -= log(rinv[i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if (lane == 0) s_red[warp] = lsum;
    }
    if (solve && info == 0) {
        // backward substitution L^T x = y, VB_BW rows per step from the bottom: every warp sums
        // four of the block's columns over the rows below (their loads together in flight) while
        // the block itself comes into shared memory, then one warp runs the block's chain
        double* st = T8;
        T* blk = reinterpret_cast<T*>(smem);  // [c][r], the slices' stages are free
        constexpr int CW = VB_BW / (VB_NT / 32), LDK = VB_BW + 1;
        for (int J = ((n - 1) / VB_BW) * VB_BW; J >= 0; J -= VB_BW) {
            const int nw = min(VB_BW, n - J);
            for (int x = t; x < VB_BW * VB_BW; x += VB_NT) {
                const int c = x / VB_BW, r = x % VB_BW;
                blk[c * LDK + r] = c < nw && r < nw && r >= c ? A[(J + r) + (long long)(J + c) * lda] : T(0);
            }
            double acc[CW];
#pragma unroll
            for (int c = 0; c < CW; ++c) acc[c] = 0.0;
            const T* col = A + (long long)(J + CW * warp) * lda;
            if (J + VB_BW < n)  // the columns are all there
#pragma unroll 4
                for (int i = J + VB_BW + lane; i < n; i += 32) {
                    const double xi = bs[i];
#pragma unroll
                    for (int c = 0; c < CW; ++c) acc[c] = fma((double)col[i + c * lda], xi, acc[c]);
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < CW; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < CW; ++c) st[CW * warp + c] = acc[c];
            __syncthreads();
            if (warp == 0) {
                double v = lane < nw ? bs[J + lane] - st[lane] : 0.0;
                const double ri = lane < nw ? rinv[J + lane] : 0.0;
#pragma unroll 8
                for (int j = VB_BW - 1; j >= 0; --j) {
                    if (lane == j) v *= ri;
                    const double xj = wshfl(v, j);
                    if (lane < j) v = fma(-(double)blk[lane * LDK + j], xj, v);
                }
                if (lane < nw) bs[J + lane] = v;
            }
            __syncthreads();
        }
        for (int i = t; i < n; i += VB_NT) b[i] = (T)bs[i];
    }
    __syncthreads();
    if (t == 0) {
        double ld = 0.0;
        for (int w = 0; w < VB_NT / 32; ++w) ld += s_red[w];
        *info_out = info;
        *logdet_out = info ? __longlong_as_double(0x7ff8000000000000LL) : 2.0 * ld;
    }
    __syncthreads();
}

template <class T, int NMAX>
__global__ void __launch_bounds__(VB_NT, 2)
    k_posv_vbatched(int batch, const int* __restrict__ d_n, T* const* __restrict__ d_A, const int* __restrict__ d_lda,
                    T* const* __restrict__ d_B, double* __restrict__ d_logdet, int* __restrict__ d_info,
                    const int* __restrict__ order, const unsigned char* __restrict__ wsel, int* counters)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_m;
    __shared__ int s_flag[2];
    __shared__ double s_red[VB_NT / 32];
    for (;;) {
        if (threadIdx.x == 0) s_m = atomicAdd(&counters[0], 1);
        __syncthreads();
        const int m = s_m;
        __syncthreads();
        if (m >= batch) break;
        const int id = order ? order[m] : m;
        const int n = d_n[id];
        if (n <= 0 || n > NMAX || d_lda[id] < n) {
            if (threadIdx.x == 0) {
                d_info[id] = n == 0 ? 0 : -1;
                d_logdet[id] = n == 0 ? 0.0 : __longlong_as_double(0x7ff8000000000000LL);
            }
            continue;
        }
        T* A = d_A[id];
        T* B = d_B ? d_B[id] : nullptr;
        const long long lda = d_lda[id];
        if (wsel && wsel[id])
            vb_matrix<T, NMAX, VbWidths::w1>(n, A, lda, B, d_logdet + id, d_info + id, smem_raw, s_flag, s_red);
        else
            vb_matrix<T, NMAX, VbWidths::w0>(n, A, lda, B, d_logdet + id, d_info + id, smem_raw, s_flag, s_red);
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&counters[1], 1) == (int)gridDim.x - 1) {
            atomicExch(&counters[0], 0);
            atomicExch(&counters[1], 0);
            __threadfence();
        }
    }
}

// A well-conditioned SPD stand-in for the autotuner: n on the diagonal,
// 1/(1+|i-j|) off it (diagonally dominant for n >= 16).
template <class T>
__global__ void k_fill_spd(int batch, const int* __restrict__ d_n, T* const* __restrict__ d_A,
                           const int* __restrict__ d_lda, T* const* __restrict__ d_B)
{
    const int id = blockIdx.x;
    if (id >= batch) return;
    const int n = d_n[id];
    const long long lda = d_lda[id];
    T* A = d_A[id];
    for (long long e = threadIdx.x; e < (long long)n * n; e += blockDim.x) {
        const int i = (int)(e % n), j = (int)(e / n);
        A[i + j * lda] = i == j ? T(n) : T(1) / T(1 + abs(i - j));
    }
    if (d_B && d_B[id])
        for (int i = threadIdx.x; i < n; i += blockDim.x) d_B[id][i] = T(1);
}

template <class T, int NMAX>
cudaError_t vb_launch(int batch, const int* d_n, void* const* d_A, const int* d_lda, void* const* d_B,
                      double* d_logdet, int* d_info, const int* order, const unsigned char* wsel, int* counters,
                      int grid, cudaStream_t st)
{
    constexpr size_t smem = VbSmem<T, NMAX>::bytes;
    if (cudaError_t e = smem_optin(k_posv_vbatched<T, NMAX>, smem); e != cudaSuccess) return e;
    k_posv_vbatched<T, NMAX><<<grid, VB_NT, smem, st>>>(batch, d_n, reinterpret_cast<T* const*>(d_A), d_lda,
                                                        reinterpret_cast<T* const*>(d_B), d_logdet, d_info, order,
                                                        wsel, counters);
    note_launches(1);
    return cudaGetLastError();
}

template <class T, int NMAX>
int vb_max_grid()
{
    constexpr size_t smem = VbSmem<T, NMAX>::bytes;
    if (smem_optin(k_posv_vbatched<T, NMAX>, smem) != cudaSuccess) return 0;
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_posv_vbatched<T, NMAX>, VB_NT, smem) != cudaSuccess)
        return 0;
    return sms * per;
}

}  // namespace
}  // namespace ddlak

extern "C" int ddlak_vbatched_variants(char type, int nmax, int* widths)
{
    if (nmax != 512 && nmax != 1024) return (int)cudaErrorInvalidValue;
    using namespace ddlak;
    if (type != 'd' && type != 's') return (int)cudaErrorInvalidValue;
    widths[0] = VbWidths::w0;
    widths[1] = VbWidths::w1;
    return 0;
}

extern "C" int ddlak_vbatched_max_grid(char type, int nmax)
{
    using namespace ddlak;
    if (type == 'd') return nmax == 512 ? vb_max_grid<double, 512>() : nmax == 1024 ? vb_max_grid<double, 1024>() : 0;
    if (type == 's') return nmax == 512 ? vb_max_grid<float, 512>() : nmax == 1024 ? vb_max_grid<float, 1024>() : 0;
    return 0;
}

extern "C" int ddlak_posv_vbatched(char type, int nmax, int batch, const int* d_n, void* const* d_A,
                                   const int* d_lda, void* const* d_B, double* d_logdet, int* d_info,
                                   const int* d_order, const unsigned char* d_wsel, int* d_counters, int grid,
                                   void* stream)
{
    using namespace ddlak;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (batch <= 0) return 0;
    if (grid <= 0 || !d_n || !d_A || !d_lda || !d_logdet || !d_info || !d_counters) return (int)cudaErrorInvalidValue;
    ProfScope ps(PK_BATCHED, st, 0.0, 0.0);
    if (type == 'd') {
        if (nmax == 512)
            return (int)vb_launch<double, 512>(batch, d_n, d_A, d_lda, d_B, d_logdet, d_info, d_order, d_wsel,
                                               d_counters, grid, st);
        if (nmax == 1024)
            return (int)vb_launch<double, 1024>(batch, d_n, d_A, d_lda, d_B, d_logdet, d_info, d_order, d_wsel,
                                                d_counters, grid, st);
    } else if (type == 's') {
        if (nmax == 512)
            return (int)vb_launch<float, 512>(batch, d_n, d_A, d_lda, d_B, d_logdet, d_info, d_order, d_wsel,
                                              d_counters, grid, st);
        if (nmax == 1024)
            return (int)vb_launch<float, 1024>(batch, d_n, d_A, d_lda, d_B, d_logdet, d_info, d_order, d_wsel,
                                               d_counters, grid, st);
    }
    return (int)cudaErrorInvalidValue;
}

extern "C" int ddlak_fill_spd_vbatched(char type, int batch, const int* d_n, void* const* d_A, const int* d_lda,
                                       void* const* d_B, void* stream)
{
    using namespace ddlak;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (batch <= 0) return 0;
    if (type == 'd')
        k_fill_spd<double><<<batch, 256, 0, st>>>(batch, d_n, reinterpret_cast<double* const*>(d_A), d_lda,
                                                  reinterpret_cast<double* const*>(d_B));
    else if (type == 's')
        k_fill_spd<float><<<batch, 256, 0, st>>>(batch, d_n, reinterpret_cast<float* const*>(d_A), d_lda,
                                                 reinterpret_cast<float* const*>(d_B));
    else
        return (int)cudaErrorInvalidValue;
    note_launches(1);
    return (int)cudaGetLastError();
}
