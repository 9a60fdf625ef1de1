// Fused forward + backward substitution with a Cholesky factor (ddla::ppotrs on
// a 1x1 grid).
//
// The reference applies two vendor triangular solves, L then L^H
// (src/Cholesky/ppotrs.cpp:44-61 -> src/PBLAS/ptrtrs.cpp:150-155 ->
// src/BLAS/trsm.cpp:154-159, cublas?trsm).  Here both solves are ONE launch:
// the solution is split into block rows of RB rows and every CTA takes a
// ticket from a global counter.  Tickets 0..N-1 solve the forward block rows
// 0..N-1 (L Y = B), tickets N..2N-1 the backward block rows N-1..0
// (L^H X = Y).  A CTA only ever waits for a block row published under a
// smaller ticket, and every smaller ticket belongs to a CTA that has already
// started, so the waits always end; each wait is additionally bounded by a
// clock budget and reports DDLAK_WAIT_TIMEOUT instead of spinning forever.
//
// Each CTA streams the off-diagonal tiles of its block row through a
// double-buffered cp.async ring (the tile loads do not depend on other CTAs,
// only the solved blocks do), visiting them in publication order, then solves
// its diagonal block: the real types on the FP64 tensor cores by substitution over
// 8 x 8 tiles (k_potrs_dmma), the complex types with one warp per pair of
// right-hand sides using reciprocal pivots and warp shuffles (k_potrs_fused).
//
// The right-hand sides are a view X(i, r): B[i + r*ldb] for side 'L' and
// conj(B[r + i*ldb]) for side 'R' (X * A = B  <=>  A * X^H = B^H, since A is
// Hermitian).  They are processed in chunks of RC columns; chunk c uses its own
// flag row and tickets interleave chunks so the ordering argument holds per
// chunk.
#include <mutex>

#include <ddla_kernels.h>

#include "common.cuh"
#include "ddla_kernels_internal.h"
#include "profile.h"
#include "tile8.cuh"

namespace ddlak {

namespace {

constexpr int RB = 64;   // rows per block row
constexpr int RC = 16;   // right-hand sides per chunk
constexpr int NT = 256;  // threads per CTA

template <class T, bool BT>
__device__ __forceinline__ T x_ld_cg(const T* B, long long ldb, long long i, long long r)
{
    const T* p = BT ? B + r + i * ldb : B + i + r * ldb;
    T v;
    if constexpr (sizeof(T) == 4) { float t = __ldcg(reinterpret_cast<const float*>(p)); v = *reinterpret_cast<T*>(&t); }
    else if constexpr (sizeof(T) == 8) { double t = __ldcg(reinterpret_cast<const double*>(p)); v = *reinterpret_cast<T*>(&t); }
    else { double2 t = __ldcg(reinterpret_cast<const double2*>(p)); v = *reinterpret_cast<T*>(&t); }
    return BT ? cj(v) : v;
}
template <class T, bool BT>
__device__ __forceinline__ void x_st(T* B, long long ldb, long long i, long long r, T v)
{
    if (BT) B[r + i * ldb] = cj(v);
    else B[i + r * ldb] = v;
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <class T>
__device__ __forceinline__ T shfl_t(T v, int src)
{
    if constexpr (Traits<T>::cplx) {
        v.x = __shfl_sync(0xffffffffu, v.x, src);
        v.y = __shfl_sync(0xffffffffu, v.y, src);
        return v;
    } else {
        return __shfl_sync(0xffffffffu, v, src);
    }
}

// Shared-memory layout (elements of T unless noted):
//   Lbuf[2][RB][RB+1]  raw off-diagonal tiles, Lbuf[b][k][i]
//   Xs[RB][RC+1]       the solved block of the other block row
//   Acc[RB][RC+1]      this block row's right-hand sides
//   Rinv[RB]           reciprocal pivots (real type)
template <class T>
__host__ __device__ constexpr size_t potrs_smem_bytes()
{
    return sizeof(T) * (2 * (size_t)RB * (RB + 1) + 2 * (size_t)RB * (RC + 1)) + sizeof(real_t<T>) * RB;
}

// Complex types.  FO: forward substitution only, on B: X = L^-1 B (side 'L') or B L^-H
// (side 'R'); the forward half of the two-sided solve, every CTA a forward one.
template <class T, bool UP, bool BT, bool FO = false>
__global__ void __launch_bounds__(NT) k_potrs_fused(const T* __restrict__ A, long long lda, T* B, long long ldb,
                                                    int n, int nrhs, int nchunks, int* flags, int* ticket,
                                                    int* status, const int* __restrict__ skip)
{
    if (skip != nullptr && *skip != 0) return;
    using TL = T;
    using R = real_t<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TL (*Lbuf)[RB][RB + 1] = reinterpret_cast<TL (*)[RB][RB + 1]>(smem_raw);
    T (*Xs)[RC + 1] = reinterpret_cast<T (*)[RC + 1]>(smem_raw + sizeof(TL) * 2 * RB * (RB + 1));
    T (*Acc)[RC + 1] = Xs + RB;
    R* Rinv = reinterpret_cast<R*>(Acc + RB);
    __shared__ int s_t;
    __shared__ int s_abort;
    __shared__ int s_next;
    if (threadIdx.x == 0) { s_t = atomicAdd(ticket, 1); s_abort = 0; }
    __syncthreads();
    const int N = (int)ceil_div(n, RB);
    const int t = s_t;
    const int chunk = t % nchunks;
    const int step = t / nchunks;
    const bool fwd = FO || step < N;
    const int blk = fwd ? step : 2 * N - 1 - step;
    int* cflags = flags + (size_t)chunk * 2 * N;  // [0,N) forward, [N,2N) backward
    const long long r0 = (long long)chunk * RC;
    const int nr = (int)((nrhs - r0) < RC ? (nrhs - r0) : RC);
    const long long i0 = (long long)blk * RB;
    const int nrows = (int)((n - i0) < RB ? (n - i0) : RB);
    // raw tile element (i, k): A[(i0+i) + (j0+k)*lda] when p1, A[(j0+k) + (i0+i)*lda] otherwise;
    // the operator entry is that value, conjugated when !p1 (see the four cases of the L view)
    const bool p1 = (fwd != UP);

    const int tr = threadIdx.x & (RB - 1);  // row of the block row
    const int tg = threadIdx.x >> 6;        // rhs group: columns tg, tg+4, tg+8, tg+12
    T acc[RC / 4];

    // Visit the other block rows in publication order (forward 0, 1, ..; backward N-1, N-2, ..):
    // every wait but the last one is already satisfied when reached.
    const int nvisit = fwd ? blk : N - 1 - blk;
    auto visit = [&](int v) { return fwd ? v : N - 1 - v; };
    auto issue_tile = [&](int j, int buf) {
        const long long j0 = (long long)j * RB;
        const int ncols = (int)((n - j0) < RB ? (n - j0) : RB);
        for (int idx = threadIdx.x; idx < RB * RB; idx += NT) {
            int i, k;
            const TL* src;
            if (p1) { i = idx % RB; k = idx / RB; src = A + (i0 + i) + (j0 + k) * lda; }
            else { k = idx % RB; i = idx / RB; src = A + (j0 + k) + (i0 + i) * lda; }
            const bool valid = i < nrows && k < ncols;
            cp_async_elem<sizeof(TL)>(&Lbuf[buf][k][i], valid ? src : A, valid);
        }
    };
    // the diagonal block, raw: D[c][r] = A[(i0+r) + (i0+c)*lda] for 'L', A[(i0+c) + (i0+r)*lda] for 'U';
    // L(r, c) = D[c][r] ('L') or conj(D[c][r]) ('U') for r >= c.  Prefetched into the ring slot
    // the last off-diagonal tile leaves free, so it is resident when the solve reaches it.
    auto issue_diag = [&](int buf) {
        for (int idx = threadIdx.x; idx < RB * RB; idx += NT) {
            int r, c;
            const TL* src;
            if (!UP) { r = idx % RB; c = idx / RB; src = A + (i0 + r) + (i0 + c) * lda; }
            else { c = idx % RB; r = idx / RB; src = A + (i0 + c) + (i0 + r) * lda; }
            const bool valid = r < nrows && c < nrows;
            cp_async_elem<sizeof(TL)>(&Lbuf[buf][c][r], valid ? src : A, valid);
        }
    };
    if (nvisit > 0) issue_tile(visit(0), 0);
    else issue_diag(0);
    cp_commit();

    if (!fwd) {
        // the block row's own forward result must be published first
        if (threadIdx.x == 0) {
            if (!bounded_wait_geq(&cflags[blk], 1, status)) s_abort = 1;
            __threadfence();
        }
        __syncthreads();
        if (s_abort) { cp_wait<0>(); return; }
    }
#pragma unroll
    for (int q = 0; q < RC / 4; ++q) {
        const int r = tg + 4 * q;
        acc[q] = (tr < nrows && r < nr) ? x_ld_cg<T, BT>(B, ldb, i0 + tr, r0 + r) : zero<T>();
    }

    // The solved block of the next visit is fetched into registers (L2 loads) while
    // the current tile is multiplied whenever its flag is already set, so only the
    // visits that really wait (the last ones) pay the load latency after the wait.
    constexpr int XE = RB * RC / NT;
    T xr[XE];
    bool pre = false;
    auto load_x = [&](int jj) {
        const long long jj0 = (long long)jj * RB;
        const int nc = (int)((n - jj0) < RB ? (n - jj0) : RB);
#pragma unroll
        for (int e = 0; e < XE; ++e) {
            const int idx = threadIdx.x + e * NT;
            const int k = idx % RB, r = idx / RB;
            xr[e] = (k < nc && r < nr) ? x_ld_cg<T, BT>(B, ldb, jj0 + k, r0 + r) : zero<T>();
        }
    };
    for (int v = 0; v < nvisit; ++v) {
        const int j = visit(v);
        if (v + 1 < nvisit) issue_tile(visit(v + 1), (v + 1) & 1);
        else issue_diag((v + 1) & 1);
        cp_commit();
        if (!pre) {
            if (threadIdx.x == 0) {
                if (!bounded_wait_geq(&cflags[fwd ? j : N + j], 1, status)) s_abort = 1;
                __threadfence();
            }
            __syncthreads();
            if (s_abort) { cp_wait<0>(); return; }
            load_x(j);
        }
#pragma unroll
        for (int e = 0; e < XE; ++e) {
            const int idx = threadIdx.x + e * NT;
            Xs[idx % RB][idx / RB] = xr[e];
        }
        if (threadIdx.x == 0) {
            bool ready = false;
            if (v + 1 < nvisit) {
                const int jn = visit(v + 1);
                ready = ld_acquire(&cflags[fwd ? jn : N + jn]) >= 1;
                if (ready) __threadfence();
            }
            s_next = ready ? 1 : 0;
        }
        cp_wait<1>();
        __syncthreads();
        pre = s_next != 0;
        if (pre) load_x(visit(v + 1));
        const TL (*Lt)[RB + 1] = Lbuf[v & 1];
        if (p1) {
#pragma unroll 8
            for (int k = 0; k < RB; ++k) {
                const T l = Lt[k][tr];
#pragma unroll
                for (int q = 0; q < RC / 4; ++q) acc[q] = fms(acc[q], l, Xs[k][tg + 4 * q]);
            }
        } else {
#pragma unroll 8
            for (int k = 0; k < RB; ++k) {
                const T l = cj(Lt[k][tr]);
#pragma unroll
                for (int q = 0; q < RC / 4; ++q) acc[q] = fms(acc[q], l, Xs[k][tg + 4 * q]);
            }
        }
        __syncthreads();
    }
    cp_wait<0>();

    const TL (*D)[RB + 1] = Lbuf[nvisit & 1];
    // L(r, c) for r >= c, and conj(L(c, r)) for c > r, from the raw diagonal block
    auto lval = [&](int r, int c) { return UP ? cj(D[c][r]) : D[c][r]; };
    auto lcval = [&](int c, int r) { return UP ? D[r][c] : cj(D[r][c]); };
#pragma unroll
    for (int q = 0; q < RC / 4; ++q) Acc[tr][tg + 4 * q] = acc[q];
    __syncthreads();
    for (int k = threadIdx.x; k < RB; k += NT) Rinv[k] = k < nrows ? R(1) / re(D[k][k]) : R(0);
    __syncthreads();
    {
        // warp w solves right-hand sides 2w and 2w+1 together; lanes own rows lane and lane+32
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int ra = 2 * warp, rb = 2 * warp + 1;
        T a0 = Acc[lane][ra], a1 = Acc[lane + 32][ra];
        T b0 = Acc[lane][rb], b1 = Acc[lane + 32][rb];
        if (fwd) {
            for (int k = 0; k < nrows; ++k) {
                const R rk = Rinv[k];
                if (k < 32) {
                    if (lane == k) { a0 = scal(a0, rk); b0 = scal(b0, rk); }
                    const T xa = shfl_t(a0, k), xb = shfl_t(b0, k);
                    const T l0 = lval(lane, k), l1 = lval(lane + 32, k);
                    if (lane > k) { a0 = fms(a0, l0, xa); b0 = fms(b0, l0, xb); }
                    a1 = fms(a1, l1, xa);
                    b1 = fms(b1, l1, xb);
                } else {
                    if (lane == k - 32) { a1 = scal(a1, rk); b1 = scal(b1, rk); }
                    const T xa = shfl_t(a1, k - 32), xb = shfl_t(b1, k - 32);
                    if (lane + 32 > k) {
                        const T l1 = lval(lane + 32, k);
                        a1 = fms(a1, l1, xa);
                        b1 = fms(b1, l1, xb);
                    }
                }
            }
        } else {
            // x_k = v_k / L_kk; v_i -= conj(L(k, i)) x_k for i < k
            for (int k = nrows - 1; k >= 0; --k) {
                const R rk = Rinv[k];
                if (k < 32) {
                    if (lane == k) { a0 = scal(a0, rk); b0 = scal(b0, rk); }
                    const T xa = shfl_t(a0, k), xb = shfl_t(b0, k);
                    if (lane < k) {
                        const T l0 = lcval(k, lane);
                        a0 = fms(a0, l0, xa);
                        b0 = fms(b0, l0, xb);
                    }
                } else {
                    if (lane == k - 32) { a1 = scal(a1, rk); b1 = scal(b1, rk); }
                    const T xa = shfl_t(a1, k - 32), xb = shfl_t(b1, k - 32);
                    const T l0 = lcval(k, lane);
                    a0 = fms(a0, l0, xa);
                    b0 = fms(b0, l0, xb);
                    if (lane + 32 < k) {
                        const T l1 = lcval(k, lane + 32);
                        a1 = fms(a1, l1, xa);
                        b1 = fms(b1, l1, xb);
                    }
                }
            }
        }
        Acc[lane][ra] = a0;
        Acc[lane + 32][ra] = a1;
        Acc[lane][rb] = b0;
        Acc[lane + 32][rb] = b1;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < RB * RC; idx += NT) {
        const int i = idx % RB, r = idx / RB;
        if (i < nrows && r < nr) x_st<T, BT>(B, ldb, i0 + i, r0 + r, Acc[i][r]);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) st_release(&cflags[fwd ? blk : N + blk], 1);
}

// ---------------------------------------------------------------------------
// The same solve for real types on the FP64 tensor cores (DMMA, FP64 arithmetic for FP32
// and FP64 storage).  Eight warps.  The off-diagonal tiles: warp w owns rows
// 16 (w % 4) .. + 15 of the block row and right-hand sides 8 (w / 4) .. + 7 of the
// chunk, as one accumulator fragment.
//   * The diagonal block is solved by substitution over 8 x 8 tiles, as the panel solve of
//     panel.cu: only the 8 x 8 tiles on the diagonal are inverted (before the CTA joins the
//     chain).  The transpose is kept (rows are right-hand sides), so that a step's
//     result is the next product's operand without a shuffle: warp w owns rows
//     16 (w / 2) .. + 15 for right-hand sides 8 (w % 2) .. + 7 and hands its solution to the
//     other three warps of its right-hand sides through shared memory.  The inverse
//     of the whole 64 x 64 block in place of this is not backward stable: for
//     a squared-exponential kernel on a line, condition 1e14, n = 256, the backward error
//     is 1e-12 with 64-row inverses, 1e-15 with 16-row ones and 4e-17 with 8-row
//     ones, as by substitution (restated in numpy).
//   * One thread polls the flag of the block needed; behind it a warp looks how many of the
//     next 32 blocks are up too, so that blocks known to be up cost no look and no fence.
//     A block's solution goes through shared memory, four entries a thread, fetched under
//     the product before it when its flag is up.  (With a look per block, and the solution
//     read by each of the four warps that need it in 16 loads a thread, n = 5003 with as many
//     right-hand sides took 47.7 ms, 18.4 now.)
// What bounds it: with few right-hand sides the chain of n / 64 links per direction; with many
// the latency of a visit (tile, solution, product, two barriers), two CTAs per SM over it.
// Measured (one call, factor and flags in place) against the substitution form by warps, FP64:
// n = 2048, 16 right-hand sides 256 against 556 us, 2048 of them 1.26 against 2.42 ms;
// n = 5003, 16 of them 0.65 against 1.41 ms, 5003 of them 18.4 against 32.8 ms; n = 8192,
// 64 of them 1.10 against 2.57 ms.  FP32: n = 5003, 16 of them 0.61 against 1.11 ms, 5003 of
// them 16.5 against 24.2 ms.
// ---------------------------------------------------------------------------
constexpr int PD_LD = RB + 4;  // 4 mod 16 doubles: conflict-free fragment reads either way round
constexpr int PD_LDX = RC + 4;
constexpr int PD_LDV = RB + 4;

constexpr int PD_XT = RB / 8 * 64;  // doubles of one half's published solution: 8 tiles, 2 a lane

// two tiles of the ring (the block row's right-hand sides and the published solution of the
// diagonal step take their place afterwards), the diagonal block in FP64, another block
// row's solution
template <class TL>
__host__ __device__ constexpr size_t potrs_dmma_smem()
{
    static_assert(2 * RB * PD_LD * sizeof(TL) >= (RB * PD_LDX + 2 * PD_XT) * sizeof(double), "diagonal step");
    return 2 * (size_t)RB * PD_LD * sizeof(TL) + (size_t)(RB * PD_LD + RC * PD_LDV) * sizeof(double);
}

__device__ __forceinline__ void pd_mma(double (&d)[4], double a_up, double a_lo, double b)
{
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a_up), "d"(a_lo), "d"(b));
}

// d += a b with m8n8k4: lane (g = lane / 4, q = lane % 4) supplies A(g, q) and B(q, g) and holds
// D(g, 2q), D(g, 2q + 1); these two are the A operands of a next product over k in the
// order {0, 2, 4, 6}, {1, 3, 5, 7}.
__device__ __forceinline__ void pd_mma8(double (&d)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// One thread: until *flag >= 1 or the budget runs out (DDLAK_WAIT_TIMEOUT in *status, false).
// Relaxed polls and one fence: an acquire per poll would invalidate L1 each time.
__device__ __forceinline__ bool poll_flag(const int* flag, int* status, bool near)
{
    const long long t0 = clock64(), budget = wait_budget_cycles();
    for (unsigned it = 0;; ++it) {
        if (ld_relaxed(flag) >= 1) {
            __threadfence();
            return true;
        }
        if ((it & 31) == 31) {
            if (ld_relaxed(status) != DDLAK_OK) return false;
            if (clock64() - t0 > budget) {
                atomicCAS(status, DDLAK_OK, DDLAK_WAIT_TIMEOUT);
                return false;
            }
        }
        if (!near) __nanosleep(200);
    }
}

template <class TL, class TX, bool UP, bool BT, bool ID, bool FO>
__global__ void __launch_bounds__(NT, 2) k_potrs_dmma(const TL* __restrict__ A, long long lda, TX* B, long long ldb,
                                                      int n, int nrhs, int nchunks, int* flags, int* ticket,
                                                      int* status, const int* __restrict__ skip)
{
    if (skip != nullptr && *skip != 0) return;  // the factorization before it failed: B stays
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TL* Lb = reinterpret_cast<TL*>(smem_raw);  // two tiles of RB lines of PD_LD
    double* Db = reinterpret_cast<double*>(smem_raw + 2 * (size_t)RB * PD_LD * sizeof(TL));  // the diagonal block
    double* Xs = reinterpret_cast<double*>(smem_raw);  // the block row's right-hand sides, over the (then free) tiles
    double* Xt = Xs + RB * PD_LDX;                     // and the diagonal step's solution, a tile's fragment at a time
    double* Xv = Db + RB * PD_LD;                      // the other block row's solution, negated: [r][k]
    __shared__ int s_t, s_ready;
    if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
    __syncthreads();
    const int N = (int)ceil_div(n, RB);
    const int t = s_t;
    const int chunk = t % nchunks;
    const int step = t / nchunks;
    const bool fwd = ID || FO || step < N;
    const int blk = ID ? step : (fwd ? step : 2 * N - 1 - step);
    int* cflags = flags + (size_t)chunk * 2 * N;  // [0,N) forward, [N,2N) backward
    const long long r0 = (long long)chunk * RC;
    const int jfirst = ID ? (int)(r0 / RB) : 0;  // first block row with a nonzero right-hand side
    if (ID && blk < jfirst) return;
    const long long i0 = (long long)blk * RB;
    const int nrows = (int)((n - i0) < RB ? (n - i0) : RB);
    // operator entry (i, k) of a tile: A[(i0+i) + (j0+k)*lda] when p1, A[(j0+k) + (i0+i)*lda] otherwise
    const bool p1 = (fwd != UP);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int row = 16 * (warp & 3) + g;              // and row + 8
    const long long rc = r0 + 8 * (warp >> 2);         // this warp's first right-hand side
    const bool live = rc < nrhs;                       // uniform over the warp

    const int nvisit = ID ? blk - jfirst : (fwd ? blk : N - 1 - blk);
    auto visit = [&](int v) { return ID ? jfirst + v : (fwd ? v : N - 1 - v); };
    // tile lines: p1 [k][i], otherwise [i][k]; the line's words are contiguous in A
    auto issue_tile = [&](int j, int buf) {
        const long long j0 = (long long)j * RB;
        const int ncols = (int)((n - j0) < RB ? (n - j0) : RB);
        TL* dst = Lb + buf * RB * PD_LD;
        const TL* src0 = p1 ? A + i0 + j0 * lda : A + j0 + i0 * lda;
        const int wlim = p1 ? nrows : ncols, llim = p1 ? ncols : nrows;
        if (sizeof(TL) == 8 && !(lda & 1) && !(reinterpret_cast<uintptr_t>(A) & 15) && wlim == RB) {
            for (int idx = threadIdx.x; idx < RB * RB / 2; idx += NT) {
                const int l = idx >> 5, w = 2 * (idx & 31);
                const bool in = l < llim;
                cp_async_elem16(dst + l * PD_LD + w, in ? src0 + l * lda + w : A, in);
            }
        } else {
            for (int idx = threadIdx.x; idx < RB * RB; idx += NT) {
                const int l = idx >> 6, w = idx & (RB - 1);
                const bool in = l < llim && w < wlim;
                cp_async_elem<sizeof(TL)>(dst + l * PD_LD + w, in ? src0 + l * lda + w : A, in);
            }
        }
    };
    // the diagonal block: lines [c][r] ('L') or [r][c] ('U'), zero in its strict upper part and
    // past the matrix; FP32 storage by way of tile 0
    {
        const TL* src0 = A + i0 + i0 * lda;
        TL* dst = sizeof(TL) == 8 ? reinterpret_cast<TL*>(Db) : Lb;
        for (int idx = threadIdx.x; idx < RB * RB; idx += NT) {
            const int l = idx >> 6, w = idx & (RB - 1);
            const bool in = l < nrows && w < nrows && (UP ? w <= l : w >= l);
            cp_async_elem<sizeof(TL)>(dst + l * PD_LD + w, in ? src0 + l * lda + w : A, in);
        }
    }
    cp_commit();
    if (nvisit > 0) issue_tile(visit(0), 1);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    if constexpr (sizeof(TL) < 8) {
        for (int idx = threadIdx.x; idx < RB * RB; idx += NT) {
            const int l = idx >> 6, w = idx & (RB - 1);
            Db[l * PD_LD + w] = (double)Lb[l * PD_LD + w];
        }
        __syncthreads();
    }
    if (threadIdx.x < 64) {
        // column c of diagonal tile b's inverse, in the tile's place (rows past the matrix: the identity)
        const int b = threadIdx.x >> 3, c = threadIdx.x & 7;
        double* tile = Db + 8 * b * (PD_LD + 1);
        double y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            double v = i == c ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < i; ++k) v = fma(-tile[UP ? i * PD_LD + k : k * PD_LD + i], y[k], v);
            y[i] = 8 * b + i < nrows ? v / tile[i * (PD_LD + 1)] : v;
        }
        __syncwarp();  // a tile's eight threads are in one warp
#pragma unroll
        for (int i = 0; i < 8; ++i) tile[UP ? i * PD_LD + c : c * PD_LD + i] = y[i];
    }
    __syncthreads();

    // ---- the block row -------------------------------------------------------------------
    // one thread waits for a block's solution; the CTA learns of it at the next barrier.  A wait
    // that is not the block row's last polls rarely: hundreds of CTAs wait at a time, and
    // their polls of one word would delay the publication itself.
    bool fail = false;
    auto wait_flag = [&](const int* f, bool near) {
        if (threadIdx.x == 0) fail = !poll_flag(f, status, near);
        fail = __syncthreads_or(fail);
    };
    if (!fwd) wait_flag(&cflags[blk], nvisit == 0);  // the block row's own forward result
    if (fail) {
        cp_wait<0>();
        return;
    }
    double acc[4], acc2[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const long long i = i0 + row + 8 * h, r = rc + 2 * q + e;
            if (ID) {
                acc[2 * h + e] = i == r && i < n ? 1.0 : 0.0;
            } else {
                const bool in = row + 8 * h < nrows && r < nrhs;
                const double v = (double)x_ld_cg<TX, BT>(B, ldb, in ? i : 0, in ? r : 0);
                acc[2 * h + e] = in ? v : 0.0;
            }
        }
    // The other block's solution: four entries a thread (of B(0, 0) where there is nothing to
    // load: unconditional, so that the loads are in flight together), by way of shared memory
    double xv[4];
    auto xk = [](int i) { return BT ? (threadIdx.x + NT * i) / RC : (threadIdx.x + NT * i) % RB; };
    auto xr = [](int i) { return BT ? (threadIdx.x + NT * i) % RC : (threadIdx.x + NT * i) / RB; };
    auto load_x = [&](int j) {
        const long long j0 = (long long)j * RB;
#pragma unroll
        for (int i = 0; i < RB * RC / NT; ++i) {
            const long long k = j0 + xk(i), r = r0 + xr(i);
            const bool in = k < n && r < nrhs;
            const double v = (double)x_ld_cg<TX, BT>(B, ldb, in ? k : 0, in ? r : 0);
            xv[i] = in ? -v : 0.0;
        }
    };
    int ready = 0;  // visits whose solution is known to be published
    for (int v = 0; v < nvisit; ++v) {
        if (v + 1 < nvisit) issue_tile(visit(v + 1), v & 1);  // tile v sits in buffer (v + 1) & 1
        cp_commit();
        if (v >= ready) {
            const int j = visit(v);
            wait_flag(&cflags[fwd ? j : N + j], v + 1 == nvisit);
            if (fail) {
                cp_wait<0>();
                return;
            }
            load_x(j);
            ready = v + 1;
        }
#pragma unroll
        for (int i = 0; i < RB * RC / NT; ++i) Xv[xr(i) * PD_LDV + xk(i)] = xv[i];
        const bool look = v + 1 < nvisit && ready == v + 1;  // uniform over the CTA
        if (look && warp == 0) {
            // how many of the next 32 visits' solutions are up
            const int vn = v + 1 + lane;
            bool up = false;
            if (vn < nvisit) {
                const int j = visit(vn);
                up = ld_relaxed(&cflags[fwd ? j : N + j]) >= 1;
            }
            const unsigned m = __ballot_sync(0xffffffffu, up);
            if (m & 1) __threadfence();
            if (lane == 0) s_ready = v + 1 + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
        }
        cp_wait<1>();
        __syncthreads();
        if (look) ready = s_ready;
        if (v + 1 < ready) load_x(visit(v + 1));  // under the product
        if (live) {
            const TL* Lt = Lb + ((v + 1) & 1) * RB * PD_LD;
            const double* b = Xv + (8 * (warp >> 2) + g) * PD_LDV + q;
            if (p1) {
#pragma unroll
                for (int m = 0; m < RB / 4; m += 2) {
                    const TL* p = Lt + (4 * m + q) * PD_LD + row;
                    pd_mma(acc, (double)p[0], (double)p[8], b[4 * m]);
                    pd_mma(acc2, (double)p[4 * PD_LD], (double)p[4 * PD_LD + 8], b[4 * m + 4]);
                }
            } else {
#pragma unroll
                for (int m = 0; m < RB / 4; m += 2) {
                    const TL* p = Lt + row * PD_LD + 4 * m + q;
                    pd_mma(acc, (double)p[0], (double)p[8 * PD_LD], b[4 * m]);
                    pd_mma(acc2, (double)p[4], (double)p[8 * PD_LD + 4], b[4 * m + 4]);
                }
            }
        }
        __syncthreads();  // the tile and Xv are free
    }
    cp_wait<0>();

    // ---- the diagonal block: rows 16 w .. of right-hand sides 8 h .., transposed ------
    // forward x L^T = c through the tiles 0 .. 7, backward x L = c through 7 .. 0
    const int h = warp & 1, w = warp >> 1;
    const bool mine = r0 + 8 * h < nrhs;  // uniform over the four warps of a half
    const int ta = 2 * w + (fwd ? 0 : 1), tb = 2 * w + (fwd ? 1 : 0);  // this warp's first and second tile
    // operand of C_l -= X_j (.): L_lj^T (forward) or L_jl (backward), entries (2q + e, g)
    auto off = [&](int l, int j) {
        const double* p = Db + (p1 ? (8 * j + 2 * q) * PD_LD + 8 * l + g : (8 * l + g) * PD_LD + 8 * j + 2 * q);
        return make_double2(p[0], p[p1 ? PD_LD : 1]);
    };
    const double2 va = off(ta, ta), vb = off(tb, tb), vab = off(tb, ta);  // (inverses on the diagonal)
    bool odd = false;  // NaN or infinities among the right-hand sides
    {
        double* p = Xs + row * PD_LDX + 8 * (warp >> 2) + 2 * q;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double c = acc[i] + acc2[i];
            p[8 * (i >> 1) * PD_LDX + (i & 1)] = c;
            odd |= (__double2hiint(c) & 0x7ff00000) == 0x7ff00000;
        }
    }
    odd = __syncthreads_or(odd);
    if (mine) {
        const double* xa = Xs + (8 * ta + 2 * q) * PD_LDX + 8 * h + g;
        const double* xb = Xs + (8 * tb + 2 * q) * PD_LDX + 8 * h + g;
        double Ca[2] = {xa[0], xa[PD_LDX]}, Cb[2] = {xb[0], xb[PD_LDX]};
        double Xa[2] = {0.0, 0.0}, Xb[2] = {0.0, 0.0};
        double* xt = Xt + h * PD_XT + 2 * lane;
        auto solve = [&](const double (&C)[2], int j, double2 v, double (&X)[2]) {
            if (odd) {
                const double2 x = tri_row(C[0], C[1], Db + 8 * j * (PD_LD + 1), p1 ? PD_LD : 1, p1 ? 1 : PD_LD, fwd, lane);
                X[0] = x.x, X[1] = x.y;
                return;
            }
            X[0] = X[1] = 0.0;
            pd_mma8(X, C[0], v.x);
            pd_mma8(X, C[1], v.y);
        };
        auto update = [&](double (&C)[2], double x0, double x1, double2 v) {
            pd_mma8(C, -x0, v.x);
            pd_mma8(C, -x1, v.y);
        };
#pragma unroll
        for (int s = 0; s < RB / 16; ++s) {
            const int jb = fwd ? s : RB / 16 - 1 - s;  // the block solved in this step
            const int ja = 2 * jb + (fwd ? 0 : 1), jc = 2 * jb + (fwd ? 1 : 0);
            double2 o[4];
            if (w == jb) {
                solve(Ca, ta, va, Xa);
                update(Cb, Xa[0], Xa[1], vab);
                solve(Cb, tb, vb, Xb);
                if (s + 1 < RB / 16) {
                    *reinterpret_cast<double2*>(xt + ta * 64) = make_double2(Xa[0], Xa[1]);
                    *reinterpret_cast<double2*>(xt + tb * 64) = make_double2(Xb[0], Xb[1]);
                }
            }
            if (s + 1 == RB / 16) break;
            const bool below = fwd ? w > jb : w < jb;
            if (below) {  // the operands while the block is being solved
                o[0] = off(ta, ja);
                o[1] = off(ta, jc);
                o[2] = off(tb, ja);
                o[3] = off(tb, jc);
            }
            if (h == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
            else asm volatile("bar.sync 2, 128;" ::: "memory");
            if (below) {
                const double2 x0 = *reinterpret_cast<const double2*>(xt + ja * 64);
                const double2 x1 = *reinterpret_cast<const double2*>(xt + jc * 64);
                update(Ca, x0.x, x0.y, o[0]);
                update(Cb, x0.x, x0.y, o[2]);
                update(Ca, x1.x, x1.y, o[1]);
                update(Cb, x1.x, x1.y, o[3]);
            }
        }
        const long long r = r0 + 8 * h + g;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int ia = 8 * ta + 2 * q + e, ib = 8 * tb + 2 * q + e;
            if (r < nrhs && ia < nrows) x_st<TX, BT>(B, ldb, i0 + ia, r, (TX)Xa[e]);
            if (r < nrhs && ib < nrows) x_st<TX, BT>(B, ldb, i0 + ib, r, (TX)Xb[e]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) st_release(&cflags[fwd ? blk : N + blk], 1);  // orders the CTA's stores too
}

template <class T, bool UP, bool BT, class TL = T, bool ID = false, bool FO = false>
cudaError_t potrs_launch(const TL* A, long long lda, T* B, long long ldb, int n, int nrhs, int* flags, int* ticket,
                         int* status, cudaStream_t st, const int* skip = nullptr)
{
    const int N = (int)ceil_div(n, RB);
    const int nchunks = (int)ceil_div(nrhs, RC);
    const long long grid = (ID || FO ? 1LL : 2LL) * N * nchunks;
    const double cf = Traits<T>::cplx ? 4.0 : 1.0;
    const double nd = n, rd = nrhs;
    ProfScope ps(PK_POTRS_FUSED, st,
                 ID ? cf * nd * nd * nd / 3.0 : (FO ? cf * nd * nd * rd : cf * 2.0 * nd * nd * rd),
                 sizeof(TL) * nd * (nd + 1) + sizeof(T) * 4.0 * nd * rd);
    if constexpr (Traits<T>::cplx) {
        const size_t smem = potrs_smem_bytes<T>();
        if (cudaError_t e = smem_optin(k_potrs_fused<T, UP, BT, FO>, smem); e != cudaSuccess) return e;
        k_potrs_fused<T, UP, BT, FO><<<(unsigned)grid, NT, smem, st>>>(A, lda, B, ldb, n, nrhs, nchunks, flags, ticket,
                                                                       status, skip);
    } else {
        const size_t smem = potrs_dmma_smem<TL>();
        if (cudaError_t e = smem_optin(k_potrs_dmma<TL, T, UP, BT, ID, FO>, smem); e != cudaSuccess) return e;
        k_potrs_dmma<TL, T, UP, BT, ID, FO><<<(unsigned)grid, NT, smem, st>>>(A, lda, B, ldb, n, nrhs, nchunks, flags,
                                                                              ticket, status, skip);
    }
    note_launches(1);
    return cudaGetLastError();
}

template <class T>
cudaError_t potrs_typed(char uplo, char side, int n, int nrhs, const void* A, long long lda, void* B, long long ldb,
                        int* flags, int* ticket, int* status, cudaStream_t st, const int* skip)
{
    const T* a = static_cast<const T*>(A);
    T* b = static_cast<T*>(B);
    const bool up = uplo == 'U', bt = side == 'R';
    if (up && bt) return potrs_launch<T, true, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st, skip);
    if (up) return potrs_launch<T, true, false>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st, skip);
    if (bt) return potrs_launch<T, false, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st, skip);
    return potrs_launch<T, false, false>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st, skip);
}

template <class T>
cudaError_t forward_typed(char uplo, char side, int n, int nrhs, const void* A, long long lda, void* B,
                          long long ldb, int* flags, int* ticket, int* status, cudaStream_t st)
{
    const T* a = static_cast<const T*>(A);
    T* b = static_cast<T*>(B);
    const bool up = uplo == 'U', bt = side == 'R';
    if (up && bt)
        return potrs_launch<T, true, true, T, false, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st);
    if (up)
        return potrs_launch<T, true, false, T, false, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st);
    if (bt)
        return potrs_launch<T, false, true, T, false, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st);
    return potrs_launch<T, false, false, T, false, true>(a, lda, b, ldb, n, nrhs, flags, ticket, status, st);
}

cudaError_t potrs_dispatch(char type, char uplo, char side, int n, int nrhs, const void* A, long long lda, void* B,
                           long long ldb, int* flags, int* ticket, int* status, cudaStream_t st,
                           const int* skip = nullptr)
{
    switch (type) {
    case 's': return potrs_typed<float>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st, skip);
    case 'd': return potrs_typed<double>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st, skip);
    case 'c': return potrs_typed<cf32>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st, skip);
    case 'z': return potrs_typed<cf64>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st, skip);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace
}  // namespace ddlak

// Solve with an FP32 factor (uplo 'L') and FP64 right-hand sides in place
// (the refinement solves of the mixed-precision path); same scratch as
// ddlak_potrs.
extern "C" int ddlak_potrs_mixed(int n, int nrhs, const void* L32, long long ldl, const void* /*Dinv*/, void* B,
                                 long long ldb, void* work, unsigned long long work_bytes, void* stream)
{
    using namespace ddlak;
    if (n <= 0 || nrhs <= 0) return 0;
    if (work_bytes < ddlak_potrs_workspace(n, nrhs)) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(work, 0, ddlak_potrs_workspace(n, nrhs), st);
    if (e != cudaSuccess) return (int)e;
    int* status = static_cast<int*>(work);
    int* flags = reinterpret_cast<int*>(static_cast<char*>(work) + 256);
    return (int)potrs_launch<double, false, false, float>(static_cast<const float*>(L32), ldl,
                                                          static_cast<double*>(B), ldb, n, nrhs, flags, status + 1,
                                                          status, st);
}

// Scratch: [status int][ticket int] padded to 256 B, then nchunks * 2N flags.
extern "C" unsigned long long ddlak_potrs_workspace(int n, int nrhs)
{
    if (n <= 0 || nrhs <= 0) return 0;
    const unsigned long long N = (unsigned long long)ddlak::ceil_div(n, ddlak::RB);
    const unsigned long long C = (unsigned long long)ddlak::ceil_div(nrhs, ddlak::RC);
    return 256 + ((C * 2 * N * sizeof(int) + 255) / 256) * 256;
}

// ---------------------------------------------------------------------------
// The same fused solve with its scratch in a fixed, library-owned device array
// instead of memory the caller or the allocator provides.  The array lives
// for the whole process on every device that loads the library (128 KB + 256 B),
// which bounds the problem: n <= 65536 (1024 block rows of 64) and nrhs <= 256
// (16 chunks of 16).  All calls share it, so calls that overlap on the GPU
// race on it; the words that must start at zero are cleared on the caller's
// stream before each launch.
// ---------------------------------------------------------------------------
namespace ddlak {
namespace {
constexpr int kFixedMaxN = 65536;
constexpr int kFixedMaxRhs = 256;
constexpr int kFixedHeaderInts = 64;  // status, ticket, padding to 256 bytes
constexpr int kFixedFlagInts = 2 * (kFixedMaxN / RB) * (kFixedMaxRhs / RC);
__device__ __align__(256) int g_potrs_fixed_scratch[kFixedHeaderInts + kFixedFlagInts];

// Device address of the array on the current device; looked up once per
// device (the first call on a device does the lookup, with that device current)
// and kept for the process's life, which assumes the device's primary context
// is never reset (cudaDeviceReset) while the library is in use.
int* fixed_scratch_ptr(int* err)
{
    static std::mutex mu;
    static int* ptrs[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        *err = e != cudaSuccess ? (int)e : (int)cudaErrorInvalidDevice;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (ptrs[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_potrs_fixed_scratch);
        if (e != cudaSuccess) {
            *err = (int)e;
            return nullptr;
        }
        ptrs[dev] = static_cast<int*>(p);
    }
    *err = 0;
    return ptrs[dev];
}
}  // namespace
}  // namespace ddlak

extern "C" int ddlak_potrs_fixed_scratch_limits(int* max_n, int* max_nrhs)
{
    if (max_n) *max_n = ddlak::kFixedMaxN;
    if (max_nrhs) *max_nrhs = ddlak::kFixedMaxRhs;
    return 0;
}

extern "C" int ddlak_potrs_fixed_scratch(char type, char uplo, char side, int n, int nrhs, const void* A,
                                         long long lda, void* B, long long ldb, int** status_word, void* stream)
{
    using namespace ddlak;
    if (n <= 0 || nrhs <= 0) return 0;
    if (n > kFixedMaxN || nrhs > kFixedMaxRhs) return (int)cudaErrorInvalidValue;
    int err = 0;
    int* base = fixed_scratch_ptr(&err);
    if (base == nullptr) return err;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t flag_ints = (size_t)2 * ceil_div(n, RB) * ceil_div(nrhs, RC);
    cudaError_t e = cudaMemsetAsync(base, 0, (kFixedHeaderInts + flag_ints) * sizeof(int), st);
    if (e != cudaSuccess) return (int)e;
    if (status_word) *status_word = base;
    return (int)potrs_dispatch(type, uplo, side, n, nrhs, A, lda, B, ldb, base + kFixedHeaderInts, base + 1, base,
                               st);
}

extern "C" int ddlak_potrs_after(char type, char uplo, char side, int n, int nrhs, const void* A, long long lda,
                                 void* B, long long ldb, void* work, unsigned long long work_bytes, const int* dinfo,
                                 void* stream)
{
    using namespace ddlak;
    if (n <= 0 || nrhs <= 0) return 0;
    if (work_bytes < ddlak_potrs_workspace(n, nrhs)) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(work, 0, ddlak_potrs_workspace(n, nrhs), st);
    if (e != cudaSuccess) return (int)e;
    int* status = static_cast<int*>(work);
    int* ticket = status + 1;
    int* flags = reinterpret_cast<int*>(static_cast<char*>(work) + 256);
    return (int)potrs_dispatch(type, uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st, dinfo);
}

extern "C" int ddlak_potrs(char type, char uplo, char side, int n, int nrhs, const void* A, long long lda, void* B,
                           long long ldb, void* work, unsigned long long work_bytes, void* stream)
{
    return ddlak_potrs_after(type, uplo, side, n, nrhs, A, lda, B, ldb, work, work_bytes, nullptr, stream);
}

// X = L^-1 B (side 'L', B n x nrhs) or X = B L^-H (side 'R', B nrhs x n), in place,
// with the factor read through its L view (uplo 'L': A's lower triangle; 'U': L = U^H):
// the forward half of ddlak_potrs.  Same scratch (ddlak_potrs_workspace(n, nrhs)) and
// status word.
extern "C" int ddlak_forward_solve(char type, char uplo, char side, int n, int nrhs, const void* A, long long lda,
                                   void* B, long long ldb, void* work, unsigned long long work_bytes, void* stream)
{
    using namespace ddlak;
    if (n <= 0 || nrhs <= 0) return 0;
    if (!A || !B || work_bytes < ddlak_potrs_workspace(n, nrhs)) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(work, 0, ddlak_potrs_workspace(n, nrhs), st);
    if (e != cudaSuccess) return (int)e;
    int* status = static_cast<int*>(work);
    int* ticket = status + 1;
    int* flags = reinterpret_cast<int*>(static_cast<char*>(work) + 256);
    switch (type) {
    case 's': return (int)forward_typed<float>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st);
    case 'd': return (int)forward_typed<double>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st);
    case 'c': return (int)forward_typed<cf32>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st);
    case 'z': return (int)forward_typed<cf64>(uplo, side, n, nrhs, A, lda, B, ldb, flags, ticket, status, st);
    default: return (int)cudaErrorInvalidValue;
    }
}

// FP32 order from which the inversion is done by doubling (sgemm.cu); below it by the fused
// substitution on the identity, whose time is n / 64 links where doubling has two launches and
// a 64-wide serial leaf per level.  us, substitution / doubling, leading dimension n:
//   n = 200 28 / 130   1025 88 / 674   2048 282 / 616   3600 1183 / 1300   3800 1357 / 1346
//   4096 1605 / 1393   4100 1678 / 2040   8192 11790 / 5562
//   odd, without TMA: 5003 2879 / 3079   6001 4733 / 4183   8191 11861 / 7530
static constexpr int kTrtriDoubling = 3800;

// W = L^-1 for a lower factor: FP64, and FP32 below that order, by the fused forward
// substitution on the identity, FP32 from there by doubling (sgemm.cu).
extern "C" int ddlak_trtri_blocked(char type, int n, const void* L, long long ldl, void* W, long long ldw, void* work,
                                   unsigned long long work_bytes, void* stream)
{
    using namespace ddlak;
    if (n <= 0) return 0;
    if (!L || !W || ldl < n || ldw < n || work_bytes < ddlak_potrs_workspace(n, n)) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(work, 0, ddlak_potrs_workspace(n, n), st);
    if (e != cudaSuccess) return (int)e;
    int* status = static_cast<int*>(work);
    int* ticket = status + 1;
    int* flags = reinterpret_cast<int*>(static_cast<char*>(work) + 256);
    if (type == 'd')
        return (int)potrs_launch<double, false, false, double, true>(
            static_cast<const double*>(L), ldl, static_cast<double*>(W), ldw, n, n, flags, ticket, status, st);
    if (type == 's' && n < kTrtriDoubling)
        return (int)potrs_launch<float, false, false, float, true>(
            static_cast<const float*>(L), ldl, static_cast<float*>(W), ldw, n, n, flags, ticket, status, st);
    if (type == 's') return (int)trtri_large_f32(n, static_cast<const float*>(L), ldl, static_cast<float*>(W), ldw,
                                                 status, st);
    return (int)cudaErrorInvalidValue;
}
