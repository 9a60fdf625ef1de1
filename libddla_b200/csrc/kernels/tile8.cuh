// Cholesky of one 8 x 8 tile with its inverse, by one warp (the pivot chain of panel.cu and
// vbatched.cu).
#pragma once
#include "common.cuh"

namespace ddlak {

// Is an entry of the N tiles NaN or infinite, in any lane of the warp?  (integer pipe)
template <int N>
__device__ __forceinline__ bool any_nonfinite(const double (&C)[N][4])
{
    constexpr int e = 0x7ff00000;
    bool odd = false;
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
        for (int i = 0; i < 4; ++i) odd |= (__double2hiint(C[l][i]) & e) == e;
    return __any_sync(0xffffffffu, odd);
}

// One row of X = C M for an 8 x 8 triangular M, M(m, c) = mat[m * sm + c * sc] zero for m > c
// (low) or m < c, without its zeros' products: an infinite or NaN entry of C reaches
// the columns it belongs to and no others, as in substitution.  For rows that hold one;
// the others take the tensor-core product of the whole tile.  Lanes 4g .. 4g + 3 hold row g,
// lane q of them the entries 2q and 2q + 1; all lanes of the warp.  Out of line: inlined it cost
// the batched kernel 4 % (FP32, code size) on matrices that never take it.
static __device__ __noinline__ double2 tri_row(double c0, double c1, const double* mat, int sm, int sc, bool low, int lane)
{
    double x[2] = {0.0, 0.0};
#pragma unroll 1
    for (int m = 0; m < 8; ++m) {
        const int src = (lane & ~3) | (m >> 1);
        const double u = __shfl_sync(0xffffffffu, c0, src), v = __shfl_sync(0xffffffffu, c1, src);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = 2 * (lane & 3) + e;
            if (low ? m <= c : m >= c) x[e] = fma(m & 1 ? v : u, mat[m * sm + c * sc], x[e]);
        }
    }
    return make_double2(x[0], x[1]);
}

// factor_tile8 for a tile with a pivot that is subnormal or infinite, outside the range of
// rsqrt_pivot: by CUDA's square root and division, lane 0 the factor, lane c column c of the
// inverse.
static __device__ __noinline__ int factor_tile8_wide(const double* T, double* Inv, double* Lt, double* rinv, int kv,
                                                     int lane)
{
    int good = kv;
    if (lane == 0) {
        for (int e = 0; e < 64; ++e) Lt[e] = (e & 7) <= (e >> 3) ? T[e] : 0.0;
        for (int k = 0; k < kv; ++k) {
            const double d = Lt[k * 9];
            if (!(d > 0.0)) {
                good = k;
                break;
            }
            const double s = sqrt(d);
            Lt[k * 9] = s;
            for (int i = k + 1; i < 8; ++i) Lt[i * 8 + k] /= s;
            for (int i = k + 1; i < 8; ++i)
                for (int m = k + 1; m <= i && m < kv; ++m) Lt[i * 8 + m] -= Lt[i * 8 + k] * Lt[m * 8 + k];
        }
    }
    good = __shfl_sync(0xffffffffu, good, 0);
    __syncwarp();
    if (lane < 8) {
        for (int i = 0; i < 8; ++i) {
            double s = i == lane ? 1.0 : 0.0;
            if (i < good)
                for (int k = lane; k < i; ++k) s -= Lt[i * 8 + k] * Inv[k * 8 + lane];
            Inv[i * 8 + lane] = i >= lane && i < good ? s / Lt[i * 9] : 0.0;
        }
        if (rinv != nullptr && lane < good) rinv[lane] = 1.0 / Lt[lane * 9];
    }
    __syncwarp();
    return good;
}

// T: the tile in shared memory, row-major, lower part.  Its first kv columns are factored,
// redundantly in every lane (a column costs one reciprocal square root, a multiply and a
// multiply-add, no shuffles; lane c carries column c of the inverse along): L into Lt
// (row-major; the columns before a failed one final, that one with the values updated by
// them), the inverse into Inv (row-major; its rows from a failed column on are zero), 1 / l_kk
// into rinv[k] when given.  Returns the number of factored columns: kv, or the index of the
// first pivot that is not positive.  Rows from kv on are solved against the columns before kv
// like any row below; their own columns are decoupled by a huge diagonal.
// Everything is straight-line code on values all lanes hold, stores included (every lane
// stores the same word): predicating the 36 stores of L on a lane each made the tile take
// 7900 clocks instead of 1000.
__device__ __forceinline__ int factor_tile8(const double* T, double* Inv, double* Lt, double* rinv, int kv, int lane)
{
    double a[8][8], y[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int h = 0; h <= r / 2; ++h) {
            const double2 v = *reinterpret_cast<const double2*>(&T[r * 8 + 2 * h]);
            a[r][2 * h] = v.x;
            a[r][2 * h + 1] = v.y;
        }
#pragma unroll
    for (int r = 1; r < 8; ++r)
        if (r >= kv) {  // uniform
#pragma unroll
            for (int c = 0; c < r; ++c)
                if (c >= kv) a[r][c] = 0.0;
            a[r][r] = 1e300;
        }
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = (lane & 7) == i ? 1.0 : 0.0;
    int good = 8;
    double rk = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double d = a[k][k];
        if (good == 8 && !(d > 0.0)) good = k;
        const bool live = good == 8;
        const double rs = rsqrt_pivot(d);
        const double r = live ? rs : 0.0;
        rk = lane == k ? r : rk;
#pragma unroll
        for (int i = k + 1; i < 8; ++i) {
            const double l = a[i][k] * r;
#pragma unroll
            for (int m = k + 1; m < i; ++m) a[i][m] = fma(-l, a[m][k], a[i][m]);
            a[i][i] = fma(-l, l, a[i][i]);
            a[i][k] = live ? l : a[i][k];
        }
        const double s = d * r;
        a[k][k] = live ? fma(0.5 * r, fma(-s, s, d), s) : d;
        y[k] *= r;
#pragma unroll
        for (int i = k + 1; i < 8; ++i) y[i] = fma(live ? -a[i][k] : 0.0, y[k], y[i]);
    }
    good = good < kv ? good : kv;
    if (lane < 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Inv[i * 8 + lane] = y[i];
        if (rinv != nullptr && lane < good) rinv[lane] = rk;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int h = 0; h <= r / 2; ++h)
            *reinterpret_cast<double2*>(&Lt[r * 8 + 2 * h]) = make_double2(a[r][2 * h], 2 * h + 1 <= r ? a[r][2 * h + 1] : 0.0);
    __syncwarp();
    // once more where a pivot was subnormal or infinite: its reciprocal root is NaN or infinite then
    // (asked here, behind the stores, which hide behind the chain of pivots)
    if (__any_sync(0xffffffffu, (__double2hiint(rk) & 0x7ff00000) == 0x7ff00000))
        good = factor_tile8_wide(T, Inv, Lt, rinv, kv, lane);
    return good;
}

}  // namespace ddlak
