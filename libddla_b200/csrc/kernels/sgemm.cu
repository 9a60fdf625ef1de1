// FP32 products of the blocked Cholesky on the CUDA cores (sgemm.cuh): the trailing
// update of either triangle, and the recursive inversion of a large lower factor.
#include <type_traits>

#include <ddla_kernels.h>

#include "common.cuh"
#include "ddla_kernels_internal.h"
#include "profile.h"
#include "sgemm.cuh"

namespace ddlak {

namespace {

// The code of an update wait that gave up, for a debugger: the caller sees NaN in the tile and the
// failed pivot it makes.
__device__ int g_sgemm_status;

// C(i, j) -= sum_{k0 <= k < k0 + nbk} L(i, k) L(j, k) on the lower tiles of the region from
// row / column t0 (cols == 0: all of it; else its first cols columns).
// What bounds it: the FP32 pipe.
template <bool UP, bool TMA>
__global__ void __launch_bounds__(sg::NT, UP ? 1 : 2)
    k_syrk_f32(const __grid_constant__ CUtensorMap map, float* __restrict__ A, long long lda, int k0, int nbk, int n,
               long long t0, int cols, const int* __restrict__ info)
{
    extern __shared__ __align__(128) unsigned char sg_raw[];
    if (*(volatile const int*)info != 0) return;
    int I, J;
    if (cols == 0) {
        tile_of_tri(blockIdx.x, I, J);
    } else {
        const int nct = (cols + sg::TILE - 1) / sg::TILE;
        J = blockIdx.x % nct;
        I = blockIdx.x / nct;
        if (I < J) return;
    }
    const long long cend = cols == 0 ? (long long)n : t0 + cols;
    const long long ri = t0 + (long long)I * sg::TILE, rj = t0 + (long long)J * sg::TILE;
    float acc[8][8];
    sg::tile<UP, UP, TMA, sg::ALL, sg::ALL>(&map, &map, A, lda, A, lda, ri, rj, n, n, k0, nbk / sg::KC, k0 + nbk, 0, 0,
                                            sg_raw, &g_sgemm_status, acc);
    const int ty = sg::thread_row(), tx = sg::thread_col();
    if (!UP && TMA && I > J && ri + sg::TILE <= n && rj + sg::TILE <= cend) {
        // a whole tile below the diagonal: four rows per access (TMA: 16-byte aligned columns)
#pragma unroll
        for (int o = 0; o < 8; o += 2) {
            float4 c[2][2];
            float* p = A + ri + 4 * ty + (rj + sg::col_of<UP, UP>(tx, o)) * lda;  // columns o, o + 1 are neighbours
#pragma unroll
            for (int x = 0; x < 4; ++x)
                c[x >> 1][x & 1] = __ldcg(reinterpret_cast<const float4*>(p + (x >> 1) * lda + 64 * (x & 1)));
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int v = o + (x >> 1), u = 4 * (x & 1);
                float4 q = c[x >> 1][x & 1];
                q.x -= acc[u][v], q.y -= acc[u + 1][v], q.z -= acc[u + 2][v], q.w -= acc[u + 3][v];
                *reinterpret_cast<float4*>(p + (x >> 1) * lda + 64 * (x & 1)) = q;
            }
        }
        return;
    }
    // C -= acc, a row's (UP) or a column's (lower) values loaded together before any store
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        float c[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int u = UP ? o : x, v = UP ? x : o;
            const long long i = ri + sg::row_of<UP, UP>(ty, u), j = rj + sg::col_of<UP, UP>(tx, v);
            c[x] = i < n && j < cend && i >= j ? __ldcg(UP ? A + j + i * lda : A + i + j * lda) : 0.f;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int u = UP ? o : x, v = UP ? x : o;
            const long long i = ri + sg::row_of<UP, UP>(ty, u), j = rj + sg::col_of<UP, UP>(tx, v);
            if (i < n && j < cend && i >= j) *(UP ? A + j + i * lda : A + i + j * lda) = c[x] - acc[u][v];
        }
    }
}

// ---------------------------------------------------------------------------
// W = L^-1 (lower, any order) by doubling: 64 x 64 leaves, then at each level h the
// inverses W11 and W22 of neighbouring h-blocks give W21 = -W22 (L21 W11).  The product
// T = L21 W11 waits, transposed, in W's strictly upper triangle (rows r0 .., columns
// r0 + h ..), so what lies above the diagonal of W is scratch and is masked wherever a
// tile reaches it.  blockIdx.y: the pair; tiles of 128 x 128.
// ---------------------------------------------------------------------------
template <int STEP, bool TMA>
__global__ void __launch_bounds__(sg::NT, 2)
    k_trtri_level_f32(const __grid_constant__ CUtensorMap lmap, const __grid_constant__ CUtensorMap wmap, int n, int h,
                      int nt, const float* __restrict__ L, long long ldl, float* __restrict__ W, long long ldw,
                      int* status)
{
    extern __shared__ __align__(128) unsigned char sg_raw[];
    const long long r0 = 2LL * h * blockIdx.y;
    const int m2 = (int)min((long long)h, (long long)n - r0 - h);  // rows of the second block
    const int ti = blockIdx.x / nt, tj = blockIdx.x % nt;
    const int i0 = ti * sg::TILE, j0 = tj * sg::TILE;
    if (m2 <= 0 || i0 >= m2) return;
    float acc[8][8];
    const int ty = sg::thread_row(), tx = sg::thread_col();
    if constexpr (STEP == 1) {
        // T(i, j) = sum_{j0 <= k < h} L21(i, k) W11(k, j); W11(k, j) counts for k >= j
        sg::tile<false, true, TMA, sg::ALL, sg::K_GE_ROW>(&lmap, &wmap, L, ldl, W, ldw, r0 + h + i0, r0 + j0, n, n,
                                                          r0 + j0, (h - j0 + sg::KC - 1) / sg::KC, r0 + h,
                                                          sg::TILE / sg::KC, 1 << 30, sg_raw, status, acc);
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const int i = i0 + sg::row_of<false, true>(ty, u), j = j0 + sg::col_of<false, true>(tx, v);
                if (i < m2 && j < h) W[(r0 + j) + (r0 + h + i) * ldw] = acc[u][v];
            }
    } else {
        // W21(i, j) = -sum_{k <= i} W22(i, k) T(k, j)
        const int kn = min(i0 + sg::TILE, m2);
        sg::tile<false, false, TMA, sg::K_LE_ROW, sg::ALL>(&wmap, &wmap, W, ldw, W, ldw, r0 + h + i0, r0 + j0, n, n,
                                                           r0 + h, (kn + sg::KC - 1) / sg::KC, r0 + h + kn, 0,
                                                           i0 / sg::KC, sg_raw, status, acc);
#pragma unroll
        for (int v = 0; v < 8; ++v)
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + sg::row_of<false, false>(ty, u), j = j0 + sg::col_of<false, false>(tx, v);
                if (i < m2 && j < h) W[(r0 + h + i) + (r0 + j) * ldw] = -acc[u][v];
            }
    }
}

// The 64 x 64 diagonal blocks' inverses: one thread per column, four blocks per CTA, FP64
// arithmetic, the column in registers (152 bytes of them spilled) and L through the L1 cache.
// What bounds it: one thread's serial column, 87 us at n = 8192 and 54 at 64, which is why small
// factors are inverted another way (kTrtriDoubling, potrs.cu).
constexpr int SL = 64;
__global__ void __launch_bounds__(256) k_trtri_leaf_f32(int nleaf, int n, const float* __restrict__ Lg, long long ldl,
                                                        float* __restrict__ Wg, long long ldw)
{
    const int leaf = blockIdx.x * 4 + (threadIdx.x >> 6);
    if (leaf >= nleaf) return;
    const int o = leaf * SL, nb = min(SL, n - o), j = threadIdx.x & 63;
    const float* L = Lg + o + (long long)o * ldl;
    float* W = Wg + o + (long long)o * ldw;
    double w[SL];
#pragma unroll
    for (int i = 0; i < SL; ++i) {
        double s = 0.0;
        const bool row = i < nb;
#pragma unroll
        for (int k = 0; k < i; ++k)
            if (row && k >= j) s = fma((double)__ldg(&L[i + (long long)k * ldl]), w[k], s);
        const double lii = row ? (double)__ldg(&L[i + (long long)i * ldl]) : 1.0;
        w[i] = (i < j || !row) ? 0.0 : (i == j ? 1.0 / lii : -s / lii);
    }
    if (j < nb)
#pragma unroll
        for (int i = 0; i < SL; ++i)
            if (i >= j && i < nb) W[i + (long long)j * ldw] = (float)w[i];
}

}  // namespace

template <bool UP>
cudaError_t syrk_f32(float* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                     cudaStream_t st)
{
    const long long m = (long long)n - t0;
    if (m <= 0) return cudaSuccess;
    if (nbk <= 0 || nbk % sg::KC != 0) return cudaErrorInvalidValue;
    const long long t = ceil_div(m, sg::TILE);
    const unsigned grid = (unsigned)(cols == 0 ? t * (t + 1) / 2 : t * ceil_div(cols, sg::TILE));
    constexpr size_t smem = sg::smem<UP, UP>();
    CUtensorMap map{};
    if (!(t0 & 3) && sg::encode<UP>(&map, A, n, lda)) {
        if (cudaError_t e = smem_optin(k_syrk_f32<UP, true>, smem); e != cudaSuccess) return e;
        k_syrk_f32<UP, true><<<grid, sg::NT, smem, st>>>(map, A, lda, k0, nbk, n, t0, cols, dinfo);
    } else {
        if (cudaError_t e = smem_optin(k_syrk_f32<UP, false>, smem); e != cudaSuccess) return e;
        k_syrk_f32<UP, false><<<grid, sg::NT, smem, st>>>(map, A, lda, k0, nbk, n, t0, cols, dinfo);
    }
    return cudaGetLastError();
}
template cudaError_t syrk_f32<false>(float*, long long, int, int, int, long long, int, const int*, cudaStream_t);
template cudaError_t syrk_f32<true>(float*, long long, int, int, int, long long, int, const int*, cudaStream_t);

cudaError_t trtri_large_f32(int n, const float* L, long long ldl, float* W, long long ldw, int* status, cudaStream_t st)
{
    const int nleaf = (int)ceil_div(n, SL);
    k_trtri_leaf_f32<<<(unsigned)ceil_div(nleaf, 4), 256, 0, st>>>(nleaf, n, L, ldl, W, ldw);
    note_launches(1);
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
    CUtensorMap lrow{}, wrow{}, wk{};
    const bool tma = sg::encode<false>(&lrow, L, n, ldl) && sg::encode<false>(&wrow, W, n, ldw) &&
                     sg::encode<true>(&wk, W, n, ldw);
    constexpr size_t s1 = sg::smem<false, true>(), s2 = sg::smem<false, false>();
    cudaError_t e = tma ? smem_optin(k_trtri_level_f32<1, true>, s1) : smem_optin(k_trtri_level_f32<1, false>, s1);
    if (e == cudaSuccess)
        e = tma ? smem_optin(k_trtri_level_f32<2, true>, s2) : smem_optin(k_trtri_level_f32<2, false>, s2);
    if (e != cudaSuccess) return e;
    for (int h = SL; h < n; h *= 2) {
        const int nt = (int)ceil_div(h, sg::TILE);
        const dim3 grid((unsigned)(nt * nt), (unsigned)ceil_div(n - h, 2 * h));
        if (tma) {
            k_trtri_level_f32<1, true><<<grid, sg::NT, s1, st>>>(lrow, wk, n, h, nt, L, ldl, W, ldw, status);
            k_trtri_level_f32<2, true><<<grid, sg::NT, s2, st>>>(lrow, wrow, n, h, nt, L, ldl, W, ldw, status);
        } else {
            k_trtri_level_f32<1, false><<<grid, sg::NT, s1, st>>>(lrow, wk, n, h, nt, L, ldl, W, ldw, status);
            k_trtri_level_f32<2, false><<<grid, sg::NT, s2, st>>>(lrow, wrow, n, h, nt, L, ldl, W, ldw, status);
        }
        note_launches(2);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ddlak
