// FP32 tile products on the CUDA cores: acc(i, j) = sum_k A(i, k) B(j, k) for one
// 128 x 128 tile, 256 threads, 8 x 8 results per thread, packed two-wide FMAs
// (fma.rn.f32x2), K in slices of 32 through a three-stage ring.
//
// Each operand is read as it lies in memory:
//   rows contiguous (AK / BK false)  A(i, k) = A[i + k * lda], slice [32 k][128 rows]
//   k contiguous    (AK / BK true)   A(i, k) = A[k + i * lda], slice [128 rows][36]
// With both k contiguous a packed FMA takes two k of one (i, j); otherwise two rows i.
// Slices come by TMA (16-byte aligned base, lda a multiple of 4) or by 4-byte cp.async
// (any lda); rows past the matrix arrive as zeros.  Each warp releases a stage by itself
// and the stage of slice c - 1 is refilled after slice c (no CTA barrier per slice).
// Every wait is bounded; a tile whose wait gave up is all NaN (its code goes to *status).
// Spills (-Xptxas -v): 20 to 28 bytes in the update, 76 in the inversion's first product with TMA
// and 508 without (odd leading dimensions), 44 to 180 in the contraction: a packed tile is 64
// registers of sums and 48 of operands, the masks and the epilogue do not fit beside them.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tc_common.cuh"

namespace ddlak {
namespace sg {

constexpr int TILE = 128, KC = 32, NS = 3, NT = 256;
template <bool K>
__host__ __device__ constexpr int ld() { return K ? KC + 4 : TILE; }
template <bool K>
__host__ __device__ constexpr int box() { return K ? TILE * ld<K>() : KC * ld<K>(); }
template <bool AK, bool BK>
__host__ __device__ constexpr size_t smem() { return (size_t)NS * (box<AK>() + box<BK>()) * sizeof(float) + 128; }

template <bool K>
inline bool encode(CUtensorMap* map, const float* A, int n, long long lda)
{
    return tc::encode_colmajor_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, A, n, n, lda, K ? ld<K>() : TILE,
                                  K ? TILE : KC, CU_TENSOR_MAP_SWIZZLE_NONE);
}

__device__ __forceinline__ uint64_t pack2(float x, float y)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// the rows and columns of thread t's results, relative to the tile
template <bool AK, bool BK>
__device__ __forceinline__ int row_of(int ty, int u) { return AK ? ty + 16 * u : (u < 4 ? 4 * ty + u : 60 + 4 * ty + u); }
template <bool AK, bool BK>
__device__ __forceinline__ int col_of(int tx, int v) { return BK ? tx + 16 * v : (v < 4 ? 4 * tx + v : 60 + 4 * tx + v); }
__device__ __forceinline__ int thread_row() { return (threadIdx.x >> 6) * 4 + ((threadIdx.x & 31) >> 3); }
__device__ __forceinline__ int thread_col() { return ((threadIdx.x >> 5) & 1) * 8 + (threadIdx.x & 7); }

// Which entries of an operand count (absolute indices): all, k <= row, or k >= row.
enum Mask { ALL, K_LE_ROW, K_GE_ROW };

// The tile with first rows ar (of A) and br (of B), k in [k0, k0 + 32 nchunks) cut at klim.
// Entries at or past alim / blim rows and klim are zero (with TMA: the map's extents).
// Slices c < edge_lo or c >= edge_hi are read through the masks.
template <bool AK, bool BK, bool TMA, Mask MA, Mask MB>
__device__ __forceinline__ void tile(const CUtensorMap* amap, const CUtensorMap* bmap, const float* A, long long lda,
                                     const float* B, long long ldb, long long ar, long long br, long long alim,
                                     long long blim, long long k0, int nchunks, long long klim, int edge_lo,
                                     int edge_hi, unsigned char* raw, int* status, float (&acc)[8][8])
{
    __shared__ __align__(8) uint64_t full[NS], empty[NS];
    constexpr int LA = ld<AK>(), LB = ld<BK>(), ABOX = box<AK>(), BBOX = box<BK>();
    constexpr bool KP = AK && BK;  // packed along k
    float* sm = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(raw) + 127) & ~uintptr_t(127));
    const int t = threadIdx.x, lane = t & 31;
    const int ty = thread_row(), tx = thread_col();
    if (t == 0) {
        for (int s = 0; s < NS; ++s) {
            tc::mbar_init(&full[s], TMA ? 1 : NT);
            tc::mbar_init(&empty[s], NT / 32);
        }
        tc::mbar_fence_init();
    }
    auto copy = [&](float* dst, const float* M, long long ldm, long long r0, long long rlim, long long kk, bool kcon) {
        for (int x = t; x < TILE * KC; x += NT) {
            const int r = kcon ? x / KC : x % TILE, k = kcon ? x % KC : x / TILE;
            const bool in = r0 + r < rlim && kk + k < klim;
            cp_async_elem<4>(dst + (kcon ? r * (KC + 4) + k : k * TILE + r),
                             in ? (kcon ? M + (kk + k) + (r0 + r) * ldm : M + (r0 + r) + (kk + k) * ldm) : M, in);
        }
    };
    auto issue = [&](int c) {
        const int s = c % NS;
        float* st = sm + (size_t)s * (ABOX + BBOX);
        const long long kk = k0 + (long long)c * KC;
        if constexpr (TMA) {
            tc::mbar_expect_tx(&full[s], (ABOX + BBOX) * 4u);
            tc::tma_load_2d(st, amap, &full[s], (int)(AK ? kk : ar), (int)(AK ? ar : kk));
            tc::tma_load_2d(st + ABOX, bmap, &full[s], (int)(BK ? kk : br), (int)(BK ? br : kk));
        } else {
            copy(st, A, lda, ar, alim, kk, AK);
            copy(st + ABOX, B, ldb, br, blim, kk, BK);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(&full[s])) : "memory");
        }
    };
    const bool issuer = !TMA || t == 0;
    if (TMA && issuer) {
        tc::prefetch_tmap(amap);
        tc::prefetch_tmap(bmap);
        for (int c = 0; c < NS && c < nchunks; ++c) issue(c);
    }
    __syncthreads();
    if (!TMA)
        for (int c = 0; c < NS && c < nchunks; ++c) issue(c);

    constexpr int PR = KP ? 8 : 4;
    uint64_t p[PR][8];
#pragma unroll
    for (int u = 0; u < PR; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) p[u][v] = 0;

    auto keep = [](Mask m, long long k, long long r) { return m == ALL || (m == K_LE_ROW ? k <= r : k >= r); };
    auto step = [&](const float* As, const float* Bs, long long kk, auto edge) {
        constexpr bool EDGE = decltype(edge)::value;
#pragma unroll
        for (int k4 = 0; k4 < KC; k4 += 4) {
            float b[8][4];  // BK: columns' four k; otherwise transposed below
            if constexpr (BK) {
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    const float4 q = *reinterpret_cast<const float4*>(Bs + (tx + 16 * v) * LB + k4);
                    b[v][0] = q.x, b[v][1] = q.y, b[v][2] = q.z, b[v][3] = q.w;
                    if constexpr (EDGE && MB != ALL) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (!keep(MB, kk + k4 + k, br + tx + 16 * v)) b[v][k] = 0.f;
                    }
                }
            }
            if constexpr (KP) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    float4 q = *reinterpret_cast<const float4*>(As + (ty + 16 * u) * LA + k4);
                    if constexpr (EDGE && MA != ALL) {
                        const long long r = ar + ty + 16 * u;
                        if (!keep(MA, kk + k4, r)) q.x = 0.f;
                        if (!keep(MA, kk + k4 + 1, r)) q.y = 0.f;
                        if (!keep(MA, kk + k4 + 2, r)) q.z = 0.f;
                        if (!keep(MA, kk + k4 + 3, r)) q.w = 0.f;
                    }
                    const uint64_t a0 = pack2(q.x, q.y), a1 = pack2(q.z, q.w);
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        fma2(p[u][v], a0, pack2(b[v][0], b[v][1]));
                        fma2(p[u][v], a1, pack2(b[v][2], b[v][3]));
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float a[8];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 q = *reinterpret_cast<const float4*>(As + (k4 + k) * LA + 64 * h + 4 * ty);
                        a[4 * h] = q.x, a[4 * h + 1] = q.y, a[4 * h + 2] = q.z, a[4 * h + 3] = q.w;
                    }
                    if constexpr (EDGE && MA != ALL) {
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (!keep(MA, kk + k4 + k, ar + row_of<AK, BK>(ty, u))) a[u] = 0.f;
                    }
                    if constexpr (!BK) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float4 q = *reinterpret_cast<const float4*>(Bs + (k4 + k) * LB + 64 * h + 4 * tx);
                            b[4 * h][k] = q.x, b[4 * h + 1][k] = q.y, b[4 * h + 2][k] = q.z, b[4 * h + 3][k] = q.w;
                        }
                    }
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        const uint64_t bb = pack2(b[v][k], b[v][k]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) fma2(p[u][v], pack2(a[2 * u], a[2 * u + 1]), bb);
                    }
                }
            }
        }
    };

    bool ok = true;
    int consumed = 0, issued = nchunks < NS ? nchunks : NS;
    for (int c = 0; c < nchunks; ++c) {
        const int s = c % NS;
        if (!tc::mbar_wait(&full[s], (uint32_t)((c / NS) & 1), status, 0x61)) {
            ok = false;
            break;
        }
        consumed = c + 1;
        const float* As = sm + (size_t)s * (ABOX + BBOX);
        const float* Bs = As + ABOX;
        const long long kk = k0 + (long long)c * KC;
        if constexpr (MA == ALL && MB == ALL) {
            step(As, Bs, kk, std::false_type{});
        } else {
            if (c < edge_lo || c >= edge_hi) step(As, Bs, kk, std::true_type{});
            else step(As, Bs, kk, std::false_type{});
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);
        if (issuer && c >= 1 && c - 1 + NS < nchunks) {
            const int cp = c - 1;
            if (!tc::mbar_wait(&empty[cp % NS], (uint32_t)((cp / NS) & 1), status, 0x64)) {
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
        if (t == 0)
            for (int c = consumed; c < issued; ++c)
                (void)tc::mbar_wait(&full[c % NS], (uint32_t)((c / NS) & 1), status, 0x62);
        __syncthreads();
    }
    const float bad = ok ? 0.f : __int_as_float(0x7fc00000);
#pragma unroll
    for (int u = 0; u < PR; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const float2 r = unpack2(p[u][v]);
            if constexpr (KP) {
                acc[u][v] = r.x + r.y + bad;
            } else {
                acc[2 * u][v] = r.x + bad;
                acc[2 * u + 1][v] = r.y + bad;
            }
        }
}

}  // namespace sg
}  // namespace ddlak
