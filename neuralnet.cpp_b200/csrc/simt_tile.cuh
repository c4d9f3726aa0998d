// Building blocks of the fp32 attention kernels (attention_simt.cu, engine_prims.cu): a block of 256 threads works on
// 64 x 64 tiles, thread (ty, tx) = (t / 16, t % 16) owning rows 4 ty .. 4 ty + 3 and columns 4 tx .. 4 tx + 3 (or a run of
// W columns at W tx).  Operands are staged as X[k][64], so that a step of k reads two 16-byte vectors per thread for 16
// fused multiply-adds; the packed fp32 pair instructions halve their issue slots.
#pragma once
#include "kernels.h"
#include "tc_ptx.cuh"

namespace nnb {

constexpr int kTile = 64, kTilePitch = 68;                       // rows of 68 floats: vectors stay 16-byte aligned
constexpr int kTileFloats = kTile * kTilePitch;

// X[k][i] = base[(i0 + i) * si + (k0 + k) * sk] for i < 64, k < KC; zero outside i < ni, k < nk.  Lanes run along the
// index whose stride is 1.
template <int KC, typename T>
__device__ __forceinline__ void stage_tile(float* __restrict__ X, const T* __restrict__ base, long long si, long long sk, int i0, int ni,
                                           int k0, int nk)
{
    static_assert(KC % 8 == 0 && KC <= 64, "chunk of the contraction");
    constexpr int N = kTile * KC / 256;
    float v[N];
    if (sk == 1) {
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int e = threadIdx.x + u * 256, k = e % KC, i = e / KC;
            v[u] = (i0 + i < ni && k0 + k < nk) ? to_f32(base[(i0 + i) * si + k0 + k]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < N; ++u) { const int e = threadIdx.x + u * 256; X[(e % KC) * kTilePitch + e / KC] = v[u]; }
    } else {
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int e = threadIdx.x + u * 256, i = e & 63, k = e >> 6;
            v[u] = (i0 + i < ni && k0 + k < nk) ? to_f32(base[(i0 + i) * si + (k0 + k) * sk]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < N; ++u) { const int e = threadIdx.x + u * 256; X[(e >> 6) * kTilePitch + (e & 63)] = v[u]; }
    }
}

// X[r][c] = base[(r0 + r) * sr + (c0 + c) * sc] for r < 64, c < C, rows of C + 4 floats; zero outside r < nr, c < nc
template <int C, typename T>
__device__ __forceinline__ void stage_rows(float* __restrict__ X, const T* __restrict__ base, long long sr, long long sc, int r0, int nr,
                                           int c0, int nc)
{
    constexpr int N = (kTile * C + 255) / 256;
#pragma unroll 8
    for (int u = 0; u < N; ++u) {
        const int e = threadIdx.x + u * 256;
        int r, c;
        if (sc == 1) { r = e / C; c = e % C; } else { r = e & 63; c = e >> 6; }
        if (r < kTile && c < C) X[r * (C + 4) + c] = (r0 + r < nr && c0 + c < nc) ? to_f32(base[(r0 + r) * sr + (c0 + c) * sc]) : 0.f;
    }
}

// acc[r][c] += sum_k A[k][4 ty + r] * B[k][4 tx + c]
template <int KC>
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float* __restrict__ A, const float* __restrict__ B)
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    uint64_t s[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) { s[r][0] = pack2(acc[r][0], acc[r][1]); s[r][1] = pack2(acc[r][2], acc[r][3]); }
#pragma unroll 8
    for (int k = 0; k < KC; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(A + k * kTilePitch + ty * 4);
        const float4 b = *reinterpret_cast<const float4*>(B + k * kTilePitch + tx * 4);
        const uint64_t b0 = pack2(b.x, b.y), b1 = pack2(b.z, b.w);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t ar = pack2(av[r], av[r]);
            s[r][0] = fma2(ar, b0, s[r][0]);
            s[r][1] = fma2(ar, b1, s[r][1]);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) { unpack2(s[r][0], acc[r][0], acc[r][1]); unpack2(s[r][1], acc[r][2], acc[r][3]); }
}

// acc[r][c] += sum_{k < 64} A[k][4 ty + r] * B[k][W tx + c] over the terms with open(k, 4 ty + r), rows of B of C + 4 floats;
// threads with W tx >= C have nothing.  The terms are added up in runs of RUN, the runs of a tile with one another, and the
// tile to acc: one chain over all rows rounds at its full size every time, an error that grows with their number.
struct AllOpen { __device__ __forceinline__ bool operator()(int, int) const { return true; } };
template <int W, int C, int RUN = kTile, typename Open = AllOpen>
__device__ __forceinline__ void tile_rows_product(float (&acc)[4][W], const float* __restrict__ A, const float* __restrict__ B, Open open = {})
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (W * tx >= C) return;
    auto add_terms = [&](float (&to)[4][W], int k0) {
#pragma unroll(RUN < 8 ? RUN : RUN == kTile ? 4 : 8)
        for (int k = k0; k < k0 + RUN; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(A + k * kTilePitch + ty * 4);
            const float av[4] = {a.x, a.y, a.z, a.w};
            float b[W];
            // W >= 4: columns 4 tx .. of each run of 64, so that a warp's vectors are contiguous
            if constexpr (W >= 4) {
#pragma unroll
                for (int g = 0; g < W / 4; ++g) {
                    const float4 x = *reinterpret_cast<const float4*>(B + k * (C + 4) + g * 64 + tx * 4);
                    b[4 * g] = x.x; b[4 * g + 1] = x.y; b[4 * g + 2] = x.z; b[4 * g + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < W; ++c) b[c] = B[k * (C + 4) + W * tx + c];
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!open(k, ty * 4 + r)) continue;
#pragma unroll
                for (int c = 0; c < W; ++c) to[r][c] = fmaf(av[r], b[c], to[r][c]);
            }
        }
    };
    if constexpr (RUN == kTile) {
        add_terms(acc, 0);
    } else {
        float tile[4][W] = {};
#pragma unroll 1
        for (int k0 = 0; k0 < kTile; k0 += RUN) {
            float part[4][W] = {};
            add_terms(part, k0);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < W; ++c) tile[r][c] += part[r][c];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < W; ++c) acc[r][c] += tile[r][c];
    }
}
// column of accumulator entry c of tile_rows_product
template <int W> __device__ __forceinline__ int tile_col(int c) { return W >= 4 ? (c / 4) * 64 + static_cast<int>(threadIdx.x & 15) * 4 + c % 4 : W * static_cast<int>(threadIdx.x & 15) + c; }
__host__ __device__ constexpr int tile_width(int C) { return C >= 16 ? C / 16 : 1; }

// over the 16 threads of a row
__device__ __forceinline__ float row_max16(float v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float row_sum16(float v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// X[c][r] = v: the transposed tile that the next product reads (thread's 4 x 4 block, 16-byte stores)
__device__ __forceinline__ void put_transposed(float* __restrict__ X, const float (&v)[4][4])
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<float4*>(X + (tx * 4 + c) * kTilePitch + ty * 4) = make_float4(v[0][c], v[1][c], v[2][c], v[3][c]);
}

}  // namespace nnb
