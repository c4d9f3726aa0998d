// Engine primitives the reference CudaEngine leaves unimplemented (cuda_engine.hpp:213-261, 461-469),
// in the reference's own layouts, fp32: the five fused two-pass attention primitives, the two fused
// cross-entropy primitives and the ExprSpec interpreter.  They make the unchanged reference Layer /
// Loss code run on the GPU one primitive at a time (the strict drop-in); the fused training step in
// gpt_step.cu is the fast path.  Semantics follow the CPU engine line by line:
//   batched_matmul_reduce / _softmax_denom / _softmax_apply / _softmax_backward_q / _kv
//                                   cpu_engine.hpp:426-915
//   col_softmax_denom / col_softmax_sparse_forward          cpu_engine.hpp:922-1006
//   eval_expr / eval_expr_reduce                            cpu_engine.hpp:1298-1659
#include <algorithm>

#include "kernels.h"
#include "nnb200.h"
#include "simt_tile.cuh"

namespace nnb {

// The five attention primitives work on 64 x 64 tiles of the scores (simt_tile.cuh); a block owns a tile row (or column,
// for the key / value gradients) of one batch entry and walks the tiles of the other index, leaving out tiles whose mask is
// -inf throughout (half of them under a causal mask).  The score product is done again in every
// primitive, because each is a call of its own that gets no scores.  At 48 x 256 x 256 x 64 (causal) the chain of six calls takes
// 333 us, and took 2572 us with one warp per row and a dot product per score.  What bounds it is latency: staging by scalar
// loads, two barriers and a product with no load in flight per tile, and 192 blocks of unequal length on 148 SMs; the 2.5 GFLOP
// are about 8 of the fp32 pipe's 70 TFLOP/s.
struct BmmDims {
    int batch, M, N, K, transA, transB;
    float alpha;
};
// one operand of the scores: element (index, k) of batch entry b, as the CPU engine indexes it (cpu_engine.hpp:452-469)
struct BmmSide {
    const float* p;
    int n;                        // extent of the index
    long long si, sk;
};
__device__ __forceinline__ BmmSide side_a(const float* A, const BmmDims& d, int b)
{
    const float* p = A + static_cast<size_t>(b) * d.M * d.K;
    return d.transA ? BmmSide{p, d.M, 1, d.M} : BmmSide{p, d.M, d.K, 1};
}
__device__ __forceinline__ BmmSide side_b(const float* B, const BmmDims& d, int b)
{
    const float* p = B + static_cast<size_t>(b) * d.K * d.N;
    return d.transB ? BmmSide{p, d.N, d.K, 1} : BmmSide{p, d.N, 1, d.N};
}
__device__ __forceinline__ float combine(int op, float acc, float v) { return op == 1 ? fmaxf(acc, v) : (op == 2 ? fminf(acc, v) : acc + v); }

// s[r][c] = X(i0 + 4 ty + r) . Y(j0 + 4 tx + c).  `keep`: 0 stage both, 1 X is staged already, 2 Y is (operands of one chunk)
template <int KC>
__device__ __forceinline__ void score_tile(float (&s)[4][4], const BmmSide& X, const BmmSide& Y, int i0, int j0, int K, float* Xs, float* Ys, int keep)
{
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[r][c] = 0.f;
    for (int k = 0; k < K; k += KC) {
        __syncthreads();
        if (keep != 1 || K > KC) stage_tile<KC>(Xs, X.p, X.si, X.sk, i0, X.n, k, K);
        if (keep != 2 || K > KC) stage_tile<KC>(Ys, Y.p, Y.si, Y.sk, j0, Y.n, k, K);
        __syncthreads();
        tile_product<KC>(s, Xs, Ys);
    }
}
// the mask of a thread's 4 x 4 scores (0 without a mask, -inf outside the matrix); false when the whole tile is -inf
__device__ __forceinline__ bool mask_tile(float (&mv)[4][4], const float* __restrict__ mask, int i0, int ni, int j0, int nj, long long si, long long sj)
{
    const int i = i0 + (threadIdx.x >> 4) * 4, j = j0 + (threadIdx.x & 15) * 4;
    bool any = false;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            mv[r][c] = (i + r < ni && j + c < nj) ? (mask ? mask[(i + r) * si + (j + c) * sj] : 0.f) : -INFINITY;
            any = any || mv[r][c] != -INFINITY;
        }
    return !mask || __syncthreads_or(any);
}

// op 0 Sum, 1 Max, 2 Min of the scores over one index; DENOM: sum of exp(score - row_max) instead
template <int KC, bool DENOM>
__global__ void __launch_bounds__(256) bmm_reduce_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ row_max,
                                                         const float* __restrict__ mask, float* __restrict__ out, BmmDims d, int op, int reduce_cols)
{
    __shared__ __align__(16) float Xs[KC * kTilePitch], Ys[KC * kTilePitch];
    const int outer = reduce_cols ? d.M : d.N, inner = reduce_cols ? d.N : d.M;
    const int tiles = static_cast<int>(ceil_div(outer, kTile)), b = blockIdx.x / tiles, i0 = (blockIdx.x - b * tiles) * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const BmmSide X = reduce_cols ? side_a(A, d, b) : side_b(B, d, b), Y = reduce_cols ? side_b(B, d, b) : side_a(A, d, b);
    const long long mi = reduce_cols ? d.N : 1, mj = reduce_cols ? 1 : d.N;
    const float init = DENOM ? 0.f : (op == 1 ? -3.402823466e38f : (op == 2 ? 3.402823466e38f : 0.f));   // lowest() / max() / 0
    float acc[4], mx[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        acc[r] = init;
        mx[r] = (DENOM && i0 + ty * 4 + r < outer) ? row_max[static_cast<size_t>(b) * outer + i0 + ty * 4 + r] : 0.f;
    }
    int keep = 0;
    for (int j0 = 0; j0 < inner; j0 += kTile) {
        float mv[4][4], s[4][4];
        if (!mask_tile(mv, mask, i0, outer, j0, inner, mi, mj)) continue;
        score_tile<KC>(s, X, Y, i0, j0, d.K, Xs, Ys, keep);
        keep = 1;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float part = init;                                    // of the tile: a chain over all tiles has one addition for each
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (mv[r][c] == -INFINITY) continue;              // masked entries: skipped for Sum and Min, no effect on Max
                const float v = d.alpha * s[r][c] + mv[r][c];
                part = DENOM ? part + expf(v - mx[r]) : combine(op, part, v);
            }
            acc[r] = combine(DENOM ? 0 : op, acc[r], part);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float v = acc[r];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v = combine(DENOM ? 0 : op, v, __shfl_xor_sync(0xffffffffu, v, o));
        if (tx == 0 && i0 + ty * 4 + r < outer) out[static_cast<size_t>(b) * outer + i0 + ty * 4 + r] = v;
    }
}

// softmax weight: exp(alpha*s + mask - m_i) / l_i, zero where the mask is -inf
__device__ __forceinline__ float softmax_weight(float s, float mv, float alpha, float mx, float inv_l)
{
    return mv == -INFINITY ? 0.f : expf(alpha * s + mv - mx) * inv_l;
}

// O[(b*M+i)*D + c] = sum_j W_ij V[(b*N+j)*D + c], C columns per walk over the keys
template <int KC, int C>
__global__ void __launch_bounds__(256) bmm_apply_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ V,
                                                        const float* __restrict__ row_max, const float* __restrict__ denom,
                                                        const float* __restrict__ mask, float* __restrict__ out, BmmDims d, int D)
{
    extern __shared__ __align__(16) float sm[];
    float *Xs = sm, *Ys = Xs + KC * kTilePitch, *Ps = Ys + KC * kTilePitch, *Vs = Ps + kTileFloats;
    constexpr int W = tile_width(C);
    const int tiles = static_cast<int>(ceil_div(d.M, kTile)), b = blockIdx.x / tiles, i0 = (blockIdx.x - b * tiles) * kTile;
    const int ty = threadIdx.x >> 4;
    const BmmSide X = side_a(A, d, b), Y = side_b(B, d, b);
    float mx[4], inv_l[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        mx[r] = i < d.M ? row_max[static_cast<size_t>(b) * d.M + i] : 0.f;
        inv_l[r] = i < d.M ? 1.0f / denom[static_cast<size_t>(b) * d.M + i] : 0.f;
    }
    int keep = 0;
    for (int c0 = 0; c0 < D; c0 += C) {
        float acc[4][W];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < W; ++c) acc[r][c] = 0.f;
        for (int j0 = 0; j0 < d.N; j0 += kTile) {
            float mv[4][4], s[4][4];
            if (!mask_tile(mv, mask, i0, d.M, j0, d.N, d.N, 1)) continue;
            score_tile<KC>(s, X, Y, i0, j0, d.K, Xs, Ys, keep);
            keep = 1;
            stage_rows<C>(Vs, V + static_cast<size_t>(b) * d.N * D, D, 1, j0, d.N, c0, D);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[r][c] = softmax_weight(s[r][c], mv[r][c], d.alpha, mx[r], inv_l[r]);
            put_transposed(Ps, s);
            __syncthreads();
            tile_rows_product<W, C>(acc, Ps, Vs);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = i0 + ty * 4 + r;
#pragma unroll
            for (int c = 0; c < W; ++c)
                if (i < d.M && tile_col<W>(c) < C && c0 + tile_col<W>(c) < D) out[(static_cast<size_t>(b) * d.M + i) * D + c0 + tile_col<W>(c)] = acc[r][c];
        }
    }
}

// a thread's 4 x 4 of the (M, N) gradient w.r.t. the weights, zero outside
__device__ __forceinline__ void load_p(float (&pv)[4][4], const float* __restrict__ P, int i0, int M, int j0, int N)
{
    const int i = i0 + (threadIdx.x >> 4) * 4, j = j0 + (threadIdx.x & 15) * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) pv[r][c] = (i + r < M && j + c < N) ? P[static_cast<size_t>(i + r) * N + j + c] : 0.f;
}

// R_i = sum_j W_ij P_ij ; gradQ[(b*K+k)*M + i] = alpha * sum_j W_ij (P_ij - R_i) B_b(k, j), KT tiles of 64 k per walk
template <int KC, int KT>
__global__ void __launch_bounds__(256) bmm_backward_q_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ P,
                                                             const float* __restrict__ row_max, const float* __restrict__ denom,
                                                             const float* __restrict__ mask, float* __restrict__ grad_q, float* __restrict__ r_out,
                                                             BmmDims d)
{
    extern __shared__ __align__(16) float sm[];
    float *Xs = sm, *Ys = Xs + KC * kTilePitch, *Ts = Ys + KC * kTilePitch, *Bs = Ts + kTileFloats;      // Bs: KT tiles
    const int tiles = static_cast<int>(ceil_div(d.M, kTile)), b = blockIdx.x / tiles, i0 = (blockIdx.x - b * tiles) * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const BmmSide X = side_a(A, d, b), Y = side_b(B, d, b);
    const float* Pb = P + static_cast<size_t>(b) * d.M * d.N;
    float mx[4], inv_l[4], R[4] = {};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        mx[r] = i < d.M ? row_max[static_cast<size_t>(b) * d.M + i] : 0.f;
        inv_l[r] = i < d.M ? 1.0f / denom[static_cast<size_t>(b) * d.M + i] : 0.f;
    }
    int keep = 0;
    for (int j0 = 0; j0 < d.N; j0 += kTile) {
        float mv[4][4], s[4][4], pv[4][4];
        if (!mask_tile(mv, mask, i0, d.M, j0, d.N, d.N, 1)) continue;
        load_p(pv, Pb, i0, d.M, j0, d.N);
        score_tile<KC>(s, X, Y, i0, j0, d.K, Xs, Ys, keep);
        keep = 1;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float part = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) part += softmax_weight(s[r][c], mv[r][c], d.alpha, mx[r], inv_l[r]) * pv[r][c];
            R[r] += part;
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        R[r] = row_sum16(R[r]);
        if (tx == 0 && i0 + ty * 4 + r < d.M) r_out[static_cast<size_t>(b) * d.M + i0 + ty * 4 + r] = R[r];
    }
    for (int k0 = 0; k0 < d.K; k0 += KT * kTile) {
        float acc[KT][4][4] = {};                                 // rows k, columns i
        for (int j0 = 0; j0 < d.N; j0 += kTile) {
            float mv[4][4], s[4][4], pv[4][4];
            if (!mask_tile(mv, mask, i0, d.M, j0, d.N, d.N, 1)) continue;
            load_p(pv, Pb, i0, d.M, j0, d.N);
            score_tile<KC>(s, X, Y, i0, j0, d.K, Xs, Ys, keep);
#pragma unroll
            for (int t = 0; t < KT; ++t) stage_rows<kTile>(Bs + t * kTileFloats, Y.p, Y.si, Y.sk, j0, d.N, k0 + t * kTile, d.K);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[r][c] = softmax_weight(s[r][c], mv[r][c], d.alpha, mx[r], inv_l[r]) * (pv[r][c] - R[r]);
            put_transposed(Ts, s);
            __syncthreads();
#pragma unroll
            for (int t = 0; t < KT; ++t) tile_rows_product<4, kTile>(acc[t], Bs + t * kTileFloats, Ts);
        }
#pragma unroll
        for (int t = 0; t < KT; ++t)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int k = k0 + t * kTile + ty * 4 + r;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (k < d.K && i0 + tx * 4 + c < d.M) grad_q[(static_cast<size_t>(b) * d.K + k) * d.M + i0 + tx * 4 + c] = d.alpha * acc[t][r][c];
            }
    }
}

// gradK[(b*K+k)*N + j] = alpha * sum_i W_ij (P_ij - R_i) A_b(i, k) ; gradV[(b*K+k)*N + j] = sum_i W_ij G[(b*M+i)*D + k]
// (the reference sizes gradV by K and reads the first K columns of G, cpu_engine.hpp:870-908)
template <int KC>
__global__ void __launch_bounds__(256) bmm_backward_kv_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ P,
                                                              const float* __restrict__ G, const float* __restrict__ R,
                                                              const float* __restrict__ row_max, const float* __restrict__ denom,
                                                              const float* __restrict__ mask, float* __restrict__ grad_k, float* __restrict__ grad_v,
                                                              BmmDims d, int D)
{
    extern __shared__ __align__(16) float sm[];
    float *Xs = sm, *Ys = Xs + KC * kTilePitch, *Ws = Ys + KC * kTilePitch, *Ts = Ws + kTileFloats, *As = Ts + kTileFloats, *Gs = As + kTileFloats;
    const int tiles = static_cast<int>(ceil_div(d.N, kTile)), b = blockIdx.x / tiles, j0 = (blockIdx.x - b * tiles) * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const BmmSide X = side_a(A, d, b), Y = side_b(B, d, b);
    const float* Pb = P + static_cast<size_t>(b) * d.M * d.N;
    const size_t row0 = static_cast<size_t>(b) * d.M;
    int keep = 0;
    for (int k0 = 0; k0 < d.K; k0 += kTile) {
        float ak[4][4] = {}, av[4][4] = {};                       // rows k, columns j
        for (int i0 = 0; i0 < d.M; i0 += kTile) {
            float mv[4][4], s[4][4], pv[4][4], t[4][4];
            if (!mask_tile(mv, mask, i0, d.M, j0, d.N, d.N, 1)) continue;
            load_p(pv, Pb, i0, d.M, j0, d.N);
            score_tile<KC>(s, X, Y, i0, j0, d.K, Xs, Ys, keep);
            keep = 2;
            stage_rows<kTile>(As, X.p, X.si, X.sk, i0, d.M, k0, d.K);
            stage_rows<kTile>(Gs, G + row0 * D, D, 1, i0, d.M, k0, d.K);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = i0 + ty * 4 + r;
                const float mx = i < d.M ? row_max[row0 + i] : 0.f, inv_l = i < d.M ? 1.0f / denom[row0 + i] : 0.f, Ri = i < d.M ? R[row0 + i] : 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[r][c] = softmax_weight(s[r][c], mv[r][c], d.alpha, mx, inv_l);
                    t[r][c] = s[r][c] * (pv[r][c] - Ri);
                }
                *reinterpret_cast<float4*>(Ws + (ty * 4 + r) * kTilePitch + tx * 4) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
                *reinterpret_cast<float4*>(Ts + (ty * 4 + r) * kTilePitch + tx * 4) = make_float4(t[r][0], t[r][1], t[r][2], t[r][3]);
            }
            __syncthreads();
            tile_rows_product<4, kTile>(ak, As, Ts);
            tile_rows_product<4, kTile>(av, Gs, Ws);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = k0 + ty * 4 + r;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (k < d.K && j0 + tx * 4 + c < d.N) {
                    const size_t o = (static_cast<size_t>(b) * d.K + k) * d.N + j0 + tx * 4 + c;
                    grad_k[o] = d.alpha * ak[r][c];
                    grad_v[o] = av[r][c];
                }
        }
    }
}

// ---------------------------------------------------------------- cross-entropy, (classes, tokens) layout
// a block owns 32 token columns; 8 row lanes walk the classes, so every access is a coalesced 128-byte row piece
__global__ void __launch_bounds__(256)
col_softmax_denom_kernel(const float* __restrict__ logits, const float* __restrict__ col_max, float* __restrict__ out, int C, int N)
{
    __shared__ float red[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, n = blockIdx.x * 32 + tx;
    float acc = 0.f;
    if (n < N) { const float mx = col_max[n]; for (int r = ty; r < C; r += 8) acc += expf(logits[static_cast<size_t>(r) * N + n] - mx); }
    red[ty][tx] = acc;
    __syncthreads();
    if (ty == 0 && n < N) { for (int k = 1; k < 8; ++k) acc += red[k][tx]; out[n] = acc; }
}

__global__ void __launch_bounds__(256)
col_softmax_sparse_kernel(const float* __restrict__ logits, const float* __restrict__ labels, const float* __restrict__ mask,
                          float* __restrict__ grad, float* __restrict__ loss_vec, int C, int N, int vocab, float inv_nv)
{
    __shared__ float red[8][33];
    __shared__ float smax[32], sden[32];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, n = blockIdx.x * 32 + tx;
    const bool in = n < N;
    const float lf = in ? labels[n] : 0.f;
    const long long lbl = lf >= 0.f ? static_cast<long long>(lf) : 0;
    const bool valid = in && (!mask || mask[n] >= 0.5f) && lbl < vocab;
    float mx = -INFINITY;
    if (valid) for (int r = ty; r < C; r += 8) mx = fmaxf(mx, logits[static_cast<size_t>(r) * N + n]);
    red[ty][tx] = mx;
    __syncthreads();
    if (ty == 0) { for (int k = 1; k < 8; ++k) mx = fmaxf(mx, red[k][tx]); smax[tx] = mx; }
    __syncthreads();
    mx = smax[tx];
    float den = 0.f;
    if (valid) for (int r = ty; r < C; r += 8) den += expf(logits[static_cast<size_t>(r) * N + n] - mx);
    __syncthreads();
    red[ty][tx] = den;
    __syncthreads();
    if (ty == 0) { for (int k = 1; k < 8; ++k) den += red[k][tx]; sden[tx] = den; }
    __syncthreads();
    den = sden[tx];
    if (in) {
        for (int r = ty; r < C; r += 8) {
            float g = 0.f;
            if (valid) { g = inv_nv * expf(logits[static_cast<size_t>(r) * N + n] - mx) / den; if (r == lbl) g -= inv_nv; }
            grad[static_cast<size_t>(r) * N + n] = g;
        }
        if (ty == 0) loss_vec[n] = valid ? logits[static_cast<size_t>(lbl) * N + n] - mx - logf(den) : 0.f;
    }
}

static int check_bmm(const BmmDims& d)
{
    return (d.batch > 0 && d.M > 0 && d.N > 0 && d.K > 0 && ceil_div(std::max(d.M, d.N), kTile) * d.batch <= INT_MAX) ? 0 : -1;
}
static unsigned bmm_blocks(const BmmDims& d, int n) { return static_cast<unsigned>(ceil_div(n, kTile) * d.batch); }
// launch with more than the default shared memory; Kernel: one instantiation, so that each opts in once per device
template <auto Kernel, typename... Args> static int bmm_launch(unsigned blocks, size_t smem, cudaStream_t s, Args... args)
{
    static PerDeviceOnce once;
    NNB_TRY(once.run([smem] { return cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)); }));
    Kernel<<<blocks, 256, smem, s>>>(args...);
    NNB_LAUNCH_CHECK();
    return 0;
}
template <int KC> static int bmm_apply(const float* A, const float* B, const float* V, const float* row_max, const float* denom, const float* mask,
                                       float* out, const BmmDims& d, int D, cudaStream_t s)
{
    // columns of O per walk: as many as D has, up to 128 (every further walk repeats the scores)
    const size_t base = (2 * KC * kTilePitch + kTileFloats) * sizeof(float);
    if (D <= 32) return bmm_launch<bmm_apply_kernel<KC, 32>>(bmm_blocks(d, d.M), base + kTile * 36 * sizeof(float), s, A, B, V, row_max, denom, mask, out, d, D);
    if (D <= 64) return bmm_launch<bmm_apply_kernel<KC, 64>>(bmm_blocks(d, d.M), base + kTile * 68 * sizeof(float), s, A, B, V, row_max, denom, mask, out, d, D);
    return bmm_launch<bmm_apply_kernel<KC, 128>>(bmm_blocks(d, d.M), base + kTile * 132 * sizeof(float), s, A, B, V, row_max, denom, mask, out, d, D);
}

}  // namespace nnb

using namespace nnb;

extern "C" {

int nnb200_batched_matmul(const float* A, const float* B, float* C, size_t A_rows, size_t A_cols, size_t B_rows, size_t B_cols,
                          unsigned int batch, int transA, int transB, float alpha, void* stream)
{
    if (batch == 0 || A_rows % batch || B_rows % batch) return -1;
    const long long a_rpb = A_rows / batch, b_rpb = B_rows / batch;
    const long long M = transA ? A_cols : a_rpb, K = transA ? a_rpb : A_cols;
    const long long K2 = transB ? B_cols : b_rpb, N = transB ? b_rpb : B_cols;
    if (K != K2) return -1;
    for (unsigned b0 = 0; b0 < batch; b0 += 65535) {
        const unsigned nb = batch - b0 < 65535 ? batch - b0 : 65535;
        NNB_TRY(sgemm_strided(A + b0 * a_rpb * A_cols, B + b0 * b_rpb * B_cols, C + b0 * M * N, static_cast<int>(M),
                              static_cast<int>(N), static_cast<int>(K), transA ? 1 : static_cast<long long>(A_cols),
                              transA ? static_cast<long long>(A_cols) : 1, transB ? static_cast<long long>(B_cols) : 1,
                              transB ? 1 : static_cast<long long>(B_cols), N, static_cast<int>(nb), a_rpb * A_cols,
                              b_rpb * B_cols, M * N, alpha, nullptr, nullptr, nullptr, 0, to_stream(stream)));
    }
    return 0;
}

int nnb200_bmm_reduce(const float* A, const float* B, const float* mask, float* out, int batch, int M, int N, int K, int op,
                      int transA, int transB, float alpha, int reduce_cols, void* stream)
{
    const BmmDims d{batch, M, N, K, transA, transB, alpha};
    if (check_bmm(d) || op < 0 || op > 2) return -1;
    const unsigned blocks = bmm_blocks(d, reduce_cols ? M : N);
    if (K <= 32) bmm_reduce_kernel<32, false><<<blocks, 256, 0, to_stream(stream)>>>(A, B, nullptr, mask, out, d, op, reduce_cols);
    else bmm_reduce_kernel<64, false><<<blocks, 256, 0, to_stream(stream)>>>(A, B, nullptr, mask, out, d, op, reduce_cols);
    NNB_LAUNCH_CHECK();
    return 0;
}

int nnb200_bmm_softmax_denom(const float* A, const float* B, const float* row_max, const float* mask, float* out, int batch,
                             int M, int N, int K, int transA, int transB, float alpha, void* stream)
{
    const BmmDims d{batch, M, N, K, transA, transB, alpha};
    if (check_bmm(d)) return -1;
    if (K <= 32) bmm_reduce_kernel<32, true><<<bmm_blocks(d, M), 256, 0, to_stream(stream)>>>(A, B, row_max, mask, out, d, 0, 1);
    else bmm_reduce_kernel<64, true><<<bmm_blocks(d, M), 256, 0, to_stream(stream)>>>(A, B, row_max, mask, out, d, 0, 1);
    NNB_LAUNCH_CHECK();
    return 0;
}

int nnb200_bmm_softmax_apply(const float* A, const float* B, const float* V, const float* row_max, const float* denom,
                             const float* mask, float* out, int batch, int M, int N, int K, int D, int transA, int transB,
                             float alpha, void* stream)
{
    const BmmDims d{batch, M, N, K, transA, transB, alpha};
    if (check_bmm(d) || D <= 0) return -1;
    return K <= 32 ? bmm_apply<32>(A, B, V, row_max, denom, mask, out, d, D, to_stream(stream)) : bmm_apply<64>(A, B, V, row_max, denom, mask, out, d, D, to_stream(stream));
}

int nnb200_bmm_softmax_backward_q(const float* A, const float* B, const float* P, const float* row_max, const float* denom,
                                  const float* mask, float* grad_q, float* r_out, int batch, int M, int N, int K, int transA,
                                  int transB, float alpha, void* stream)
{
    const BmmDims d{batch, M, N, K, transA, transB, alpha};
    if (check_bmm(d)) return -1;
    const unsigned blocks = bmm_blocks(d, M);
    cudaStream_t s = to_stream(stream);
    const size_t tile = kTileFloats * sizeof(float);
    if (K <= 32) return bmm_launch<bmm_backward_q_kernel<32, 1>>(blocks, 3 * tile, s, A, B, P, row_max, denom, mask, grad_q, r_out, d);
    if (K <= 64) return bmm_launch<bmm_backward_q_kernel<64, 1>>(blocks, 4 * tile, s, A, B, P, row_max, denom, mask, grad_q, r_out, d);
    return bmm_launch<bmm_backward_q_kernel<64, 2>>(blocks, 5 * tile, s, A, B, P, row_max, denom, mask, grad_q, r_out, d);
}

int nnb200_bmm_softmax_backward_kv(const float* A, const float* B, const float* P, const float* G, const float* R,
                                   const float* row_max, const float* denom, const float* mask, float* grad_k, float* grad_v,
                                   int batch, int M, int N, int K, int D, int transA, int transB, float alpha, void* stream)
{
    const BmmDims d{batch, M, N, K, transA, transB, alpha};
    if (check_bmm(d) || D < K) return -1;
    const size_t tile = kTileFloats * sizeof(float);
    if (K <= 32) return bmm_launch<bmm_backward_kv_kernel<32>>(bmm_blocks(d, N), 5 * tile, to_stream(stream), A, B, P, G, R, row_max, denom, mask, grad_k, grad_v, d, D);
    return bmm_launch<bmm_backward_kv_kernel<64>>(bmm_blocks(d, N), 6 * tile, to_stream(stream), A, B, P, G, R, row_max, denom, mask, grad_k, grad_v, d, D);
}

int nnb200_col_softmax_denom(const float* logits, const float* col_max, float* out, int classes, int tokens, void* stream)
{
    if (classes <= 0 || tokens <= 0) return -1;
    col_softmax_denom_kernel<<<static_cast<unsigned>(ceil_div(tokens, 32)), 256, 0, to_stream(stream)>>>(logits, col_max, out, classes, tokens);
    NNB_LAUNCH_CHECK();
    return 0;
}

int nnb200_col_softmax_sparse_forward(const float* logits, const float* labels, const float* mask, float* grad, float* loss_vec,
                                      int classes, int tokens, int vocab_size, float inv_num_valid, void* stream)
{
    if (classes <= 0 || tokens <= 0) return -1;
    if (vocab_size > classes) { fprintf(stderr, "nnb200_col_softmax_sparse_forward: vocab_size > classes\n"); return -1; }
    col_softmax_sparse_kernel<<<static_cast<unsigned>(ceil_div(tokens, 32)), 256, 0, to_stream(stream)>>>(logits, labels, mask, grad, loss_vec, classes, tokens, vocab_size, inv_num_valid);
    NNB_LAUNCH_CHECK();
    return 0;
}

}  // extern "C"
