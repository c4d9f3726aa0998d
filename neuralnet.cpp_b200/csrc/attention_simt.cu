// Fused causal / document-masked / ALiBi attention, SIMT fp32-accumulate version.
//
// This is the check-mode path (fp32 in, fp32 math) and the path for head sizes the tensor-core
// kernel does not tile.  It computes exactly what AttentionBase::forward/backward compute
// (compute_layer.hpp:1133-1412) with the mask of build_attention_mask (:2081-2128):
//   s_ij = q_i.k_j / sqrt(dk) - slope_h*(i-j)   where j <= i and doc_i == doc_j, else -inf
//   O_i = sum_j softmax_j(s_ij) v_j
// without materialising the (B*H*S, S) score, mask and probability matrices.
// Layout: qkv is (tokens, 3*d) row-major, q | k | v side by side, head h at columns h*dk.. of each;
// out / dout are (tokens, d); lse and dvec are (B*H*S) with index (b*H + h)*S + i.
#include "kernels.h"
#include "simt_tile.cuh"

namespace nnb {

__device__ __forceinline__ float alibi_slope(int h, int H)
{
    // m_h = 2^(-8h/H), h from 0 (compute_layer.hpp:2179-2187)
    return powf(2.0f, -8.0f * static_cast<float>(h) / static_cast<float>(H));
}

// dvec[row] = sum_c dout[i][h*dk+c] * out[i][h*dk+c]  (= R_i = sum_j W_ij P_ij of the reference's
// backward_q primitive, cpu_engine.hpp:767-783)
template <typename T>
__global__ void attn_dvec_kernel(const T* __restrict__ out, const T* __restrict__ dout, float* __restrict__ dvec,
                                 int B, int S, int H, int dk)
{
    const int lane = threadIdx.x & 31;
    const long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (row >= static_cast<long long>(B) * H * S) return;
    const int i = static_cast<int>(row % S), h = static_cast<int>((row / S) % H), b = static_cast<int>(row / S / H);
    const size_t off = (static_cast<size_t>(b) * S + i) * (H * dk) + h * dk;
    float s = 0.f;
    for (int c = lane; c < dk; c += 32) s += to_f32(out[off + c]) * to_f32(dout[off + c]);
    s = warp_sum(s);
    if (lane == 0) dvec[row] = s;
}

// Vectorised variant: a warp walks a whole token row (all heads) with 16-byte loads; the lanes that
// share a head fold their partial dot products with shuffles.  Needs dk a multiple of the vector
// width with dk/width a power of two <= 32.
template <typename T>
__global__ void __launch_bounds__(256)
attn_dvec_vec_kernel(const T* __restrict__ out, const T* __restrict__ dout, float* __restrict__ dvec, int B, int S,
                     int H, int dk)
{
    constexpr int VN = Vec16<T>::N;
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int d = H * dk, nvec = d / VN, L = dk / VN;
    const int nvec_pad = (nvec + 31) & ~31;
    const long long ntok = static_cast<long long>(B) * S;
    for (long long t = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); t < ntok; t += static_cast<long long>(gridDim.x) * wpb) {
        const int b = static_cast<int>(t / S), i = static_cast<int>(t % S);
        for (int v = lane; v < nvec_pad; v += 32) {
            float sacc = 0.f;
            if (v < nvec) {
                const Vec16<T> ov = ld16(out + t * d + v * VN), gv = ld16(dout + t * d + v * VN);
#pragma unroll
                for (int k = 0; k < VN; ++k) sacc += to_f32(ov.v[k]) * to_f32(gv.v[k]);
            }
            for (int off = L >> 1; off > 0; off >>= 1) sacc += __shfl_xor_sync(0xffffffffu, sacc, off);
            if (v < nvec && (lane & (L - 1)) == 0) dvec[(static_cast<size_t>(b) * H + v / L) * S + i] = sacc;
        }
    }
}

template <typename T>
static int launch_dvec(const T* out, const T* dout, float* dvec, int B, int S, int H, int dk, cudaStream_t s)
{
    constexpr int VN = Vec16<T>::N;
    const long long rows = static_cast<long long>(B) * H * S;
    const int L = dk / VN;
    const bool vec = (dk % VN) == 0 && L >= 1 && L <= 32 && (L & (L - 1)) == 0 &&
                     ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0;
    if (vec) attn_dvec_vec_kernel<T><<<grid_for(static_cast<long long>(B) * S, 8), 256, 0, s>>>(out, dout, dvec, B, S, H, dk);
    else attn_dvec_kernel<T><<<static_cast<unsigned>(ceil_div(rows * 32, 256)), 256, 0, s>>>(out, dout, dvec, B, S, H, dk);
    NNB_LAUNCH_CHECK();
    return 0;
}

// ---- tiles of 64 queries x 64 keys; a block of 256 threads per tile row (forward, dQ) or tile column (dK, dV).
// What bounds them: the fp32 pipe at long sequences; at short ones (few blocks) the chain stage - product - exponential.
// 8 x 128 x 4 heads of 32, fp32: forward 15 us, dQ 14, dK / dV 18 (with one warp per row and lanes over the keys, whose loads
// were a row length apart: 123, 132, 179).
// Terms of a run in the sums over keys and queries (tile_rows_product).  Errors of out, dQ, dK, dV against float64, 2048 queries
// and keys, heads of 64 (units of 1e-7): runs of 8: 2.5, 3.8, 4.0, 3.4; one chain: 4.0, 5.2, 10.8, 11.1; a warp per row with its
// lanes over the other index: 2.4, 3.7, 4.1, 3.6.  8 x 512 x 6 heads of 64, gradients: 304 us as one chain, 303 in runs.
// bf16 results are rounded a thousand times coarser: one chain.
template <typename T> constexpr int kRun = sizeof(T) == 4 ? 8 : kTile;
template <int DK> struct SimtDims {
    static constexpr int KC = DK < 64 ? DK : 64, W = tile_width(DK), ROWS = kTile * (DK + 4);
};

// score of (i, j) after scale and ALiBi, -inf where the mask leaves nothing
struct ScoreMask {
    const int* doc;          // this sequence's document ids, or null
    int S;
    float scale, slope;
    __device__ __forceinline__ bool open(int i, int j) const { return j <= i && i < S && (!doc || doc[j] == doc[i]); }
    __device__ __forceinline__ float score(float s, int i, int j) const { return scale * s - slope * static_cast<float>(i - j); }
};

// is anything of the 64 x 64 tile at (i0, j0) open?  Only document masks close tiles on or below the diagonal.
__device__ __forceinline__ bool tile_open(const ScoreMask& mk, int i0, int j0)
{
    if (!mk.doc) return true;
    bool any = false;
    const int i = i0 + (threadIdx.x & 63);
    for (int u = threadIdx.x >> 6; u < kTile; u += 4) any = any || mk.open(i, j0 + u);
    return __syncthreads_or(any);
}

// A closed pair has weight 0, which takes it out of the sums as long as what it multiplies is finite.  So each block looks at
// its results when it is done: one that is infinite or NaN may come of a closed pair, and the block starts again with the
// guarded form, which adds open pairs only.  An infinite or NaN row thus reaches the positions that see it and no others,
// whose results are the same bits either way.  (Looking at the staged rows of every tile instead cost 3 to 9 % of the forward.)
template <int W> __device__ __forceinline__ bool not_finite(const float (&v)[4][W], int row0, int rows, int cols)
{
    bool bad = false;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < W; ++c) bad = bad || (row0 + r < rows && tile_col<W>(c) < cols && !isfinite(v[r][c]));
    return bad;
}

// Queries are rows q0 .. S - 1 of a sequence of S keys (q0 = 0 in training; a prompt pass continues behind q0 cached rows), so
// q and out point at the row of query q0; `lse` may be null.  True, with nothing written: to be done again, guarded.
template <typename T, int DK, bool GUARD>
__device__ __forceinline__ bool attn_fwd_block(float* sm, const T* __restrict__ q, long long ldq, const T* __restrict__ kc, const T* __restrict__ vc,
                                               long long ldk, T* __restrict__ out, float* __restrict__ lse, const int* __restrict__ doc,
                                               int B, int S, int q0, int H, int alibi, float scale)
{
    using D = SimtDims<DK>;
    float *Qs = sm, *Ks = Qs + DK * kTilePitch, *Vs = Ks + DK * kTilePitch, *Ps = Vs + D::ROWS;
    const int nq = S - q0;
    const int bh = blockIdx.x % (B * H), qt = static_cast<int>(ceil_div(nq, kTile)) - 1 - blockIdx.x / (B * H), h = bh % H, b = bh / H;   // long rows first
    const int d = H * DK, i0 = q0 + qt * kTile, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const T* qb = q + static_cast<size_t>(b) * nq * ldq + h * DK;
    const T* kb = kc + static_cast<size_t>(b) * S * ldk + h * DK;
    const T* vb = vc + static_cast<size_t>(b) * S * ldk + h * DK;
    const ScoreMask mk{doc ? doc + static_cast<size_t>(b) * S : nullptr, S, scale, alibi ? alibi_slope(h, H) : 0.f};
    for (int k = 0; k < DK; k += D::KC) stage_tile<D::KC>(Qs + k * kTilePitch, qb, ldq, 1, i0 - q0, nq, k, DK);
    float m[4], l[4], o[4][D::W];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < D::W; ++c) o[r][c] = 0.f;
    }
    for (int j0 = 0; j0 < S && j0 < i0 + kTile; j0 += kTile) {
        if (!tile_open(mk, i0, j0)) continue;
        __syncthreads();
        for (int k = 0; k < DK; k += D::KC) stage_tile<D::KC>(Ks + k * kTilePitch, kb, ldk, 1, j0, S, k, DK);
        stage_rows<DK>(Vs, vb, ldk, 1, j0, S, 0, DK);
        __syncthreads();
        float s[4][4] = {};
        tile_product<DK>(s, Qs, Ks);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = i0 + ty * 4 + r;
            float mx = m[r];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = j0 + tx * 4 + c;
                s[r][c] = mk.open(i, j) ? mk.score(s[r][c], i, j) : -INFINITY;
                mx = fmaxf(mx, s[r][c]);
            }
            mx = row_max16(mx);
            const float ref = mx == -INFINITY ? 0.f : mx, back = expf(m[r] - ref);
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) { s[r][c] = expf(s[r][c] - ref); sum += s[r][c]; }
            l[r] = l[r] * back + row_sum16(sum);
            m[r] = mx;
#pragma unroll
            for (int c = 0; c < D::W; ++c) o[r][c] *= back;
        }
        put_transposed(Ps, s);
        __syncthreads();
        if constexpr (GUARD) tile_rows_product<D::W, DK, kRun<T>>(o, Ps, Vs, [&](int k, int r) { return mk.open(i0 + r, j0 + k); });
        else tile_rows_product<D::W, DK, kRun<T>>(o, Ps, Vs);
    }
    if (!GUARD && __syncthreads_or(not_finite(o, i0 + ty * 4, S, DK))) return true;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        if (i >= S) continue;
        const float inv = 1.0f / l[r];
        T* op = out + (static_cast<size_t>(b) * nq + i - q0) * d + h * DK;
#pragma unroll
        for (int c = 0; c < D::W; ++c)
            if (tile_col<D::W>(c) < DK) op[tile_col<D::W>(c)] = from_f32<T>(o[r][c] * inv);
        if (tx == 0 && lse) lse[(static_cast<size_t>(b) * H + h) * S + i] = m[r] + logf(l[r]);
    }
    return false;
}
template <typename T, int DK>
__device__ __noinline__ void attn_fwd_guarded(float* sm, const T* q, long long ldq, const T* kc, const T* vc, long long ldk, T* out, float* lse,
                                              const int* doc, int B, int S, int q0, int H, int alibi, float scale)
{
    attn_fwd_block<T, DK, true>(sm, q, ldq, kc, vc, ldk, out, lse, doc, B, S, q0, H, alibi, scale);
}
template <typename T, int DK>
__global__ void __launch_bounds__(256) attn_fwd_simt_kernel(const T* __restrict__ q, long long ldq, const T* __restrict__ kc, const T* __restrict__ vc,
                                                            long long ldk, T* __restrict__ out, float* __restrict__ lse, const int* __restrict__ doc,
                                                            int B, int S, int q0, int H, int alibi, float scale)
{
    extern __shared__ __align__(16) float sm[];
    if (attn_fwd_block<T, DK, false>(sm, q, ldq, kc, vc, ldk, out, lse, doc, B, S, q0, H, alibi, scale))
        attn_fwd_guarded<T, DK>(sm, q, ldq, kc, vc, ldk, out, lse, doc, B, S, q0, H, alibi, scale);
}

// dQ_i = scale sum_j P_ij (dP_ij - D_i) k_j
template <typename T, int DK, bool GUARD>
__device__ __forceinline__ bool attn_bwd_dq_block(float* sm, const T* __restrict__ qkv, const T* __restrict__ dout, const float* __restrict__ lse,
                                                  const float* __restrict__ dvec, T* __restrict__ dqkv, const int* __restrict__ doc,
                                                  int B, int S, int H, int alibi, float scale)
{
    using D = SimtDims<DK>;
    float *Qs = sm, *Gs = Qs + DK * kTilePitch, *Ks = Gs + DK * kTilePitch, *Vs = Ks + D::KC * kTilePitch, *Kr = Vs + D::KC * kTilePitch, *Ps = Kr + D::ROWS;
    const int bh = blockIdx.x % (B * H), qt = static_cast<int>(ceil_div(S, kTile)) - 1 - blockIdx.x / (B * H), h = bh % H, b = bh / H;
    const int d = H * DK, ld = 3 * d, i0 = qt * kTile, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const T* base = qkv + static_cast<size_t>(b) * S * ld + h * DK;
    const T* gbase = dout + static_cast<size_t>(b) * S * d + h * DK;
    const ScoreMask mk{doc ? doc + static_cast<size_t>(b) * S : nullptr, S, scale, alibi ? alibi_slope(h, H) : 0.f};
    const size_t row0 = (static_cast<size_t>(b) * H + h) * S;
    for (int k = 0; k < DK; k += D::KC) {
        stage_tile<D::KC>(Qs + k * kTilePitch, base, ld, 1, i0, S, k, DK);
        stage_tile<D::KC>(Gs + k * kTilePitch, gbase, d, 1, i0, S, k, DK);
    }
    float L[4], Dv[4], dq[4][D::W];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        L[r] = i < S ? lse[row0 + i] : 0.f;
        Dv[r] = i < S ? dvec[row0 + i] : 0.f;
#pragma unroll
        for (int c = 0; c < D::W; ++c) dq[r][c] = 0.f;
    }
    for (int j0 = 0; j0 <= i0; j0 += kTile) {
        if (!tile_open(mk, i0, j0)) continue;
        float s[4][4] = {}, dp[4][4] = {};
        for (int k = 0; k < DK; k += D::KC) {
            __syncthreads();
            stage_tile<D::KC>(Ks, base + d, ld, 1, j0, S, k, DK);
            stage_tile<D::KC>(Vs, base + 2 * d, ld, 1, j0, S, k, DK);
            if (k == 0) stage_rows<DK>(Kr, base + d, ld, 1, j0, S, 0, DK);
            __syncthreads();
            tile_product<D::KC>(s, Qs + k * kTilePitch, Ks);
            tile_product<D::KC>(dp, Gs + k * kTilePitch, Vs);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = i0 + ty * 4 + r;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = j0 + tx * 4 + c;
                s[r][c] = mk.open(i, j) ? expf(mk.score(s[r][c], i, j) - L[r]) * (dp[r][c] - Dv[r]) : 0.f;
            }
        }
        put_transposed(Ps, s);
        __syncthreads();
        if constexpr (GUARD) tile_rows_product<D::W, DK, kRun<T>>(dq, Ps, Kr, [&](int k, int r) { return mk.open(i0 + r, j0 + k); });
        else tile_rows_product<D::W, DK, kRun<T>>(dq, Ps, Kr);
    }
    if (!GUARD && __syncthreads_or(not_finite(dq, i0 + ty * 4, S, DK))) return true;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        if (i >= S) continue;
        T* p = dqkv + (static_cast<size_t>(b) * S + i) * ld + h * DK;
#pragma unroll
        for (int c = 0; c < D::W; ++c)
            if (tile_col<D::W>(c) < DK) p[tile_col<D::W>(c)] = from_f32<T>(scale * dq[r][c]);
    }
    return false;
}
template <typename T, int DK>
__device__ __noinline__ void attn_bwd_dq_guarded(float* sm, const T* qkv, const T* dout, const float* lse, const float* dvec, T* dqkv, const int* doc,
                                                 int B, int S, int H, int alibi, float scale)
{
    attn_bwd_dq_block<T, DK, true>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
}
template <typename T, int DK>
__global__ void __launch_bounds__(256) attn_bwd_dq_simt_kernel(const T* __restrict__ qkv, const T* __restrict__ dout, const float* __restrict__ lse,
                                                               const float* __restrict__ dvec, T* __restrict__ dqkv, const int* __restrict__ doc,
                                                               int B, int S, int H, int alibi, float scale)
{
    extern __shared__ __align__(16) float sm[];
    if (attn_bwd_dq_block<T, DK, false>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale))
        attn_bwd_dq_guarded<T, DK>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
}

// dK_j = scale sum_i P_ij (dP_ij - D_i) q_i ; dV_j = sum_i P_ij dO_i.  Rows of the tile are keys, columns queries.
template <typename T, int DK, bool GUARD>
__device__ __forceinline__ bool attn_bwd_dkv_block(float* sm, const T* __restrict__ qkv, const T* __restrict__ dout, const float* __restrict__ lse,
                                                   const float* __restrict__ dvec, T* __restrict__ dqkv, const int* __restrict__ doc,
                                                   int B, int S, int H, int alibi, float scale)
{
    using D = SimtDims<DK>;
    float *Ks = sm, *Vs = Ks + D::KC * kTilePitch, *Qs = Vs + D::KC * kTilePitch, *Gs = Qs + D::KC * kTilePitch, *Qr = Gs + D::KC * kTilePitch,
          *Gr = Qr + D::ROWS, *Ps = Gr + D::ROWS, *Ss = Ps + kTileFloats;
    const int bh = blockIdx.x % (B * H), kt = blockIdx.x / (B * H), h = bh % H, b = bh / H;      // the first keys are seen by the most queries
    const int d = H * DK, ld = 3 * d, j0 = kt * kTile, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const T* base = qkv + static_cast<size_t>(b) * S * ld + h * DK;
    const T* gbase = dout + static_cast<size_t>(b) * S * d + h * DK;
    const ScoreMask mk{doc ? doc + static_cast<size_t>(b) * S : nullptr, S, scale, alibi ? alibi_slope(h, H) : 0.f};
    const size_t row0 = (static_cast<size_t>(b) * H + h) * S;
    float dk[4][D::W], dv[4][D::W];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < D::W; ++c) { dk[r][c] = 0.f; dv[r][c] = 0.f; }
    for (int i0 = j0; i0 < S; i0 += kTile) {
        if (!tile_open(mk, i0, j0)) continue;
        float s[4][4] = {}, dp[4][4] = {};
        for (int k = 0; k < DK; k += D::KC) {
            __syncthreads();
            if (DK > D::KC || i0 == j0) {                        // one chunk: the keys stay (the diagonal tile is always open)
                stage_tile<D::KC>(Ks, base + d, ld, 1, j0, S, k, DK);
                stage_tile<D::KC>(Vs, base + 2 * d, ld, 1, j0, S, k, DK);
            }
            stage_tile<D::KC>(Qs, base, ld, 1, i0, S, k, DK);
            stage_tile<D::KC>(Gs, gbase, d, 1, i0, S, k, DK);
            if (k == 0) { stage_rows<DK>(Qr, base, ld, 1, i0, S, 0, DK); stage_rows<DK>(Gr, gbase, d, 1, i0, S, 0, DK); }
            __syncthreads();
            tile_product<D::KC>(s, Ks, Qs);
            tile_product<D::KC>(dp, Vs, Gs);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = i0 + tx * 4 + c;
            const float L = i < S ? lse[row0 + i] : 0.f, Dv = i < S ? dvec[row0 + i] : 0.f;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int j = j0 + ty * 4 + r;
                const float p = mk.open(i, j) ? expf(mk.score(s[r][c], i, j) - L) : 0.f;
                s[r][c] = p;
                dp[r][c] = p * (dp[r][c] - Dv);
            }
        }
        put_transposed(Ps, s);
        put_transposed(Ss, dp);
        __syncthreads();
        if constexpr (GUARD) {
            auto open = [&](int k, int r) { return mk.open(i0 + k, j0 + r); };
            tile_rows_product<D::W, DK, kRun<T>>(dv, Ps, Gr, open);
            tile_rows_product<D::W, DK, kRun<T>>(dk, Ss, Qr, open);
        } else {
            tile_rows_product<D::W, DK, kRun<T>>(dv, Ps, Gr);
            tile_rows_product<D::W, DK, kRun<T>>(dk, Ss, Qr);
        }
    }
    if (!GUARD && __syncthreads_or(not_finite(dk, j0 + ty * 4, S, DK) || not_finite(dv, j0 + ty * 4, S, DK))) return true;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int j = j0 + ty * 4 + r;
        if (j >= S) continue;
        T* p = dqkv + (static_cast<size_t>(b) * S + j) * ld + d + h * DK;
#pragma unroll
        for (int c = 0; c < D::W; ++c) {
            const int col = tile_col<D::W>(c);
            if (col < DK) { p[col] = from_f32<T>(scale * dk[r][c]); p[d + col] = from_f32<T>(dv[r][c]); }
        }
    }
    return false;
}
template <typename T, int DK>
__device__ __noinline__ void attn_bwd_dkv_guarded(float* sm, const T* qkv, const T* dout, const float* lse, const float* dvec, T* dqkv, const int* doc,
                                                  int B, int S, int H, int alibi, float scale)
{
    attn_bwd_dkv_block<T, DK, true>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
}
template <typename T, int DK>
__global__ void __launch_bounds__(256) attn_bwd_dkv_simt_kernel(const T* __restrict__ qkv, const T* __restrict__ dout, const float* __restrict__ lse,
                                                                const float* __restrict__ dvec, T* __restrict__ dqkv, const int* __restrict__ doc,
                                                                int B, int S, int H, int alibi, float scale)
{
    extern __shared__ __align__(16) float sm[];
    if (attn_bwd_dkv_block<T, DK, false>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale))
        attn_bwd_dkv_guarded<T, DK>(sm, qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
}

template <int DK> constexpr int simt_smem_fwd() { return (2 * DK * kTilePitch + SimtDims<DK>::ROWS + kTileFloats) * 4; }
template <int DK> constexpr int simt_smem_dq() { return (2 * DK * kTilePitch + 2 * SimtDims<DK>::KC * kTilePitch + SimtDims<DK>::ROWS + kTileFloats) * 4; }
template <int DK> constexpr int simt_smem_dkv() { return (4 * SimtDims<DK>::KC * kTilePitch + 2 * SimtDims<DK>::ROWS + 2 * kTileFloats) * 4; }
static_assert(simt_smem_dq<128>() <= 232448 && simt_smem_dkv<128>() <= 232448, "exceeds the 227 KB of shared memory a block may use");

template <typename T, int DK>
static int fwd_dk(const T* q, long long ldq, const T* k, const T* v, long long ldk, T* out, float* lse, const int* doc, int B, int S, int q0,
                  int H, int alibi, cudaStream_t s)
{
    NNB_ARG_CHECK(ceil_div(S - q0, kTile) * B * H <= INT_MAX, "too many tiles for one launch");
    static PerDeviceOnce once;
    NNB_TRY(once.run([] { return cudaFuncSetAttribute(attn_fwd_simt_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, simt_smem_fwd<DK>()); }));
    attn_fwd_simt_kernel<T, DK><<<static_cast<unsigned>(ceil_div(S - q0, kTile) * B * H), 256, simt_smem_fwd<DK>(), s>>>(
        q, ldq, k, v, ldk, out, lse, doc, B, S, q0, H, alibi, 1.0f / sqrtf(static_cast<float>(DK)));
    NNB_LAUNCH_CHECK();
    return 0;
}
template <typename T, int DK>
static int bwd_dk(const T* qkv, const T* out, const T* dout, const float* lse, float* dvec, T* dqkv, const int* doc,
                  int B, int S, int H, int alibi, cudaStream_t s)
{
    NNB_ARG_CHECK(ceil_div(S, kTile) * B * H <= INT_MAX, "too many tiles for one launch");
    static PerDeviceOnce once;
    NNB_TRY(once.run([] {
        const cudaError_t e = cudaFuncSetAttribute(attn_bwd_dq_simt_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, simt_smem_dq<DK>());
        return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_bwd_dkv_simt_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, simt_smem_dkv<DK>());
    }));
    const float scale = 1.0f / sqrtf(static_cast<float>(DK));
    NNB_TRY(launch_dvec<T>(out, dout, dvec, B, S, H, DK, s));
    const unsigned grid = static_cast<unsigned>(ceil_div(S, kTile) * B * H);
    attn_bwd_dq_simt_kernel<T, DK><<<grid, 256, simt_smem_dq<DK>(), s>>>(qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
    NNB_LAUNCH_CHECK();
    attn_bwd_dkv_simt_kernel<T, DK><<<grid, 256, simt_smem_dkv<DK>(), s>>>(qkv, dout, lse, dvec, dqkv, doc, B, S, H, alibi, scale);
    NNB_LAUNCH_CHECK();
    return 0;
}

#define DISPATCH_DK(dk, CALL)                                                         \
    switch (dk) {                                                                     \
        case 8: { constexpr int DKC = 8; return CALL; }                               \
        case 16: { constexpr int DKC = 16; return CALL; }                             \
        case 32: { constexpr int DKC = 32; return CALL; }                             \
        case 64: { constexpr int DKC = 64; return CALL; }                             \
        case 128: { constexpr int DKC = 128; return CALL; }                           \
        default: fprintf(stderr, "nnb200: attention head size %d unsupported (8,16,32,64,128)\n", dk); return -1; \
    }

template <typename T>
int attention_fwd_simt(const T* qkv, T* out, float* lse, const int* doc, int B, int S, int H, int dk, int alibi,
                       cudaStream_t s)
{
    if (static_cast<long long>(B) * S * H == 0) return 0;
    const int d = H * dk;
    DISPATCH_DK(dk, (fwd_dk<T, DKC>(qkv, 3 * d, qkv + d, qkv + 2 * d, 3 * d, out, lse, doc, B, S, 0, H, alibi, s)));
}

bool attention_prompt_supported(int dk) { return dk == 8 || dk == 16 || dk == 32 || dk == 64 || dk == 128; }
int attention_prompt(const float* qkv, const float* k_cache, const float* v_cache, float* out, int start, int n, int H, int dk, int alibi, cudaStream_t s)
{
    if (n == 0) return 0;
    const int d = H * dk;
    DISPATCH_DK(dk, (fwd_dk<float, DKC>(qkv, 3 * d, k_cache, v_cache, d, out, nullptr, nullptr, 1, start + n, start, H, alibi, s)));
}
template <typename T>
int attention_bwd_simt(const T* qkv, const T* out, const T* dout, const float* lse, float* dvec, T* dqkv,
                       const int* doc, int B, int S, int H, int dk, int alibi, cudaStream_t s)
{
    if (static_cast<long long>(B) * S * H == 0) return 0;
    DISPATCH_DK(dk, (bwd_dk<T, DKC>(qkv, out, dout, lse, dvec, dqkv, doc, B, S, H, alibi, s)));
}

int attention_dvec_bf16(const bf16* out, const bf16* dout, float* dvec, int B, int S, int H, int dk, cudaStream_t s)
{
    return launch_dvec<bf16>(out, dout, dvec, B, S, H, dk, s);
}

template int attention_fwd_simt<float>(const float*, float*, float*, const int*, int, int, int, int, int, cudaStream_t);
template int attention_fwd_simt<bf16>(const bf16*, bf16*, float*, const int*, int, int, int, int, int, cudaStream_t);
template int attention_bwd_simt<float>(const float*, const float*, const float*, const float*, float*, float*,
                                       const int*, int, int, int, int, int, cudaStream_t);
template int attention_bwd_simt<bf16>(const bf16*, const bf16*, const bf16*, const float*, float*, bf16*, const int*,
                                      int, int, int, int, int, cudaStream_t);

}  // namespace nnb
