// Incremental inference with a key/value cache: one token per call through every block of the model.
// Follows GPTModel::forward_step / GPTBlock::forward_step / AttentionBase::forward_step of the reference
// (compute_layer.hpp:2906-2950, 1426-1511; ALiBi bias of a step :2267-2290; rotary encoding of a step :964-988), which
// issues about thirty engine primitives, four transposes of the whole cache and two host-built matrices per block and
// token; here a block is five launches and nothing of the cache is copied.
// A single token is all matrix-vector work over bf16 weights (the shadow copy, in bf16 mode) or the fp32 master weights
// (check mode), fp32 activations and an fp32 cache in both modes.  What bounds it is not the weights' bytes (182 MB, 27 us
// for the 12-layer benchmark model) but the chain of about sixty dependent kernels, each of which would wait for its
// predecessor, then for its first loads.  So each is launched while its predecessor runs (programmatic dependent launch),
// loads what does not depend on it - its first weights, the norm's scale, the cached keys and values - into registers,
// and only then waits for it.  What the predecessor writes changes while the dependent kernel runs: such a pointer is not
// `const __restrict__`, which would promise the compiler constant memory that it may read early, and through the
// non-coherent path.  The normalisation before a projection is done while the input vector is staged in shared
// memory (every block does it for itself: the vector is a few KB), the activation in fc1's epilogue, the rotation of Q
// and K in the attention kernel.  Nothing may read, before its wait, what a kernel of the same token writes.
// The token id, position and cache length are read from device memory, so that the launches of a token are the same
// every time and a caller may replay them as a CUDA graph (nnb200_gpt_forward_step_dev).
// One token of the 12-layer model behind 900 cached ones: 211 us, of a 6-layer model of width 384 behind 40: 84 us (585 and 163
// with plain launches, the activation in fc2's staging and attention partials merged through global memory).
#include <algorithm>
#include <cmath>
#include <vector>

#include "kernels.h"
#include "nnb200.h"
#include "tc_ptx.cuh"

namespace nnb {

struct DecodeWs { size_t kv, table, x, qkv, att, xmid, h2, logits, step, total;
                  size_t p_tok, p_x, p_xn, p_qkv, p_att, p_mid, p_h1, p_h2, p_stat; };
// Rows of a prompt that one pass takes (longer prompts go in several): enough to fill the GEMM's tiles, 60 MB of
// activations for a model of width 1024.
constexpr int kPromptRows = 1024;
// Shorter prompts go through the single-token kernels: a pass costs as much as four to six tokens whatever its length (us for 4 and 6
// tokens as steps | a pass: 2 layers of 128: 126, 187 | 120; 6 of 384: 320, 476 | 450; 12 of 768: 873, 1304 | 1100).
constexpr int kPromptMin = 8;
static DecodeWs decode_ws(const nnb200_gpt_config& c)
{
    DecodeWs W;
    const size_t d = c.d_model, S = c.seq, fc1 = c.act == 1 ? 2 * static_cast<size_t>(c.d_ff) : c.d_ff;
    size_t off = 0;
    auto take = [&](size_t floats) { const size_t o = off; off = (off + floats * 4 + 255) / 256 * 256; return o; };
    W.kv = take(static_cast<size_t>(c.layers) * 2 * S * d);
    W.table = take(S * d);
    W.x = take(d); W.qkv = take(3 * d); W.att = take(d); W.xmid = take(d); W.h2 = take(c.d_ff); W.logits = take(c.vocab);
    W.step = take(4);                                            // token id, position, cache length
    const size_t R = std::min<size_t>(S, kPromptRows);
    W.p_tok = take(R); W.p_x = take(R * d); W.p_xn = take(R * d); W.p_qkv = take(R * 3 * d); W.p_att = take(R * d); W.p_mid = take(R * d);
    W.p_h1 = take(R * fc1); W.p_h2 = take(R * c.d_ff); W.p_stat = take(2 * R);
    W.total = off;
    return W;
}

__global__ void decode_set_step_kernel(int* __restrict__ step, int token, int pos, int cur_len)
{
    step[0] = token; step[1] = pos; step[2] = cur_len;
}

// Prompt ids travel as kernel parameters: the caller's buffer is read before the launch call returns, whatever kind of host
// memory it is (a copy from page-locked memory would read it when the stream gets there).
struct PromptIds { int id[512]; };
__global__ void decode_set_prompt_kernel(int* __restrict__ tok, const __grid_constant__ PromptIds ids, int n)
{
    if (static_cast<int>(threadIdx.x) < n) tok[threadIdx.x] = ids.id[threadIdx.x];
}
static int set_prompt(int* tok, const int* tokens_host, int n, cudaStream_t s)
{
    constexpr int kIds = static_cast<int>(sizeof(PromptIds) / sizeof(int));
    for (int i = 0; i < n; i += kIds) {
        const int k = std::min(n - i, kIds);
        PromptIds ids;
        std::copy_n(tokens_host + i, k, ids.id);
        std::fill(ids.id + k, ids.id + kIds, 0);
        decode_set_prompt_kernel<<<1, kIds, 0, s>>>(tok + i, ids, k);
        NNB_LAUNCH_CHECK();
    }
    return 0;
}

// programmatic dependent launch: let the next kernel of the stream start / wait until the one before has finished
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of what the predecessor wrote: volatile, so that they stay behind the wait, and not held up by stores to shared memory.
__device__ __forceinline__ float ld_produced(const float* p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_produced4(const float* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

template <typename... P, typename... A>
static int launch_dependent(void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = static_cast<unsigned>(cluster); at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    NNB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    NNB_LAUNCH_CHECK();
    return 0;
}

// x = token embedding (+ position row); pos_table: learned or sinusoidal rows, or null.  The first kernel of a token: launched
// without the dependent-launch attribute, so that it and everything behind it starts after all earlier work of the stream.
__global__ void decode_embed_kernel(const float* __restrict__ tok_emb, const float* __restrict__ pos_table, const int* __restrict__ step,
                                    int vocab, float* __restrict__ x, int d)
{
    pdl_launch();
    const int id = step[0], pos = step[1];
    const bool ok = id >= 0 && id < vocab;                      // an id out of range looks up a zero row (cpu_engine.hpp:150-158)
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d; c += gridDim.x * blockDim.x)
        x[c] = (ok ? tok_emb[static_cast<size_t>(id) * d + c] : 0.f) + (pos_table ? pos_table[static_cast<size_t>(pos) * d + c] : 0.f);
}

// y[o] = act(W[o, :] . f(x) + bias[o]) (+ residual[o]); a warp per group of R rows, 16-byte loads along the rows, eight of
// them in flight per lane, the first eight before the wait for the previous kernel.
//   NORM: f = norm(x) * gamma (+ beta), eps 1e-5 inside the rsqrt (compute_layer.hpp:495, 687; LayerNorm when `layer`).
//   ACT 1: SwiGLU, y[o] = gate * sigmoid(gate) * up of rows o and o + out (compute_layer.hpp:375-404), R = 2;
//   ACT 2: QuickGeLU (:266-295).
// R is 1 where there are too few rows for more than a warp each (latency), 4 for the LM head (8192 rows and more: fewer blocks
// that each stage x).
template <typename WT, bool NORM, int R, int ACT>
__global__ void __launch_bounds__(256, 3) gemv_kernel(const WT* __restrict__ W, const float* x, const float* __restrict__ gamma,
                                                   const float* __restrict__ beta, int layer, const float* __restrict__ bias,
                                                   const float* residual, float* __restrict__ y, int out, int in)
{
    static_assert(ACT != 1 || R == 2, "SwiGLU takes a gate and an up row");
    constexpr int VN = Vec16<WT>::N, NC = 8 / R;
    extern __shared__ __align__(16) float xs[];                 // `in` floats
    __shared__ float red[32];
    const int t = threadIdx.x, lane = t & 31, first = blockIdx.x * 8 + (t >> 5), step = gridDim.x * 8;
    const int units = ACT == 1 ? out : (out + R - 1) / R;
    const bool vec = (in % VN) == 0;
    const bool in_regs = NORM && (in & 3) == 0 && in <= 1024 &&
                         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta)) & 15) == 0;
    auto row = [&](int u, int r) { return ACT == 1 ? u + r * out : u * R + r; };
    auto row_ok = [&](int u, int r) { return ACT == 1 || R == 1 || u * R + r < out; };
    uint4 w[R][NC];                                             // as loaded; widened where used (eight values would take eight registers)
    auto load = [&](int u, int c0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const WT* p = W + static_cast<size_t>(row(u, r)) * in;
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const int c = c0 + (i * 32 + lane) * VN;
                if (c < in && row_ok(u, r)) w[r][i] = *reinterpret_cast<const uint4*>(p + c);
            }
        }
    };
    if (vec && first < units) load(first, 0);
    float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f), b4 = g4;
    if (in_regs && t * 4 < in) {
        g4 = *reinterpret_cast<const float4*>(gamma + t * 4);
        if (beta) b4 = *reinterpret_cast<const float4*>(beta + t * 4);
    }
    pdl_launch();
    pdl_wait();
    if (in_regs) {
        const bool mine = t * 4 < in;
        float4 v = mine ? ld_produced4(x + t * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (layer) {
            const float mean = block_sum((v.x + v.y) + (v.z + v.w), red) / static_cast<float>(in);
            if (mine) { v.x -= mean; v.y -= mean; v.z -= mean; v.w -= mean; }
        }
        const float rinv = rsqrtf(block_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w), red) / static_cast<float>(in) + 1e-5f);
        if (mine) *reinterpret_cast<float4*>(xs + t * 4) = make_float4(v.x * rinv * g4.x + b4.x, v.y * rinv * g4.y + b4.y, v.z * rinv * g4.z + b4.z, v.w * rinv * g4.w + b4.w);
    } else {
        if ((in & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
#pragma unroll 4
            for (int c = t * 4; c < in; c += 1024) *reinterpret_cast<float4*>(xs + c) = ld_produced4(x + c);
        } else {
#pragma unroll 4
            for (int c = t; c < in; c += 256) xs[c] = ld_produced(x + c);
        }
        if (NORM) {
            float mean = 0.f;
            __syncthreads();
            if (layer) {
                float sacc = 0.f;
                for (int c = t; c < in; c += 256) sacc += xs[c];
                mean = block_sum(sacc, red) / static_cast<float>(in);
            }
            float q = 0.f;
            for (int c = t; c < in; c += 256) { const float v = xs[c] - mean; q += v * v; }
            const float rinv = rsqrtf(block_sum(q, red) / static_cast<float>(in) + 1e-5f);
            for (int c = t; c < in; c += 256) xs[c] = (xs[c] - mean) * rinv * gamma[c] + (beta ? beta[c] : 0.f);
        }
    }
    __syncthreads();
    for (int u = first; u < units; u += step) {
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.f;
        if (vec) {
            for (int c0 = 0; c0 < in; c0 += NC * 32 * VN) {
                if (c0 > 0 || u != first) load(u, c0);
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int i = 0; i < NC; ++i) asm volatile("" : "+r"(w[r][i].x), "+r"(w[r][i].y), "+r"(w[r][i].z), "+r"(w[r][i].w));
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    const int c = c0 + (i * 32 + lane) * VN;
                    if (c < in) {
#pragma unroll
                        for (int k = 0; k < VN; k += 4) {
                            const float4 f = *reinterpret_cast<const float4*>(xs + c + k);
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                if (!row_ok(u, r)) continue;
                                Vec16<WT> v;
                                *reinterpret_cast<uint4*>(&v) = w[r][i];
                                acc[r] = fmaf(to_f32(v.v[k]), f.x, acc[r]);
                                acc[r] = fmaf(to_f32(v.v[k + 1]), f.y, acc[r]);
                                acc[r] = fmaf(to_f32(v.v[k + 2]), f.z, acc[r]);
                                acc[r] = fmaf(to_f32(v.v[k + 3]), f.w, acc[r]);
                            }
                        }
                    }
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!row_ok(u, r)) continue;
                const WT* p = W + static_cast<size_t>(row(u, r)) * in;
                for (int c = lane; c < in; c += 32) acc[r] = fmaf(to_f32(p[c]), xs[c], acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = warp_sum(acc[r]);
        if (lane != 0) continue;
        if (ACT == 1) {
            const float g = acc[0] + bias[u];
            y[u] = g / (1.0f + expf(-g)) * (acc[R - 1] + bias[u + out]);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int o = u * R + r;
                if (!row_ok(u, r)) continue;
                float v = acc[r] + bias[o];
                if (ACT == 2) v = v / (1.0f + expf(-1.702f * v));
                y[o] = v + (residual ? ld_produced(residual + o) : 0.f);
            }
        }
    }
}

// Attention of one token over the cache: a cluster of eight blocks per head, cached row j on lane group j modulo all the groups
// of the cluster (LPR lanes carry a row, NV 16-byte vectors each), B rows in flight per group.  All cached rows but the
// token's own were written by earlier tokens, so the first B keys and values are loaded before the wait.  The token's key
// and value are appended to the cache on the way.  Scores q_h . k_j / sqrt(dk) - slope_h (cur_len - j), softmax kept online
// per group, groups merged by shuffles, warps through shared memory and blocks through the cluster's shared memory, in a
// fixed order.  The grid is the same for every cache length.
// Bound by the chain wait - scores - merge.  (12 heads of 64 behind 900 tokens took 22.6 us when blocks of 32 rows left partial
// results in global memory and the last one merged them; a whole layer, this kernel and four products, takes 17 us now.)
// Behind long contexts by the latency of a round of rows: where a row takes a whole warp, blocks have 512 threads and load the
// next round's rows as soon as this round's were used (a step of two layers, one head of 128 behind 65535 rows: 372 us; 1366
// with the loads at the start of a round and 256 threads, 780 with blocks of 32 rows).
template <int LPR, int NV, bool VEC, int THREADS>
__global__ void __launch_bounds__(THREADS) decode_attn_kernel(const float* qkv, float* __restrict__ kc, float* __restrict__ vc,
                                                          float* __restrict__ out, const float* __restrict__ rope, const int* __restrict__ step,
                                                          int seq, int d, int dk, int heads, int alibi, float scale)
{
    constexpr int B = 8 / NV, G = THREADS / LPR, RANKS = 8, DMAX = LPR * NV * 4, WARPS = THREADS / 32, ROUND = B * RANKS * G;
    constexpr bool EARLY = THREADS == 512;                       // next round's keys and values loaded as soon as this round's were used
    __shared__ float wm[WARPS], wl[WARPS];
    __shared__ __align__(16) float wo[WARPS][DMAX];
    __shared__ float part[DMAX + 2];                            // this block's maximum, sum and weighted values
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, sub = t % LPR, h = blockIdx.x / RANKS;
    const int rank = static_cast<int>(cluster_ctarank()), g0 = rank * G + t / LPR;
    const int cur = step[2], n = cur + 1;
    const size_t head = static_cast<size_t>(h) * dk;
    auto fetch = [&](const float* p, float (&v)[NV * 4]) {      // this lane's columns of a row; zero beyond dk
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = (i * LPR + sub) * 4;
            if (VEC) {
                const float4 f = c < dk ? *reinterpret_cast<const float4*>(p + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[i * 4] = f.x; v[i * 4 + 1] = f.y; v[i * 4 + 2] = f.z; v[i * 4 + 3] = f.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[i * 4 + k] = c + k < dk ? p[c + k] : 0.f;
            }
        }
    };
    float kr[B][NV * 4], vr[B][NV * 4];
    auto load = [&](int j0, bool keys, bool values) {
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int j = j0 + b * (RANKS * G);
            if (j < cur) {
                if (keys) fetch(kc + static_cast<size_t>(j) * d + head, kr[b]);
                if (values) fetch(vc + static_cast<size_t>(j) * d + head, vr[b]);
            }
        }
    };
    load(g0, true, true);
    pdl_launch();
    pdl_wait();
    // q or the new k: rotated with rotary positions by the cache row it lands in (table: cos (seq, dk/2), then sin)
    auto rotated = [&](const float* p, float (&v)[NV * 4]) {
        fetch(p, v);
        if (!rope) return;
        const int half = dk / 2;
        const float *cs = rope + static_cast<size_t>(cur) * half, *sn = rope + (static_cast<size_t>(seq) + cur) * half;
#pragma unroll
        for (int i = 0; i < NV * 4; ++i) {
            const int c = ((i / 4) * LPR + sub) * 4 + i % 4;
            if (c < half) v[i] = v[i] * cs[c] - p[c + half] * sn[c];
            else if (c < dk) v[i] = v[i] * cs[c - half] + p[c - half] * sn[c - half];
        }
    };
    float q[NV * 4], o[NV * 4];
    rotated(qkv + head, q);
#pragma unroll
    for (int i = 0; i < NV * 4; ++i) o[i] = 0.f;
    const float slope = alibi ? exp2f(-8.0f * static_cast<float>(h) / static_cast<float>(heads)) : 0.f;
    float m = -INFINITY, l = 0.f;
    for (int j0 = g0; j0 - t / LPR % (32 / LPR) < n; j0 += ROUND) {             // the same number of rounds for all groups of a warp
        if (!EARLY && j0 != g0) load(j0, true, true);
        float s[B];
        float mx = m;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int j = j0 + b * (RANKS * G);
            if (j == cur) {
                rotated(qkv + d + head, kr[b]);
                fetch(qkv + 2 * d + head, vr[b]);
#pragma unroll
                for (int i = 0; i < NV * 4; ++i) {
                    const int c = ((i / 4) * LPR + sub) * 4 + i % 4;
                    if (c < dk) {
                        kc[static_cast<size_t>(cur) * d + head + c] = kr[b][i];
                        vc[static_cast<size_t>(cur) * d + head + c] = vr[b][i];
                    }
                }
            }
            float a = 0.f;
            if (j < n) {
#pragma unroll
                for (int i = 0; i < NV * 4; ++i) a = fmaf(q[i], kr[b][i], a);
            }
#pragma unroll
            for (int w = LPR / 2; w > 0; w >>= 1) a += __shfl_xor_sync(0xffffffffu, a, w);
            s[b] = j < n ? a * scale - slope * static_cast<float>(cur - j) : -INFINITY;
            mx = fmaxf(mx, s[b]);
        }
        if (EARLY) load(j0 + ROUND, true, false);
        const float ref = mx == -INFINITY ? 0.f : mx, back = expf(m - ref);
        m = mx;
        l *= back;
#pragma unroll
        for (int i = 0; i < NV * 4; ++i) o[i] *= back;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            if (j0 + b * (RANKS * G) >= n) break;
            const float e = expf(s[b] - ref);
            l += e;
#pragma unroll
            for (int i = 0; i < NV * 4; ++i) o[i] = fmaf(e, vr[b][i], o[i]);
        }
        if (EARLY) load(j0 + ROUND, false, true);
    }
#pragma unroll
    for (int w = LPR; w < 32; w <<= 1) {                        // groups of a warp
        const float om = __shfl_xor_sync(0xffffffffu, m, w), nm = fmaxf(m, om), ref = nm == -INFINITY ? 0.f : nm;
        const float a = expf(m - ref), b = expf(om - ref);
        l = l * a + __shfl_xor_sync(0xffffffffu, l, w) * b;
#pragma unroll
        for (int i = 0; i < NV * 4; ++i) o[i] = o[i] * a + __shfl_xor_sync(0xffffffffu, o[i], w) * b;
        m = nm;
    }
    if (lane == 0) { wm[warp] = m; wl[warp] = l; }
    if (lane < LPR) {
#pragma unroll
        for (int i = 0; i < NV; ++i) *reinterpret_cast<float4*>(&wo[warp][(i * LPR + sub) * 4]) = make_float4(o[i * 4], o[i * 4 + 1], o[i * 4 + 2], o[i * 4 + 3]);
    }
    __syncthreads();
    {                                                           // warps of the block
        float bm = wm[0];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) bm = fmaxf(bm, wm[w]);
        const float ref = bm == -INFINITY ? 0.f : bm;
        if (t < DMAX) {
            float bl = 0.f, a = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) { const float e = expf(wm[w] - ref); bl += wl[w] * e; a = fmaf(wo[w][t], e, a); }
            part[2 + t] = a;
            if (t == 0) { part[0] = bm; part[1] = bl; }
        }
    }
    cluster_sync_all();
    const int cols = (dk + RANKS - 1) / RANKS, c = rank * cols + t;
    if (t < cols && c < dk) {                                   // blocks of the cluster: each finishes its share of the columns
        const uint32_t base = smem_u32(part);
        float pm[RANKS], pl[RANKS], po[RANKS], gm = -INFINITY, gl = 0.f, a = 0.f;
#pragma unroll
        for (int r = 0; r < RANKS; ++r) {
            const uint32_t p = mapa_shared(base, r);
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(pm[r]) : "r"(p) : "memory");
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(pl[r]) : "r"(p + 4) : "memory");
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(po[r]) : "r"(p + 8 + 4 * c) : "memory");
        }
#pragma unroll
        for (int r = 0; r < RANKS; ++r) gm = fmaxf(gm, pm[r]);
        const float ref = gm == -INFINITY ? 0.f : gm;
#pragma unroll
        for (int r = 0; r < RANKS; ++r) { const float e = expf(pm[r] - ref); gl += pl[r] * e; a = fmaf(po[r], e, a); }
        out[head + c] = a / gl;
    }
    cluster_sync_all();                                         // nobody's shared memory goes while a peer reads it
}

template <typename WT, bool NORM, int R, int ACT>
static int gemv(const WT* W, const float* x, const float* gamma, const float* beta, int layer, const float* bias, const float* residual,
                float* y, int out, int in, cudaStream_t s)
{
    NNB_ARG_CHECK(static_cast<size_t>(in) * sizeof(float) <= 48 * 1024, "input vector too long for the decode matrix-vector kernel");
    const long long units = ACT == 1 ? out : ceil_div(out, R);
    return launch_dependent(gemv_kernel<WT, NORM, R, ACT>, dim3(grid_for(units, 8)), 256, static_cast<size_t>(in) * sizeof(float), 1, s, W, x, gamma,
                            beta, layer, bias, residual, y, out, in);
}

static int decode_attention(const float* qkv, float* kc, float* vc, float* out, const float* rope, const int* step, const nnb200_gpt_config& c, cudaStream_t s)
{
    const int d = c.d_model, dk = d / c.heads;
    const dim3 grid(static_cast<unsigned>(c.heads) * 8);
    auto go = [&](auto* kernel, int threads) {
        return launch_dependent(kernel, grid, threads, 0, 8, s, qkv, kc, vc, out, rope, step, c.seq, d, dk, c.heads, c.pos == 2 ? 1 : 0,
                                1.0f / sqrtf(static_cast<float>(dk)));
    };
    const bool vec = dk % 4 == 0 && ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;
    if (vec && dk <= 32) return go(decode_attn_kernel<8, 1, true, 256>, 256);
    if (vec && dk <= 64) return go(decode_attn_kernel<16, 1, true, 256>, 256);
    // A row that takes a whole warp leaves a cluster of 256 threads 64 rows at a time: 512 threads halve the rounds, as long as
    // the blocks, which then fill an SM's registers, leave SMs free for the predecessor's (a step of two layers, heads of 128
    // behind 900 | 8191 rows: 8 heads 43 | 212 us with 256 threads, 38 | 88 with 512; 16 heads 88 | 252 and 91 | 173).
    if (c.heads <= 8) {
        if (dk <= 128) return vec ? go(decode_attn_kernel<32, 1, true, 512>, 512) : go(decode_attn_kernel<32, 1, false, 512>, 512);
        return vec ? go(decode_attn_kernel<32, 2, true, 512>, 512) : go(decode_attn_kernel<32, 2, false, 512>, 512);
    }
    if (dk <= 128) return vec ? go(decode_attn_kernel<32, 1, true, 256>, 256) : go(decode_attn_kernel<32, 1, false, 256>, 256);
    return vec ? go(decode_attn_kernel<32, 2, true, 256>, 256) : go(decode_attn_kernel<32, 2, false, 256>, 256);
}

// `step` (device): token id, position, cache length
template <typename WT>
static int forward_step_t(const nnb200_gpt_config& c, const float* P, const WT* Wt, uint8_t* ws, const int* step, float* logits_out,
                          cudaStream_t s)
{
    const DecodeLayout L = decode_layout(c);
    const DecodeWs W = decode_ws(c);
    const int d = c.d_model, ff = c.d_ff, dk = d / c.heads;
    const int ln = c.norm == 0 ? 1 : 0;
    NNB_ARG_CHECK(dk <= 256, "head size above 256");
    auto F = [&](size_t off) { return reinterpret_cast<float*>(ws + off); };
    auto PB = [&](long long off) { return off >= 0 ? P + off : nullptr; };
    const float* pos_table = nullptr;
    if (c.pos == 0) pos_table = P + L.pos_emb;
    else if (c.pos == 1) pos_table = F(W.table);
    decode_embed_kernel<<<grid_for(d, 256), 256, 0, s>>>(P + L.tok_emb, pos_table, step, c.vocab, F(W.x), d);
    NNB_LAUNCH_CHECK();
    const size_t layer_kv = static_cast<size_t>(2) * c.seq * d;
    float* x = F(W.x);
    float* xmid = F(W.xmid);
    for (int l = 0; l < c.layers; ++l) {
        const DecodeLayer& lp = L.layers[l];
        float* kc = F(W.kv) + static_cast<size_t>(l) * layer_kv;
        float* vc = kc + static_cast<size_t>(c.seq) * d;
        NNB_TRY((gemv<WT, true, 1, 0>(Wt + lp.wqkv, x, P + lp.g1, PB(lp.be1), ln, P + lp.bqkv, nullptr, F(W.qkv), 3 * d, d, s)));
        NNB_TRY(decode_attention(F(W.qkv), kc, vc, F(W.att), c.pos == 3 ? F(W.table) : nullptr, step, c, s));
        NNB_TRY((gemv<WT, false, 1, 0>(Wt + lp.wo, F(W.att), nullptr, nullptr, 0, P + lp.bo, x, xmid, d, d, s)));          // + residual (GPTBlock::forward_step)
        if (c.act == 1) NNB_TRY((gemv<WT, true, 2, 1>(Wt + lp.w1, xmid, P + lp.g2, PB(lp.be2), ln, P + lp.b1, nullptr, F(W.h2), ff, d, s)));
        else NNB_TRY((gemv<WT, true, 1, 2>(Wt + lp.w1, xmid, P + lp.g2, PB(lp.be2), ln, P + lp.b1, nullptr, F(W.h2), ff, d, s)));
        NNB_TRY((gemv<WT, false, 1, 0>(Wt + lp.w2, F(W.h2), nullptr, nullptr, 0, P + lp.b2, xmid, x, d, ff, s)));   // + residual
    }
    return gemv<WT, true, 4, 0>(Wt + L.lm_w, x, P + L.lnf_g, PB(L.lnf_b), ln, P + L.lm_b, nullptr, logits_out ? logits_out : F(W.logits), c.vocab, d, s);
}

// Y[n, out] = X[n, in] W[out, in]^T + bias (+ residual), fp32 rows times fp32 or bf16 weights
static int prompt_linear(const float* X, const float* W, const float* bias, const float* residual, float* Y, int n, int in, int out, cudaStream_t s)
{
    return sgemm_strided(X, W, Y, n, out, in, in, 1, in, 1, out, 1, 0, 0, 0, 1.0f, bias, nullptr, residual, 0, s);
}
static int prompt_linear(const float* X, const bf16* W, const float* bias, const float* residual, float* Y, int n, int in, int out, cudaStream_t s)
{
    return gemm_f32_bf16(X, W, Y, n, out, in, bias, residual, s);
}

// n <= kPromptRows prompt tokens (device) at cache rows start ..: the layers as products over all rows, with the fp32
// activations, weights and cache of the single-token kernels.  Leaves the last layer's output rows in p_x.
// A token at a time reads every weight per token: 501 tokens of the 12-layer benchmark model and 16 new
// ones took 282 ms, of which the prompt 260; now 6.7 ms in all.
template <typename WT>
static int prompt_pass_t(const nnb200_gpt_config& c, const float* P, const WT* Wt, uint8_t* ws, const int* tokens, int start, int n, cudaStream_t s)
{
    const DecodeLayout L = decode_layout(c);
    const DecodeWs W = decode_ws(c);
    const int d = c.d_model, ff = c.d_ff, fc1 = c.act == 1 ? 2 * ff : ff, dk = d / c.heads;
    const bool ln = c.norm == 0;
    auto F = [&](size_t off) { return reinterpret_cast<float*>(ws + off); };
    auto PB = [&](long long off) { return off >= 0 ? P + off : nullptr; };
    const float* pos_table = c.pos == 0 ? P + L.pos_emb : (c.pos == 1 ? F(W.table) : nullptr);
    float *x = F(W.p_x), *xn = F(W.p_xn), *qkv = F(W.p_qkv), *att = F(W.p_att), *mid = F(W.p_mid), *h1 = F(W.p_h1), *h2 = F(W.p_h2);
    float *rinv = F(W.p_stat), *mean = rinv + n;
    // rows of the tables and of the cache begin at `start`; the kernels count from there (n <= seq - start)
    NNB_TRY(embed_fwd<float>(P + L.tok_emb, pos_table ? pos_table + static_cast<size_t>(start) * d : nullptr, tokens, x, n, c.seq, d, c.vocab, s));
    const size_t layer_kv = static_cast<size_t>(2) * c.seq * d;
    for (int l = 0; l < c.layers; ++l) {
        const DecodeLayer& lp = L.layers[l];
        float* kc = F(W.kv) + static_cast<size_t>(l) * layer_kv;
        float* vc = kc + static_cast<size_t>(c.seq) * d;
        NNB_TRY(norm_fwd<float>(x, P + lp.g1, PB(lp.be1), xn, rinv, mean, n, d, ln, s));
        NNB_TRY(prompt_linear(xn, Wt + lp.wqkv, P + lp.bqkv, nullptr, qkv, n, d, 3 * d, s));
        if (c.pos == 3) NNB_TRY(rope_apply<float>(qkv, F(W.table) + static_cast<size_t>(start) * (dk / 2), n, c.seq, c.heads, dk, 3 * d, false, s));
        for (int w = 0; w < 2; ++w)
            NNB_CUDA_CHECK(cudaMemcpy2DAsync((w ? vc : kc) + static_cast<size_t>(start) * d, static_cast<size_t>(d) * 4, qkv + (1 + w) * d,
                                             static_cast<size_t>(3) * d * 4, static_cast<size_t>(d) * 4, n, cudaMemcpyDeviceToDevice, s));
        NNB_TRY(attention_prompt(qkv, kc, vc, att, start, n, c.heads, dk, c.pos == 2 ? 1 : 0, s));
        NNB_TRY(prompt_linear(att, Wt + lp.wo, P + lp.bo, x, mid, n, d, d, s));
        NNB_TRY(norm_fwd<float>(mid, P + lp.g2, PB(lp.be2), xn, rinv, mean, n, d, ln, s));
        NNB_TRY(prompt_linear(xn, Wt + lp.w1, P + lp.b1, nullptr, h1, n, d, fc1, s));
        NNB_TRY(act_fwd<float>(h1, h2, n, ff, c.act == 1, s));
        NNB_TRY(prompt_linear(h2, Wt + lp.w2, P + lp.b2, mid, x, n, ff, d, s));
    }
    return 0;
}

template <typename WT>
static int prefill_t(const nnb200_gpt_config& c, const float* P, const WT* Wt, uint8_t* ws, const int* tokens_host, int n, int start,
                     float* logits_out, cudaStream_t s)
{
    const DecodeWs W = decode_ws(c);
    int* tok = reinterpret_cast<int*>(ws + W.p_tok);
    const bool aligned = ((reinterpret_cast<uintptr_t>(ws) | reinterpret_cast<uintptr_t>(P)) & 15) == 0;      // the row kernels' vectors
    if (n < kPromptMin || !aligned || !attention_prompt_supported(c.d_model / c.heads)) {
        int* step = reinterpret_cast<int*>(ws + W.step);
        for (int i = 0; i < n; ++i) {
            decode_set_step_kernel<<<1, 1, 0, s>>>(step, tokens_host[i], start + i, start + i);
            NNB_LAUNCH_CHECK();
            NNB_TRY(forward_step_t<WT>(c, P, Wt, ws, step, logits_out, s));
        }
        return 0;
    }
    int rows = 0;
    for (int i = 0; i < n; i += rows) {
        rows = std::min(n - i, kPromptRows);
        NNB_TRY(set_prompt(tok, tokens_host + i, rows, s));
        NNB_TRY(prompt_pass_t<WT>(c, P, Wt, ws, tok, start + i, rows, s));
    }
    const DecodeLayout L = decode_layout(c);
    float* F = reinterpret_cast<float*>(ws);
    return gemv<WT, true, 4, 0>(Wt + L.lm_w, F + W.p_x / 4 + static_cast<size_t>(rows - 1) * c.d_model, P + L.lnf_g, L.lnf_b >= 0 ? P + L.lnf_b : nullptr,
                       c.norm == 0 ? 1 : 0, P + L.lm_b, nullptr, logits_out ? logits_out : F + W.logits / 4, c.vocab, c.d_model, s);
}

}  // namespace nnb

using namespace nnb;

extern "C" {

long long nnb200_gpt_decode_workspace_bytes(const nnb200_gpt_config* cfg)
{
    if (nnb200_gpt_arena_elems(cfg) < 0) return -1;             // validates the configuration
    return static_cast<long long>(decode_ws(*cfg).total);
}

int nnb200_gpt_decode_init(const nnb200_gpt_config* cfg, void* workspace, void* stream)
{
    if (nnb200_gpt_arena_elems(cfg) < 0 || !workspace) { fprintf(stderr, "nnb200_gpt_decode_init: bad arguments\n"); return -1; }
    const DecodeWs W = decode_ws(*cfg);
    const int S = cfg->seq, d = cfg->d_model;
    std::vector<float> tab;
    if (cfg->pos == 3) {
        tab.resize(static_cast<size_t>(S) * (d / cfg->heads));
        rope_table_host(S, d / cfg->heads, tab.data());
    } else if (cfg->pos == 1) {
        // SinusoidalPositionEncoder (compute_layer.hpp:2604-2622), with the reference's float calls
        tab.resize(static_cast<size_t>(S) * d);
        for (int pos = 0; pos < S; ++pos)
            for (int i = 0; i < d; ++i) {
                const float angle = static_cast<float>(pos) / std::pow(10000.0f, static_cast<float>(2 * (i / 2)) / static_cast<float>(d));
                tab[static_cast<size_t>(pos) * d + i] = (i % 2 == 0) ? std::sin(angle) : std::cos(angle);
            }
    }
    if (!tab.empty()) {
        NNB_CUDA_CHECK(cudaMemcpyAsync(static_cast<uint8_t*>(workspace) + W.table, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice, to_stream(stream)));
        NNB_CUDA_CHECK(cudaStreamSynchronize(to_stream(stream)));          // `tab` is pageable host memory about to go away
    }
    return 0;
}

static int forward_step_any(const nnb200_gpt_config* cfg, const float* params, const void* params_bf16, uint8_t* ws, const int* step,
                            float* logits_out, cudaStream_t s)
{
    if (cfg->precision == 1) {
        NNB_ARG_CHECK(params_bf16 != nullptr, "bf16 mode needs the bf16 parameter shadow");
        return forward_step_t<bf16>(*cfg, params, static_cast<const bf16*>(params_bf16), ws, step, logits_out, s);
    }
    return forward_step_t<float>(*cfg, params, params, ws, step, logits_out, s);
}

int nnb200_gpt_forward_step(const nnb200_gpt_config* cfg, const float* params, const void* params_bf16, void* workspace, int token_id,
                            int pos, int cur_len, float* logits_out, void* stream)
{
    if (nnb200_gpt_arena_elems(cfg) < 0 || !params || !workspace) { fprintf(stderr, "nnb200_gpt_forward_step: bad arguments\n"); return -1; }
    NNB_ARG_CHECK(cur_len >= 0 && cur_len < cfg->seq, "the cache holds seq rows: cur_len must be in [0, seq)");
    NNB_ARG_CHECK(pos >= 0 && pos < cfg->seq, "position out of range");
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    int* step = reinterpret_cast<int*>(ws + decode_ws(*cfg).step);
    decode_set_step_kernel<<<1, 1, 0, to_stream(stream)>>>(step, token_id, pos, cur_len);
    NNB_LAUNCH_CHECK();
    return forward_step_any(cfg, params, params_bf16, ws, step, logits_out, to_stream(stream));
}

int nnb200_gpt_prefill(const nnb200_gpt_config* cfg, const float* params, const void* params_bf16, void* workspace, const int32_t* tokens_host,
                       int n, int cur_len, float* logits_out, void* stream)
{
    if (nnb200_gpt_arena_elems(cfg) < 0 || !params || !workspace || !tokens_host) { fprintf(stderr, "nnb200_gpt_prefill: bad arguments\n"); return -1; }
    NNB_ARG_CHECK(n >= 1 && cur_len >= 0 && n <= cfg->seq && cur_len <= cfg->seq - n, "the cache holds seq rows: [cur_len, cur_len + n) must lie in them");
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    if (cfg->precision == 1) {
        NNB_ARG_CHECK(params_bf16 != nullptr, "bf16 mode needs the bf16 parameter shadow");
        return prefill_t<bf16>(*cfg, params, static_cast<const bf16*>(params_bf16), ws, tokens_host, n, cur_len, logits_out, to_stream(stream));
    }
    return prefill_t<float>(*cfg, params, params, ws, tokens_host, n, cur_len, logits_out, to_stream(stream));
}

int nnb200_gpt_decode_set_step(int32_t* step_dev, int token_id, int pos, int cur_len, void* stream)
{
    NNB_ARG_CHECK(step_dev != nullptr, "null step buffer");
    decode_set_step_kernel<<<1, 1, 0, to_stream(stream)>>>(step_dev, token_id, pos, cur_len);
    NNB_LAUNCH_CHECK();
    return 0;
}

int nnb200_gpt_forward_step_dev(const nnb200_gpt_config* cfg, const float* params, const void* params_bf16, void* workspace,
                                const int32_t* step_dev, float* logits_out, void* stream)
{
    if (nnb200_gpt_arena_elems(cfg) < 0 || !params || !workspace || !step_dev) { fprintf(stderr, "nnb200_gpt_forward_step_dev: bad arguments\n"); return -1; }
    return forward_step_any(cfg, params, params_bf16, static_cast<uint8_t*>(workspace), step_dev, logits_out, to_stream(stream));
}

}  // extern "C"
