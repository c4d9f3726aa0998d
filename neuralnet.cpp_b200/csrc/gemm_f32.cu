// fp32 GEMM on the bf16 tensor cores: the contraction behind cuda_matmul / cuda_batched_matmul, the fp32 mode of the
// training step and the prompt pass of incremental decoding.
//
// An fp32 number is the sum of three bf16 numbers, x = hi + mid + lo (8 significand bits each, the residuals formed
// exactly in fp32), so a product of two fp32 numbers is nine bf16 products, of which the three smallest (mid*lo, lo*mid,
// lo*lo, below 2^-25 of the product) are left out: less than the rounding of one fp32 multiplication.  Six tensor-core
// products replace one fp32 FMA, at 1/6 of the bf16 rate against 1/32 of it on the fp32 pipe.  With a bf16 operand B
// (weights of the decoding path) three products are exact.
// The tensor core adds into its accumulator without rounding to nearest, which would drift over a long K: a TMEM
// accumulator therefore holds one block of 64 k only (small products first) and all warps add it to fp32 registers,
// rounding to nearest, while the other TMEM buffer fills.
// bf16 has the exponents of fp32, so the lower planes of a small operand (below 2^-110) would fall under its smallest number:
// what the first plane leaves is enlarged by 2^15 before the other two are taken, and the MMAs take the factor out again.
// A sum that is not finite (an operand that is not, or beyond 2^121, or a sum beyond 2^115) is computed again with fp32 FMAs
// (sgemm_exact), which is what the result then is.
//
// One CTA per SM, persistent over output tiles of 128 x BN.  All 16 warps do the same work on a quarter of everything: load
// fp32 from global memory into registers a block of 64 k ahead (any row stride or alignment, either operand contiguous
// along K or along M / N), split it and write the three planes as 128-byte-swizzled tiles, and add a finished accumulator
// (32 rows x BN / 4 columns per warp) to their registers; one thread issues the MMAs.  The epilogue transposes through the
// idle operand stages so that stores are whole row pieces.  An output of too few tiles for the machine is also split along K
// over the CTAs of a cluster; the partial tiles are added in rank order through distributed shared memory, so results never
// depend on timing.
// What bounds it: the chain load - split - MMA - add of a block, of which a CTA overlaps two (about 4600 clocks per 128 x 128 x 64
// block against 1536 of MMA; issue slots 40 % busy, waits on global loads first).  4096^3: 1040 us (132 TFLOP/s; 4860 us as a SIMT
// kernel of 64 x 64 tiles); 1024 x 8192 x 384: 76 us (226 there, 408 with transposed operands); 1024 x 384 x 128: 12.0 us back
// to back (12.8).
#include <cstring>

#include "kernels.h"
#include "tc_ptx.cuh"

namespace nnb {

__device__ int g_f32gemm_error = 0;

namespace {

constexpr int FM = 128, FK = 64, F_THREADS = 512;
constexpr int F_PLANE_A = FM * FK * 2;                           // one bf16 plane of an A tile, bytes
constexpr int F_SHIFT = 15;                                      // the residual behind the first plane is enlarged by 2^15

struct F32GemmParams {
    const float* A;
    const void* B;
    float* C;
    int M, N, K, batch;
    long long lda, ldb, ldc, batch_a, batch_b, batch_c;          // lda / ldb: stride of the non-contiguous index
    int a_vec, b_vec;                                            // 16-byte loads allowed
    int tiles_m, tiles_n, kb_total, kb_per_split;
    float alpha;
    const float *bias_n, *bias_m, *residual;
    int accumulate;
};

// One element of the product in plain fp32 FMAs, ascending k.  A NaN stays one whatever follows: a product of matrices full of
// them ends in the first step (4096^3: 250 ms with every chain to its end, 4.9 ms in a SIMT kernel).  Eight k are loaded at
// a time, so that a long chain waits for memory once in eight steps.
template <typename BT, bool A_MN, bool B_MN>
__device__ __noinline__ float sgemm_exact(const F32GemmParams& p, int b, int m, int n)
{
    const float* a = p.A + b * p.batch_a + (A_MN ? m : m * p.lda);
    const BT* w = static_cast<const BT*>(p.B) + b * p.batch_b + (B_MN ? n : n * p.ldb);
    const long long sa = A_MN ? p.lda : 1, sw = B_MN ? p.ldb : 1;
    float s = 0.f;
    int k = 0;
    for (; k + 8 <= p.K; k += 8) {
        float x[8], y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { x[j] = a[(k + j) * sa]; y[j] = to_f32(w[(k + j) * sw]); }
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(x[j], y[j], s);
        if (s != s) return s;
    }
    for (; k < p.K; ++k) s = fmaf(a[k * sa], to_f32(w[k * sw]), s);
    return s;
}

// The part of an operand tile (ROWS x 64) that one loader thread carries from global to shared memory: N groups of eight
// consecutive elements (32 bytes of fp32: a warp reads whole 256-byte rows).
template <typename T, bool MN, int ROWS>
struct Frag {
    static constexpr int N = ROWS * FK / 8 / F_THREADS;
    static constexpr int G = ROWS / 8;                            // groups along the rows of an MN-major tile
    uint4 v[N][sizeof(T) / 2];

    // first element of this thread inside the tile: (row, k); group i is `istep` rows (K-major) or k (MN-major) further
    static constexpr int istep = MN ? F_THREADS / G : F_THREADS / 8;
    __device__ __forceinline__ static int row_of(int t) { return MN ? (t % G) * 8 : t >> 3; }
    __device__ __forceinline__ static int k_of(int t) { return MN ? t / G : (t & 7) * 8; }

    // `p`: this thread's first element of the k-block; whole tile inside the operand, rows on 16-byte boundaries
    __device__ __forceinline__ void load_whole(const T* p, long long ld)
    {
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < static_cast<int>(sizeof(T)) / 2; ++j) v[i][j] = *reinterpret_cast<const uint4*>(p + i * istep * ld + j * (16 / sizeof(T)));
    }
    // any edge, any alignment: elements outside are zero
    __device__ __forceinline__ void load_edge(const T* base, long long ld, int row0, int rows, int k0, int K, int t)
    {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int r = row0 + row_of(t) + (MN ? 0 : i * istep), k = k0 + k_of(t) + (MN ? i * istep : 0);
            const int left = MN ? (k < K ? rows - r : 0) : (r < rows ? K - k : 0);
            const T* q = base + (MN ? k * ld + r : r * ld + k);
            T e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = j < left ? q[j] : from_f32<T>(0.f);
#pragma unroll
            for (int j = 0; j < static_cast<int>(sizeof(T)) / 2; ++j) memcpy(&v[i][j], e + j * (16 / sizeof(T)), 16);
        }
    }
    __device__ __forceinline__ void load(const T* base, const T* mine, long long ld, int row0, int rows, int k0, int K, bool vec, int t)
    {
        if (vec && row0 + ROWS <= rows && k0 + FK <= K) load_whole(mine + (MN ? k0 * ld : k0), ld);
        else load_edge(base, ld, row0, rows, k0, K, t);
    }
    // K-major tile: row r at r * 128 bytes; MN-major: k row at k * 128 bytes, each 64 rows of the operand 8 KB apart;
    // 16-byte chunks XORed with the row number (the 128-byte swizzle of the descriptors)
    __device__ __forceinline__ void store(uint32_t tile, uint32_t plane, int t) const
    {
        // group i lies istep * 128 bytes further in both layouts, and istep is a multiple of 8: the same chunk
        const int r = row_of(t), k = k_of(t);
        uint32_t at = tile + (MN ? (r >> 6) * (FK * 128) + k * 128 + ((((r & 63) >> 3) ^ (k & 7)) << 4) : r * 128 + (((k >> 3) ^ (r & 7)) << 4));
#pragma unroll
        for (int i = 0; i < N; ++i, at += istep * 128) {
            if constexpr (sizeof(T) == 2) {
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[i][0].x), "r"(v[i][0].y), "r"(v[i][0].z), "r"(v[i][0].w) : "memory");
            } else {
                float x[8];
                memcpy(x, &v[i][0], 16);
                memcpy(x + 4, &v[i][1], 16);
                uint64_t y[4];                                    // pairs: one instruction for two values
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j] = pack2(x[2 * j], x[2 * j + 1]);
#pragma unroll
                for (int pl = 0; pl < 3; ++pl) {
                    uint32_t h[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        unpack2(y[j], x[2 * j], x[2 * j + 1]);
                        h[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
                        if (pl < 2) y[j] = fma2(pack2(__uint_as_float(h[j] << 16), __uint_as_float(h[j] & 0xffff0000u)), pack2(-1.f, -1.f), y[j]);
                        if (pl == 0) y[j] = mul2(y[j], pack2(1 << F_SHIFT, 1 << F_SHIFT));
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + pl * plane), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
                }
            }
        }
    }
};

// 32 lanes x C columns of a TMEM accumulator added to a register row
template <int C> __device__ __forceinline__ void add_accumulator(uint32_t taddr, float (&acc)[C]);
template <> __device__ __forceinline__ void add_accumulator<32>(uint32_t taddr, float (&acc)[32])
{
    uint32_t r[32];
    tmem_ld32(taddr, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] += __uint_as_float(r[j]);
}
template <> __device__ __forceinline__ void add_accumulator<16>(uint32_t taddr, float (&acc)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(r[j]);
}

// BT: type of B (float: three planes, bf16: one).  CLUSTER: K split over the CTAs of a cluster, one tile per cluster.
template <typename BT, bool A_MN, bool B_MN, int BN, bool CLUSTER>
__global__ void __launch_bounds__(F_THREADS, 1) f32_gemm_kernel(const __grid_constant__ F32GemmParams p)
{
    constexpr int NB = sizeof(BT) == 4 ? 3 : 1;
    constexpr int PLANE_B = BN * FK * 2, STAGE = 3 * F_PLANE_A + NB * PLANE_B, STAGES = NB == 3 ? 2 : 3;
    constexpr int HC = BN / 4;                                    // columns of the tile a warp adds up
    constexpr uint32_t TMEM_COLS = 2 * BN;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(A_MN) << 15) | (uint32_t(B_MN) << 16) |
                               (uint32_t(BN >> 3) << 17) | (uint32_t(FM >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t tiles0 = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * STAGES, tfull0 = empty0 + 8 * STAGES, tempty0 = tfull0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = threadIdx.x;
    if (t == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 16); mbar_init(empty0 + 8 * s, 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull0 + 8 * a, 1); mbar_init(tempty0 + 8 * a, 16); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int tiles = p.tiles_m * p.tiles_n, units = tiles * p.batch;
    uint32_t rank = 0, ranks = 1;
    if (CLUSTER) {
        rank = cluster_ctarank();
        asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    }
    const int first = CLUSTER ? blockIdx.x / ranks : blockIdx.x, step = CLUSTER ? units : gridDim.x;
    const int kb0 = CLUSTER ? static_cast<int>(rank) * p.kb_per_split : 0, kb1 = CLUSTER ? min(p.kb_total, kb0 + p.kb_per_split) : p.kb_total;

    using FA = Frag<float, A_MN, FM>;
    using FB = Frag<BT, B_MN, BN>;
    FA fa;
    FB fb;
    // the operands of work unit u and this thread's first elements in them
    const float *A = nullptr, *mine_a = nullptr;
    const BT *B = nullptr, *mine_b = nullptr;
    int tm = 0, tn = 0, b = 0;
    auto open_unit = [&](int u) {
        b = u / tiles;
        const int tt = u - b * tiles;
        tn = tt / p.tiles_m; tm = tt - tn * p.tiles_m;
        A = p.A + b * p.batch_a;
        B = static_cast<const BT*>(p.B) + b * p.batch_b;
        const int ra = tm * FM + FA::row_of(t), rb = tn * BN + FB::row_of(t);
        mine_a = A + (A_MN ? FA::k_of(t) * p.lda + ra : ra * p.lda + FA::k_of(t));
        mine_b = B + (B_MN ? FB::k_of(t) * p.ldb + rb : rb * p.ldb + FB::k_of(t));
    };
    auto load_a = [&](int kb) { fa.load(A, mine_a, p.lda, tm * FM, p.M, kb * FK, p.K, p.a_vec, t); };
    auto load_b = [&](int kb) { fb.load(B, mine_b, p.ldb, tn * BN, p.N, kb * FK, p.K, p.b_vec, t); };
    if (first < units) { open_unit(first); load_a(kb0); load_b(kb0); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int q = warp & 3, colw = (warp >> 2) * HC;             // TMEM lanes 32 q.. (a warp reads those of its number modulo 4)
    const uint32_t my_tmem = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + colw;

    // A wait that gives up sets the abort flag, after which every other wait returns at once: the loops run to their end
    // with the same barriers on all warps, and this CTA writes nothing.  What it hands to the peers of a cluster is NaN, so that
    // they compute their results again instead of adding up an unfinished tile.
    int it = 0;
    for (int u = first; u < units; u += step) {
        float acc[HC];
#pragma unroll
        for (int j = 0; j < HC; ++j) acc[j] = 0.f;
        auto add_up = [&](int i) {                                // accumulator of block i: wait, add, hand the TMEM buffer back
            const int a = i & 1;
            mbar_wait(tfull0 + 8 * a, (i >> 1) & 1, abort_flag, 4, &g_f32gemm_error);
            __syncwarp();
            tc_fence_after();
            add_accumulator<HC>(my_tmem + a * BN, acc);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8 * a);
        };
        const int m0 = tm * FM + q * 32, n0 = tn * BN + colw, ub = b;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
            const int s = it % STAGES, a = it & 1;
            mbar_wait(empty0 + 8 * s, ((it / STAGES) & 1) ^ 1, abort_flag, 1, &g_f32gemm_error);
            const uint32_t ta = tiles0 + s * STAGE;
            // the next block's loads of one operand fly while the other operand is split and while this block is multiplied
            fa.store(ta, F_PLANE_A, t);
            if (kb + 1 < kb1) load_a(kb + 1);
            fb.store(ta + 3 * F_PLANE_A, PLANE_B, t);
            if (kb + 1 < kb1) load_b(kb + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
            if (t == 0 && mbar_wait(tempty0 + 8 * a, ((it >> 1) & 1) ^ 1, abort_flag, 2, &g_f32gemm_error) &&
                mbar_wait(full0 + 8 * s, (it / STAGES) & 1, abort_flag, 3, &g_f32gemm_error)) {
                tc_fence_after();
                const uint32_t a0 = ta, b0 = a0 + 3 * F_PLANE_A, d = tmem_base + a * BN;
                // plane pairs, the smallest products first.  The second and third planes are 2^15 too large, so mid * mid is by
                // 2^30, the others but hi * hi by 2^15: the accumulator is taken down twice by 2^15 on the way
                constexpr int PAIRS = NB == 3 ? 6 : 3;
                constexpr int PA[6] = {1, 2, 0, 1, 0, 0}, PB[6] = {1, 0, 2, 0, 1, 0}, QA[3] = {2, 1, 0};
#pragma unroll
                for (int w = 0; w < PAIRS; ++w) {
                    const uint32_t ap = a0 + (NB == 3 ? PA[w] : QA[w % 3]) * F_PLANE_A, bp = b0 + (NB == 3 ? PB[w] : 0) * PLANE_B;
#pragma unroll
                    for (int k = 0; k < FK / 16; ++k) {
                        const uint64_t da = A_MN ? smem_desc(ap + k * (16 * 128), FK * 128, 1024) : smem_desc(ap + k * 32, 16, 1024);
                        const uint64_t db = B_MN ? smem_desc(bp + k * (16 * 128), FK * 128, 1024) : smem_desc(bp + k * 32, 16, 1024);
                        const bool larger = NB == 3 ? w == 1 || w == 5 : w == 2;
                        if (k == 0 && larger) umma_bf16_shift<F_SHIFT>(d, da, db, IDESC);
                        else umma_bf16(d, da, db, IDESC, (w > 0 || k > 0) ? 1u : 0u);
                    }
                }
                umma_commit(empty0 + 8 * s);
                umma_commit(tfull0 + 8 * a);
            }
            __syncwarp();
            if (kb > kb0) add_up(it - 1);
        }
        if (u + step < units) { open_unit(u + step); load_a(kb0); load_b(kb0); }
        if (kb1 > kb0) add_up(it - 1);
        // every MMA has been waited for, so the operand stages are free for the sums on their way out
        if (CLUSTER) {
            float* part = reinterpret_cast<float*>(smem) + (q * 32 + lane) * (BN + 4) + colw;
            if (*abort_flag) {
#pragma unroll
                for (int j = 0; j < HC; ++j) acc[j] = __int_as_float(0x7fc00000);
            }
#pragma unroll
            for (int j = 0; j < HC; j += 4) *reinterpret_cast<float4*>(part + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        } else {
            // a warp's 32 x HC patch, read back with its lanes along the columns: 32 / HC rows per step
            float* patch = reinterpret_cast<float*>(smem) + warp * (32 * (HC + 1));
#pragma unroll
            for (int j = 0; j < HC; ++j) patch[lane * (HC + 1) + j] = acc[j];
            __syncwarp();
            const int c = lane % HC, n = n0 + c, rows = min(32, p.M - m0);
            if (n < p.N && !*abort_flag) {
                float* C = p.C + ub * p.batch_c;
                const float* R = p.residual ? p.residual + ub * p.batch_c : nullptr;
                const float bn = p.bias_n ? p.bias_n[n] : 0.f;
#pragma unroll 8
                for (int i = lane / HC; i < rows; i += 32 / HC) {
                    float x = patch[i * (HC + 1) + c];
                    if (!isfinite(x)) x = sgemm_exact<BT, A_MN, B_MN>(p, ub, m0 + i, n);
                    x = p.alpha * x + bn;
                    if (p.bias_m) x += p.bias_m[m0 + i];
                    const long long o = (m0 + i) * p.ldc + n;
                    if (R) x += R[o];
                    if (p.accumulate) x += C[o];
                    C[o] = x;
                }
            }
            __syncthreads();                                      // the next unit's operands overwrite the patches
        }
    }
    if (CLUSTER) {
        cluster_sync_all();                                       // every partial tile is in place
        if (!*abort_flag) {
            float* C = p.C + b * p.batch_c;
            constexpr int V = BN / 4;                             // float4 per row
            const int per = FM / ranks;                           // ranks is a power of two
            for (int i = t; i < per * V; i += F_THREADS) {
                const int r = rank * per + i / V, c = (i % V) * 4, m = tm * FM + r, n = tn * BN + c;
                if (m >= p.M || n >= p.N) continue;
                float4 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k < static_cast<int>(ranks))
                        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w)
                                     : "r"(mapa_shared(tiles0 + (r * (BN + 4) + c) * 4, k)));
                float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k < static_cast<int>(ranks)) { x[0] += v[k].x; x[1] += v[k].y; x[2] += v[k].z; x[3] += v[k].w; }
                const long long o = m * p.ldc + n;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (n + j >= p.N) break;
                    if (!isfinite(x[j])) x[j] = sgemm_exact<BT, A_MN, B_MN>(p, b, m, n + j);
                    float y = p.alpha * x[j] + (p.bias_n ? p.bias_n[n + j] : 0.f);
                    if (p.bias_m) y += p.bias_m[m];
                    if (p.residual) y += p.residual[b * p.batch_c + o + j];
                    if (p.accumulate) y += C[o + j];
                    C[o + j] = y;
                }
            }
        }
        cluster_sync_all();                                       // nobody's shared memory goes while a peer reads it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <typename BT, bool A_MN, bool B_MN, int BN, bool CLUSTER>
int launch_f32(const F32GemmParams& p, int splits, cudaStream_t s)
{
    constexpr int NB = sizeof(BT) == 4 ? 3 : 1;
    constexpr int STAGES_BYTES = (NB == 3 ? 2 : 3) * (3 * F_PLANE_A + NB * BN * FK * 2), SMEM = STAGES_BYTES + 256 + 1024;
    static_assert(SMEM <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
    static_assert(FM * (BN + 4) * 4 <= STAGES_BYTES && 16 * 32 * (BN / 4 + 1) * 4 <= STAGES_BYTES, "sums and patches lie in the operand stages");
    auto kernel = f32_gemm_kernel<BT, A_MN, B_MN, BN, CLUSTER>;
    static PerDeviceOnce once;
    NNB_TRY(once.run([kernel] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); }));
    const long long units = static_cast<long long>(p.tiles_m) * p.tiles_n * p.batch;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(CLUSTER ? units * splits : (units < device_sm_count() ? units : device_sm_count())));
    cfg.blockDim = dim3(F_THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CLUSTER ? 1 : 0;
    NNB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, p));
    NNB_LAUNCH_CHECK();
    return 0;
}

template <typename BT>
int f32_gemm(F32GemmParams& p, bool a_mn, bool b_mn, cudaStream_t s)
{
    if (p.M <= 0 || p.N <= 0 || p.batch <= 0) return 0;
    NNB_ARG_CHECK(p.K >= 0, "negative K");
    p.kb_total = static_cast<int>(ceil_div(p.K, FK));
    p.tiles_m = static_cast<int>(ceil_div(p.M, FM));
    // Tile width and K split.  Cost model in units of one 128 x 128 x 64 block: a tile of half the width costs 0.6 of
    // it (the A tile is loaded and split for half the work), a CTA's start, first loads and stores about three blocks.
    // Splits stay within the eight CTAs of a portable cluster and a single wave, so that all partial tiles run at once.
    // Against all widths and splits, timed at 24 shapes from 128 x 128 x 128 to 4096 x 512 x 4096: the choice is the best or
    // within 10 % at 22; 501 x 2304 x 768 takes 32 us where a split over 144 CTAs, which the three quarters leave out, takes
    // 24, and 900 x 700 x 500 takes 23 against 18.
    const int sms = device_sm_count();
    int bn = 128, splits = 1;
    double best = 1e30;
    for (int w = 64; w <= 128; w += 64) {
        const long long tiles = p.tiles_m * ceil_div(p.N, w) * p.batch;
        const double block = w == 128 ? 1.0 : 0.6;
        for (int sp = 1; sp <= 8 && (sp == 1 || (tiles * sp <= sms * 3 / 4 && p.kb_total / sp >= 1)); sp *= 2) {
            const double cost = sp == 1 ? static_cast<double>(ceil_div(tiles, sms)) * (p.kb_total * block + 1.0) + 2.0
                                        : ceil_div(p.kb_total, sp) * block + 4.0;
            if (cost < best - 1e-9) { best = cost; bn = w; splits = sp; }
        }
    }
    p.tiles_n = static_cast<int>(ceil_div(p.N, bn));
    NNB_ARG_CHECK(static_cast<long long>(p.tiles_m) * p.tiles_n * p.batch <= INT_MAX, "too many output tiles for one launch");
    p.kb_per_split = static_cast<int>(ceil_div(p.kb_total, splits));
#define GO(am, bm)                                                                       \
    do {                                                                                 \
        if (bn == 128) return splits > 1 ? launch_f32<BT, am, bm, 128, true>(p, splits, s) : launch_f32<BT, am, bm, 128, false>(p, 1, s); \
        return splits > 1 ? launch_f32<BT, am, bm, 64, true>(p, splits, s) : launch_f32<BT, am, bm, 64, false>(p, 1, s);                  \
    } while (0)
    if constexpr (sizeof(BT) == 2) {
        NNB_ARG_CHECK(!a_mn && !b_mn, "a bf16 second operand needs both operands contiguous along K");
        GO(false, false);
    } else {
        if (!a_mn && !b_mn) GO(false, false);
        if (!a_mn && b_mn) GO(false, true);
        if (a_mn && !b_mn) GO(true, false);
        GO(true, true);
    }
#undef GO
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// C[b][m*ldc + n] = alpha * sum_k A[b][m*sam + k*sak] * B[b][n*sbn + k*sbk]
//                   (+ bias_n[n]) (+ bias_m[m]) (+ residual[b][m*ldc + n]) (+ C if accumulate)
// each operand contiguous along one of its two indices
int sgemm_strided(const float* A, const float* B, float* C, int M, int N, int K,
                  long long sam, long long sak, long long sbn, long long sbk, long long ldc,
                  int batch, long long batch_a, long long batch_b, long long batch_c,
                  float alpha, const float* bias_n, const float* bias_m, const float* residual,
                  int accumulate, cudaStream_t stream)
{
    NNB_ARG_CHECK((sak == 1 || sam == 1) && (sbk == 1 || sbn == 1), "an operand must be contiguous along one of its indices");
    const bool a_mn = sak != 1, b_mn = sbk != 1;
    F32GemmParams p{};
    p.A = A; p.B = B; p.C = C; p.M = M; p.N = N; p.K = K; p.batch = batch;
    p.lda = a_mn ? sak : sam; p.ldb = b_mn ? sbk : sbn; p.ldc = ldc;
    p.batch_a = batch_a; p.batch_b = batch_b; p.batch_c = batch_c;
    p.a_vec = aligned16(A) && p.lda % 4 == 0 && batch_a % 4 == 0;
    p.b_vec = aligned16(B) && p.ldb % 4 == 0 && batch_b % 4 == 0;
    p.alpha = alpha; p.bias_n = bias_n; p.bias_m = bias_m; p.residual = residual; p.accumulate = accumulate;
    return f32_gemm<float>(p, a_mn, b_mn, stream);
}

// C[M, N] = A[M, K] B[N, K]^T (+ bias_n) (+ residual), A fp32, B bf16, C fp32, all rows contiguous
int gemm_f32_bf16(const float* A, const bf16* B, float* C, int M, int N, int K, const float* bias_n, const float* residual, cudaStream_t stream)
{
    F32GemmParams p{};
    p.A = A; p.B = B; p.C = C; p.M = M; p.N = N; p.K = K; p.batch = 1;
    p.lda = K; p.ldb = K; p.ldc = N;
    p.a_vec = aligned16(A) && K % 4 == 0;
    p.b_vec = aligned16(B) && K % 8 == 0;
    p.alpha = 1.0f; p.bias_n = bias_n; p.residual = residual;
    return f32_gemm<bf16>(p, false, false, stream);
}

int f32_gemm_device_error(int* code)
{
    NNB_CUDA_CHECK(cudaMemcpyFromSymbol(code, g_f32gemm_error, sizeof(int)));
    const int z = 0;
    if (*code) NNB_CUDA_CHECK(cudaMemcpyToSymbol(g_f32gemm_error, &z, sizeof(int)));
    return 0;
}

}  // namespace nnb

extern "C" int nnb200_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K,
                               long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major,
                               float alpha, const float* bias_n, const float* residual, int accumulate,
                               void* stream)
{
    // A is (M,K) with K contiguous (a_mn_major=0) or stored (K,M) with M contiguous (1);
    // B is (N,K) with K contiguous (b_mn_major=0) or stored (K,N) with N contiguous (1).
    return nnb::sgemm_strided(A, B, C, M, N, K, a_mn_major ? 1 : lda, a_mn_major ? lda : 1,
                              b_mn_major ? 1 : ldb, b_mn_major ? ldb : 1, ldc, 1, 0, 0, 0, alpha, bias_n,
                              nullptr, residual, accumulate, nnb::to_stream(stream));
}
