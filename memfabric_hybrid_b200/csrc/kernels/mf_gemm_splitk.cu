// bf16 GEMM for few rows (decode steps, small batches): C[M,N] = A[M,K] . B[N,K]^T with K split over a thread-block cluster.
//
// What bounds it: reading B once from memory. The persistent kernel of mf_gemm.cu gives one SM a whole 128 x 256 tile over all
// of K, so a layer with N = 7168 keeps 28 SMs busy and the other 120 idle. Measured with B from memory, launches from a CUDA graph (us,
// the persistent kernel's better tiling / this kernel): 32 x 7168 x 8192 43.1 / 22.6, 32 x 8192 x 3584 23.2 / 13.8, 1 x 1024 x 4096
// 23.8 / 5.6. Of the 22.6, 18.5 are the loads (6.3 TB/s; the first ones arrive after 2.3), 2.5 the exchange. Here a tile is 128 x 128 and the S
// CTAs of a cluster each take 1/S of K into their own tensor memory; the partial sums meet through distributed shared memory (every CTA adds up
// and stores 1/S of the tile, in CTA order: the result does not depend on timing). No workspace, no second launch.
// Two CTAs share an SM (about 100 KB of stages each), so one CTA's prologue and reduction run under the other's loads.
// A's box in the tensor map is only as high as the rows there are, rounded up to 8: the MMA still reads 128 rows of shared
// memory, and what the rows past the box hold ends up in accumulator rows that nobody reads. All of a CTA's A stages lie in
// front of its B stages, so those reads stay inside its shared memory.
// EPI 1 fuses SwiGLU: a tile is 64 gate rows and the 64 up rows that belong to them (B holds 128 gate rows, then their 128 up
// rows, per 256).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "mf_gemm.cuh"
#include "mf_launch.cuh"

namespace mfk {

constexpr int kSkBN = 128;
constexpr int kSkThreads = 192;              // warp 0 TMA, warp 1 MMA, warps 2..5 read the accumulator, all six reduce
constexpr int kSkMaxSplit = 8;               // portable cluster size
constexpr int kSkAtOnce = 4;                 // partial sums on their way to a thread at once, from which on items follow one another
constexpr int kSkStageArea = 100 * 1024;     // two CTAs per SM
constexpr int kSkRowFloats = kSkBN + 4;      // 528-byte rows: eight lanes' 16-byte writes to eight rows hit all banks once
constexpr int kSkMaxStages = kSkStageArea / (8 * KSPAN + kSkBN * KSPAN);  // A's box is at least 8 rows
static_assert(BM * kSkRowFloats * 4 <= kSkStageArea, "the partial tile reuses the stages");

struct SplitArgs {
    TmaPair tm;
    __nv_bfloat16 *C;
    int64_t ldc;
    int M, N, K;
    int box_rows;   // rows of A per stage (multiple of 8, at most 128)
    int stages;
    int *status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
// Every thread on its own (threads of a warp come to it at different places).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// This CTA's share of the tile: the S partial sums of four columns (with SwiGLU: four gate columns and their up projections) per item, added in CTA order.
// What bounds it: the way from the neighbours' shared memory. Lanes read 16 bytes side by side, a CTA's own part does not leave the SM, and the reads
// of several items are on their way at once. Before, a thread read 32 bytes with gaps, the own part the same way, one part after another: with a tile's
// 32 rows in 4 CTAs 2.9 us from the last partial tile to the end, 1.7 so; 128 rows in 2 CTAs 5.6, 4.2; gate/up and down product (N, K = 7168, 8192 and
// 8192, 3584) in a row, us before / so: 1 row 35.1 / 34.1, 32 rows 41.6 / 37.1, 64 46.1 / 39.7, 128 55.6 / 47.9, 256 60.8 / 57.4. With eight reads at once
// 1 % slower (the code of a short kernel is fetched cold), with sixteen 6 %; with two as fast, but 64 x 8192 x 1024 6.6 for 6.2.
template <int EPI, int S> __device__ __forceinline__ void add_up(const SplitArgs &g, uint32_t part0, __nv_bfloat16 *C, int rows, int nt, uint32_t rank, uint32_t split)
{
    constexpr int kOutCols = EPI == 1 ? kSkBN / 2 : kSkBN;   // output columns of the tile
    constexpr int kVecs = kOutCols / 4;
    constexpr int H = EPI == 1 ? 2 : 1;
    constexpr int P = S ? S : kSkMaxSplit, U = kSkAtOnce / P > 0 ? kSkAtOnce / P : 1;  // parts, items at once
    const int n_out = EPI == 1 ? g.N / 2 : g.N;
    const bool vec_ok = (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 7) == 0;
    const int total = rows * kVecs, step = (int)(S ? S : split) * kSkThreads;
    int it = (int)(rank * kSkThreads + threadIdx.x);
    if (it >= total) cluster_arrive();
    for (; it < total; it += U * step) {
        float4 v[U][P][H];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = it + u * step;
            if (i >= total) continue;
            const uint32_t at = part0 + (uint32_t)((i / kVecs) * kSkRowFloats + (i % kVecs) * 4) * 4;
#pragma unroll
            for (uint32_t p = 0; p < (uint32_t)P; p++) {
                if (S == 0 && p >= split) continue;
                const uint32_t from = mapa_u32(at, p);
#pragma unroll
                for (int h = 0; h < H; h++) v[u][p][h] = p == rank ? ld_shared_f4(at + (uint32_t)(h * (kSkBN / 2) * 4)) : ld_cluster_f4(from + (uint32_t)(h * (kSkBN / 2) * 4));
            }
        }
        float acc[U][H * 4];
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
            for (int e = 0; e < H * 4; e++) acc[u][e] = 0.f;
            if (it + u * step >= total) continue;
#pragma unroll
            for (uint32_t p = 0; p < (uint32_t)P; p++) {
                if (S == 0 && p >= split) continue;
#pragma unroll
                for (int h = 0; h < H; h++) {
                    acc[u][h * 4] += v[u][p][h].x;
                    acc[u][h * 4 + 1] += v[u][p][h].y;
                    acc[u][h * 4 + 2] += v[u][p][h].z;
                    acc[u][h * 4 + 3] += v[u][p][h].w;
                }
            }
        }
        // the last reads of the neighbours' tiles: they may go once all have arrived, while the stores below are on their way
        if (it + U * step >= total) cluster_arrive();
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = it + u * step;
            if (i >= total) continue;
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (EPI == 1) {
                    const float gt = acc[u][e], up = acc[u][H * 4 - 4 + e];
                    o[e] = gt / (1.f + __expf(-gt)) * up;
                } else {
                    o[e] = acc[u][e];
                }
            }
            const int col = nt * kOutCols + (i % kVecs) * 4;
            __nv_bfloat16 *dst = C + (int64_t)(i / kVecs) * g.ldc + col;
            if (vec_ok && col + 4 <= n_out) {
                uint2 pk;
                __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&pk);
                h[0] = __floats2bfloat162_rn(o[0], o[1]);
                h[1] = __floats2bfloat162_rn(o[2], o[3]);
                *reinterpret_cast<uint2 *>(dst) = pk;
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (col + e < n_out) dst[e] = __float2bfloat16_rn(o[e]);
            }
        }
    }
}

template <int EPI> __global__ void __launch_bounds__(kSkThreads, 2) k_gemm_bf16_splitk(const __grid_constant__ SplitArgs g)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bar_full[kSkMaxStages], bar_empty[kSkMaxStages], bar_done;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t split, rank;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(split));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int m_tiles = (g.M + BM - 1) / BM;
    const int tile = (int)(blockIdx.x / split);
    const int mt = tile % m_tiles, nt = tile / m_tiles;   // CTAs running together share B tiles
    const int k_iters = (g.K * 2 + KSPAN - 1) / KSPAN;
    const int k0 = (int)((int64_t)k_iters * rank / split), k1 = (int)((int64_t)k_iters * (rank + 1) / split);
    const int a_bytes = g.box_rows * KSPAN;
    constexpr int kBBytes = kSkBN * KSPAN;
    uint8_t *b_base = base + g.stages * a_bytes;
    AbortCtl ac{&abort_flag, g.status};

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < g.stages; s++) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_empty[s], 1);
        }
        mbar_init(&bar_done, 1);
        mbar_fence_init();
        tma_prefetch_desc(&g.tm.a);
        tma_prefetch_desc(&g.tm.b);
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, kSkBN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    after_predecessor();  // everything above ran under the kernel in front of this one
    start_successor();

    // rows of B of this tile: two runs of 64
    int b0, b1;
    if (EPI == 1) {
        b0 = (nt >> 1) * 256 + (nt & 1) * 64;
        b1 = b0 + 128;
    } else {
        b0 = nt * kSkBN;
        b1 = b0 + 64;
    }
    bool have = false;
    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            for (int kb = k0; kb < k1; kb++) {
                if (!mbar_wait(&bar_empty[s], phase ^ 1, ac, 0x311)) break;
                mbar_expect_tx(&bar_full[s], (uint32_t)(a_bytes + kBBytes));
                tma_load_2d(b_base + s * kBBytes, &g.tm.b, kb * (KSPAN / 2), b0, &bar_full[s]);
                tma_load_2d(b_base + s * kBBytes + kBBytes / 2, &g.tm.b, kb * (KSPAN / 2), b1, &bar_full[s]);
                tma_load_2d(base + s * a_bytes, &g.tm.a, kb * (KSPAN / 2), mt * BM, &bar_full[s]);
                if (++s == g.stages) s = 0, phase ^= 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            bool fine = true;
            const uint32_t idesc = umma_idesc(1, 1, BM, kSkBN);
            for (int kb = k0; kb < k1; kb++) {
                fine = mbar_wait(&bar_full[s], phase, ac, 0x312);
                if (!fine) break;
                tc_fence_after();
                const uint64_t da = umma_desc_sw128(base + s * a_bytes);
                const uint64_t db = umma_desc_sw128(b_base + s * kBBytes);
#pragma unroll
                for (int k = 0; k < KSPAN / 32; k++) umma_bf16(tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb != k0) | (k != 0));
                umma_commit(&bar_empty[s]);
                if (++s == g.stages) s = 0, phase ^= 1;
            }
            if (fine) umma_commit(&bar_done);
        }
        __syncwarp();
    } else {
        // the four warps read one lane quadrant each and leave the partial sums as fp32 rows where the stages were: all
        // loads have landed and all MMAs have read them once bar_done completes
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        have = __all_sync(0xffffffffu, mbar_wait(&bar_done, 0, ac, 0x313));
        if (have) {
            tc_fence_after();
            if (quad * 32 < g.M - mt * BM) {  // uniform over the warp: the reads below are collective
                float *mine = reinterpret_cast<float *>(base) + row * kSkRowFloats;
#pragma unroll
                for (int c = 0; c < kSkBN / 64; c++) {
                    uint32_t v[2][32];
                    tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * 64), v[0]);
                    tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * 64 + 32), v[1]);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 16; q++) {
                        const uint32_t *w = v[q / 8] + q % 8 * 4;
                        *reinterpret_cast<uint4 *>(mine + c * 64 + q * 4) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            tc_fence_before();
        }
    }
    __syncwarp();
    cluster_sync_all();  // every CTA's partial tile is in its shared memory (every CTA arrives: the waits above are bounded)
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kSkBN);
    }

    const int rows = min(BM, g.M - mt * BM);
    const uint32_t part0 = smem_u32(base);
    __nv_bfloat16 *C = g.C + (int64_t)mt * BM * g.ldc;
    switch (split) {
        case 1: add_up<EPI, 1>(g, part0, C, rows, nt, rank, split); break;
        case 2: add_up<EPI, 2>(g, part0, C, rows, nt, rank, split); break;
        case 4: add_up<EPI, 4>(g, part0, C, rows, nt, rank, split); break;
        default: add_up<EPI, 0>(g, part0, C, rows, nt, rank, split); break;
    }
    cluster_wait();  // nobody leaves while a peer still reads its partial tile
}

}  // namespace mfk

using namespace mfk;

namespace {

constexpr int kSkDynBytes = kSkStageArea + 1024;

template <int EPI> bool splitk_ready()
{
    // with the carve-out that holds two CTAs per SM
    static const bool ok = cudaFuncSetAttribute(k_gemm_bf16_splitk<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSkDynBytes) == cudaSuccess &&
                           cudaFuncSetAttribute(k_gemm_bf16_splitk<EPI>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                                cudaSharedmemCarveoutMaxShared) == cudaSuccess;
    return ok;
}

int split_tiles(int M, int N) { return ((M + BM - 1) / BM) * ((N + kSkBN - 1) / kSkBN); }
int split_k_iters(int K) { return (K * 2 + KSPAN - 1) / KSPAN; }
int split_box_rows(int M) { return std::min(BM, (M + 7) / 8 * 8); }

}  // namespace

extern "C" {

// CTAs that share a tile: 1, 2, 4 or 8 (clusters of 3, 5, 6 leave more of a GPC unused and were slower throughout).
// Cost in steps of K (64 elements of a 128 x 128 tile), for rounds of resident clusters: two CTAs per SM; clusters of two fit
// everywhere, of the larger ones a tenth does not fit the rest of a GPC. A round takes K / s steps, or what memory takes for all
// tiles' steps (1.35 steps per SM at a time), and its exchange: a barrier, what grows with the rows and with how many CTAs exchange at once, and
// most of all whether clusters share their SMs (a cluster's slowest CTA counts: 17 tiles in clusters of eight, 6 x 2624 x 1856, 6.5, in clusters of
// four 5.6; 16 tiles, 3 x 2016 x 2432, 5.9, 5.9; of 128 rows and K 4096, clusters of four / eight: 15 tiles 10.5 / 9.3, 16 10.6 / 11.4, 17 10.7 / 12.1, 24 11.6 / 13.1). The constants fit
// 181 products of 1 - 1024 rows, 1 - 74 tiles of 128 x 256 and K 512 - 8192 (launches from a graph, weights from memory), and what clusters of eight share 350 more of 8 to
// 40 tiles and 8 to 1024 rows: the choice is 0.3 % from the best of the four on average, 10 % at most (with one penalty for any number of rows 1 % and 26 %: 947 x 304 x 7040 in clusters of eight 14.1, of four 11.2).
// Measured (us, persistent kernels' better tiling | s = 1, 2, 4, 8): 32 x 7168 x 8192 43.1 | 34.3, 24.3, 22.6, 27.9; 1 x 1024 x 4096 23.8 |
// 16.9, 10.1, 6.8, 5.6; 128 x 1024 x 8192 41.9 | 47.5, 26.4, 16.1, 11.8; 256 x 4096 x 8192 43.2 | 48.2, 28.7, 22.7, 33.6; 256 x 9216 x 8192 44.8 | 52.0,
// 41.0, 58.9, 74.4; 1024 x 2304 x 16384 79.2 | 93.2, 66.4, 90.6, 101; 1024 x 1280 x 1024 10.0 | 9.5, 9.8, 15.0, 25.9.
int mf_gemm_bf16_split(int M, int N, int K, int sms)
{
    const int tiles = split_tiles(M, N), k_iters = split_k_iters(K), n = sms > 0 ? sms : 148;
    const double memory = (double)tiles * k_iters / (1.35 * n);
    double best = 0;
    int split = 0;
    for (int s = 1; s <= kSkMaxSplit && s <= k_iters; s *= 2) {
        const double resident = (s <= 2 ? 2.0 : 1.8) * n / s;
        const double rounds = std::ceil(tiles / std::max(1.0, std::floor(resident)));
        const double busy = std::min(1.0, (double)tiles * s / (2.0 * n));
        const double rows = (double)split_box_rows(M) / BM, edge = std::floor(resident / 2);
        // clusters of eight share SMs from one tile earlier on, half of them at first, and share more between them the more rows they exchange
        const double shared = s < 8 ? (tiles > edge ? 5.25 : 0.0) : (tiles > edge ? 1.0 : tiles == edge ? 0.5 : 0.0) * (6 + 8 * rows);
        const double exchange = s > 1 ? 1.7 + 1.8 * s * rows * busy + shared : 0.0;
        const double cost = std::max(rounds * ((k_iters + s - 1) / s), memory) + rounds * (0.3 * s + exchange);
        if (split == 0 || cost < best) {
            best = cost;
            split = s;
        }
    }
    return split;
}

// Same contract as mf_gemm_bf16_one. split: CTAs per tile (1..8), 0: chosen here.
int mf_gemm_bf16_splitk(const void *A, const void *B, void *C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc, int *status,
                        int sms, int swiglu, int split, void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || (K & 7) != 0 || split < 0 || split > kSkMaxSplit) return -1;
    if (swiglu && (N % 256) != 0) return -3;
    if (!(swiglu ? splitk_ready<1>() : splitk_ready<0>()) || !splitk_ready<0>()) {
        (void)cudaGetLastError();
        return -2;
    }
    SplitArgs g{};
    g.box_rows = split_box_rows(M);
    int rc = make_tmap_2d(&g.tm.a, A, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, (uint32_t)g.box_rows, false);
    if (rc == 0) rc = make_tmap_2d(&g.tm.b, B, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, kSkBN / 2, false);
    if (rc != 0) return rc;
    g.C = static_cast<__nv_bfloat16 *>(C);
    g.ldc = ldc;
    g.M = M;
    g.N = N;
    g.K = K;
    g.status = status;
    g.stages = std::min(kSkMaxStages, kSkStageArea / (g.box_rows * KSPAN + kSkBN * KSPAN));
    const int tiles = split_tiles(M, N), k_iters = split_k_iters(K);
    if (split == 0) split = mf_gemm_bf16_split(M, N, K, sms);
    if (split > k_iters) return -1;
    const cudaError_t e = launch_overlapped(swiglu ? k_gemm_bf16_splitk<1> : k_gemm_bf16_splitk<0>, dim3((unsigned)(tiles * split)), dim3(kSkThreads),
                                            kSkDynBytes, (cudaStream_t)stream, (unsigned)split, g);
    return e == cudaSuccess ? 0 : (int)e;
}

}  // extern "C"
