// Shared pieces of the tcgen05 GEMM kernels: host-side tensor-map creation, the shared-memory
// pipeline layout and the three warp roles' loop skeletons.
//   warp 0      TMA producer   : fills a ring of (A tile, B tile) stages, one mbarrier pair per stage
//   warp 1      MMA issuer     : one elected thread issues tcgen05.mma into a TMEM accumulator and
//                                commits completion to the stage's "empty" barrier / the tile's "full" barrier
//   warps 2..5  epilogue       : tcgen05.ld the accumulator (each warp its own 32-lane quadrant), apply
//                                the fused epilogue, store
// Operands are K-major ("TN": A[M,K], B[N,K], the layout of activations x nn.Linear weights); tiles are
// 128 x BN x 64 bytes-of-K-per-row = one 128-byte swizzle span per row.
#pragma once
#include <cuda_bf16.h>

#include "mf_umma.cuh"

namespace mfk {

constexpr int BM = 128;          // tile rows (UMMA M, one TMEM lane per row)
constexpr int KSPAN = 128;       // bytes of K per stage row = the 128-byte swizzle span
constexpr int kGemmThreads = 192;

struct alignas(64) TmaPair {
    CUtensorMap a;
    CUtensorMap b;
};

// dynamic shared memory: [stage][A 16 KiB | B BROWS*128 B] then barriers. BROWS = BN, or BN / 2 where a CTA pair shares the tile
template <int BN, int STAGES, int BROWS = BN> struct GemmSmem {
    static constexpr int kABytes = BM * KSPAN;
    static constexpr int kBBytes = BROWS * KSPAN;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kBarOff = STAGES * kStageBytes;
    // epilogue staging: each of the 4 epilogue warps turns 32 rows x 64 columns of bf16 around (one row per lane
    // out of TMEM -> 128 contiguous bytes per row on the way to memory); rows are padded to 144 bytes so that
    // both the per-lane row writes and the 8-lanes-per-row reads are free of bank conflicts
    static constexpr int kOutRowBytes = 144;
    static constexpr int kOutWarpBytes = 32 * kOutRowBytes;
    static constexpr int kOutOff = kBarOff + 1024;
    static constexpr int kOutBytes = 20480;  // >= 4 x kOutWarpBytes (bf16 GEMM) and >= 8 x 32 x 80 (fp8 GEMM, 8 warps x 32 columns)
    static constexpr int kTotal = kOutOff + kOutBytes;
    uint8_t *base;
    __device__ explicit GemmSmem(uint8_t *raw) : base(reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023)) {}
    __device__ uint8_t *a(int s) const { return base + s * kStageBytes; }
    __device__ uint8_t *b(int s) const { return base + s * kStageBytes + kABytes; }
    __device__ uint64_t *full(int s) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + s; }
    __device__ uint64_t *empty(int s) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + STAGES + s; }
    __device__ uint64_t *tfull(int i) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + 2 * STAGES + i; }
    __device__ uint64_t *tempty(int i) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + 2 * STAGES + 4 + i; }
    __device__ uint32_t *tmem_slot() const { return reinterpret_cast<uint32_t *>(base + kBarOff + 512); }
    __device__ uint8_t *out_stage(int epi_warp) const { return base + kOutOff + epi_warp * kOutWarpBytes; }
    __device__ volatile int *abort_flag() const { return reinterpret_cast<volatile int *>(base + kBarOff + 520); }
    static constexpr int kDynBytes = kTotal + 1024;  // slack for the 1024-byte alignment
};

struct PipeState {
    int stage = 0;
    uint32_t phase = 0;
    template <int STAGES> __device__ void advance()
    {
        if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
        }
    }
};

// Second half of GEMM -> reduce-scatter: adds the `world` partial tiles (bf16) of one owned tile in rank order, scales and stores.
// `land` points at rank 0's partial of the tile's first vector, `part` is the distance between the ranks' partials, rows are
// `ld` elements apart; the tile has BM rows of `vec_row` 16-byte vectors. What bounds it is memory latency: with 1, 2, 4 and 8 ranks a
// thread keeps eight loads in flight (8 / W vectors of W partials each), with any other number below 8 one vector, that is
// as many loads as there are ranks. One vector at a time, a tile took as many latencies as a thread has vectors. GEMM and reduction
// as one rank of W (4096 x 8192 outputs of the group, K 3584, the peers' partials landed before; us, one vector at a time / now):
// bf16 W = 1 301 / 187, 2 244 / 180, 4 205 / 178, 8 186 / 185-191; fp8 178 / 128, 150 / 121, 129 / 122, 119-130 / 122-128.
template <int W>
__device__ __forceinline__ void add_partials(const __nv_bfloat16 *land, int64_t part, int64_t ld, int vec_row, int world, float scale,
                                             __nv_bfloat16 *out, int64_t ldo)
{
    constexpr int V = W > 0 ? 8 / W : 1;  // vectors per step
    constexpr int S = W > 0 ? W : 8;      // partials per batch
    const int total = BM * vec_row, stride = (int)blockDim.x, ranks = W > 0 ? W : world;
    for (int v0 = threadIdx.x; v0 < total; v0 += stride * V) {
        uint4 raw[V][S];
        auto load = [&](int s0) {
#pragma unroll
            for (int u = 0; u < V; u++) {
                const int v = v0 + u * stride;
                const __nv_bfloat16 *from = land + (int64_t)(v / vec_row) * ld + (v % vec_row) * 8;
#pragma unroll
                for (int k = 0; k < S; k++)
                    if (v < total && s0 + k < ranks) raw[u][k] = __ldcg(reinterpret_cast<const uint4 *>(from + (int64_t)(s0 + k) * part));
            }
        };
        load(0);
#pragma unroll
        for (int u = 0; u < V; u++) {
            const int v = v0 + u * stride;
            if (v >= total) break;
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int s0 = 0;;) {
#pragma unroll
                for (int k = 0; k < S; k++) {
                    if (s0 + k >= ranks) continue;
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[u][k]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float2 f = __bfloat1622float2(h[e]);
                        acc[2 * e] += f.x;
                        acc[2 * e + 1] += f.y;
                    }
                }
                s0 += S;
                if (W > 0 || s0 >= ranks) break;  // more ranks than one batch: one vector at a time
                load(s0);
            }
            uint4 pk;
            __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
            for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(acc[2 * e] * scale, acc[2 * e + 1] * scale);
            *reinterpret_cast<uint4 *>(out + (int64_t)(v / vec_row) * ldo + (v % vec_row) * 8) = pk;
        }
    }
}
__device__ __forceinline__ void add_partials(const __nv_bfloat16 *land, int64_t part, int64_t ld, int vec_row, int world, float scale,
                                             __nv_bfloat16 *out, int64_t ldo)
{
    switch (world) {
        case 1: return add_partials<1>(land, part, ld, vec_row, world, scale, out, ldo);
        case 2: return add_partials<2>(land, part, ld, vec_row, world, scale, out, ldo);
        case 4: return add_partials<4>(land, part, ld, vec_row, world, scale, out, ldo);
        default: return add_partials<0>(land, part, ld, vec_row, world, scale, out, ldo);
    }
}

// Host: 2-D tensor map over a row-major [rows, cols_bytes / elem] matrix, box = (KSPAN bytes, box_rows), 128B swizzle.
int make_tmap_2d(CUtensorMap *out, const void *base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t row_stride_bytes,
                 uint32_t box_rows, bool is_fp8);

// Host: 5-D tensor map over a row-major fp8 [rows, cols] matrix whose rows alternate in runs of 128 of two kinds (gate, up). A box is 64
// rows of each kind in turns of 16: coordinates (column, 0, 0, first 16-row run inside the 128, block of 256 rows), 128B swizzle.
int make_tmap_runs16(CUtensorMap *out, const void *base, uint64_t rows, uint64_t cols);

}  // namespace mfk
