// Grouped expert GEMM in fp8 e4m3 on CTA pairs; the block scales are applied by the tensor core (kind::mxf8f6f4.block_scale).
//   activations X [rows, K] fp8, one power-of-two fp32 scale per row per 128 elements of K      (1 x 128)
//   weights     W [experts, N, K] fp8, one power-of-two fp32 scale per 128 x 128 block          (128 x 128)
//   rows grouped by expert: group g owns rows [row_off[g], row_off[g+1]) (device array, no host sync)
//
// The WEIGHTS are the M side of the MMA (256 rows of W per tile, 128 in each CTA of the pair, always full) and the rows of X its
// N side, whose size the instruction takes in steps: a group's rows are cut into tiles of equal width, a multiple of 32 and at
// most 224. With the rows on the M side (tiles of 128 rows) 32 experts of about 1 024 rows computed 6 % of rows that nobody has,
// and a decode batch of 32 rows per expert four times its rows, fetched through the L2 with every block of weights.
// The two CTAs share a tile's X rows: each fetches half of them and the MMA reads both halves (cta_group::2). A stage is 16 KiB of W and
// at most 14 KiB of X per CTA (48 KiB before), so six stages fit, ten when no tile is wider than 32; two accumulators of
// 224 columns fit beside the scales in tensor memory, so a tile's epilogue runs under the next tile's MMAs.
//
// What bounds it: few rows per expert, the weights from HBM (6.5 TB/s); many, the power limit (tensor pipe and operand traffic); few K
// blocks, the epilogue. 32 experts, N x K 4096 x 7168 (EPI 3) and 7168 x 2048 (EPI 0), us, tiles of 128 rows x 256 on single CTAs / this kernel:
// about 32 rows per expert 166 / 144 and 86 / 82, 128 rows 201 / 172 and 104 / 93, 256 rows 261 / 257 and 150 / 143, 1024 rows 760 / 730 and
// 438 / 390. Slower than those tiles: one expert of about 1 024 rows (4096 x 7168: 28.7 / 33.5; 128 tiles are one round of single CTAs, but two
// of pairs, each of half a tile's work), and 75 to 148 tiles of few rows (5 experts of 20 rows, 4096 x 2048, EPI 0: 13.6 / 15.1).
//
// The scales must be powers of two (every quantiser of this library produces such scales): a producer warp turns them into UE8M0 bytes
// (the fp32 exponent) in the tensor core's layout in shared memory, four K blocks per 32-bit word; the leader's MMA thread
// copies a group of them into both CTAs' tensor memory (tcgen05.cp) and picks the byte of the K block through the instruction descriptor.
// Warps: 0 TMA, 1 MMA (leader; + TMEM allocation), 2 and 3 scale producers, 4..11 epilogue (two per TMEM lane quadrant, alternate 32-row chunks).
// Accumulators are transposed: a TMEM lane is an output column (a row of W), a TMEM column is a row of X.
// Epilogues (rows leave through shared memory, so that a row's columns are stored in contiguous pieces):
//   EPI 0  plain            : bf16 rows to local memory
//   EPI 1  gate/up + SwiGLU : W is tile-interleaved (128 gate rows, 128 up rows per 256); out[row, 128 cols] bf16. The TMA box takes the
//                             two kinds in alternate runs of 16 rows, so that a warp holds a gate column and its up column 16 lanes apart
//   EPI 2  down + combine   : row x routing weight stored straight into the combine slot of the token's home
//                             rank (peer stores over NVLink)
//   EPI 3  gate/up + SwiGLU + re-quantisation: the 128 outputs of a tile row are one 1 x 128 block of the next GEMM's fp8 input; its
//                             maximum is put together from the eight lane quadrants of the two CTAs (distributed shared memory)
// Parity of role: app/zbal/doc/fused_deep_moe.md:106-127,213-281 (GMM1 -> dequant + SwiGLU + dynamic re-quant
// -> GMM2 -> combine) of the reference.
#include <cuda_bf16.h>

#include "mf_fp8.cuh"
#include "mf_gemm.cuh"
#include "mf_launch.cuh"
#include "mf_team.cuh"

namespace mfk {

constexpr int kPThreads = 384;
constexpr int kPMaxGroups = 64;
constexpr int kGran = 32;        // rows of X per step of a tile's width
constexpr int kMaxGran = 7;      // widest tile: 224 rows, two accumulators and the scale columns fill the tensor memory
constexpr int kMaxWidth = kGran * kMaxGran;
constexpr int kPTileN = 256;     // rows of W per tile
constexpr int kPMaxStages = 12;
constexpr int kSfSpan = 16;      // K blocks whose scales are handed over at once
constexpr int kPSfBufs = 2;
constexpr uint32_t kPTmemCols = 512;
constexpr uint32_t kPSfaCol = 2 * kMaxWidth;  // TMEM columns [448, 452): scales of W; [452, 460): scales of X
constexpr uint32_t kPSfbCol = kPSfaCol + 4;

struct PSmem {
    static constexpr int kABytes = BM * KSPAN;
    static constexpr int kBStep = kGran / 2 * KSPAN;          // this CTA's half of 32 rows of X
    static constexpr int kRing = 6 * (kABytes + kMaxGran * kBStep);
    static constexpr int kSfOff = kRing;
    static constexpr int kSfChunk = 512 + 1024;               // four K blocks: W chunk, two X chunks
    static constexpr int kSfBufBytes = kSfSpan / 4 * kSfChunk;
    static constexpr int kBarOff = kSfOff + kPSfBufs * kSfBufBytes;
    static constexpr int kAmaxOff = kBarOff + 512;            // [2 parities][8 quadrants of the pair][224] floats
    static constexpr int kOutOff = kAmaxOff + 2 * 8 * kMaxWidth * 4;
    static constexpr int kOutRowB = 272;                      // 128 bf16 + 16: row reads of 16 lanes x 16 bytes without conflicts
    static constexpr int kOutSet = kGran * kOutRowB;          // one chunk of 32 rows per set of four epilogue warps
    static constexpr int kTotal = kOutOff + 2 * kOutSet;
    static constexpr int kDynBytes = kTotal + 1024;
    uint8_t *base;
    int stage_bytes = 0, stages = 0;
    __device__ explicit PSmem(uint8_t *raw) : base(reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023)) {}
    __device__ uint8_t *a(int s) const { return base + s * stage_bytes; }
    __device__ uint8_t *b(int s) const { return base + s * stage_bytes + kABytes; }
    __device__ uint8_t *sf(int i) const { return base + kSfOff + i * kSfBufBytes; }
    __device__ uint64_t *bar(int i) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + i; }
    __device__ uint64_t *full(int s) const { return bar(s); }
    __device__ uint64_t *empty(int s) const { return bar(kPMaxStages + s); }
    __device__ uint64_t *sf_full(int i) const { return bar(2 * kPMaxStages + i); }
    __device__ uint64_t *sf_empty(int i) const { return bar(2 * kPMaxStages + kPSfBufs + i); }
    __device__ uint64_t *tfull(int i) const { return bar(2 * kPMaxStages + 2 * kPSfBufs + i); }
    __device__ uint64_t *tempty(int i) const { return bar(2 * kPMaxStages + 2 * kPSfBufs + 2 + i); }
    __device__ uint64_t *amax_full(int i) const { return bar(2 * kPMaxStages + 2 * kPSfBufs + 4 + i); }
    __device__ uint32_t *tmem_slot() const { return reinterpret_cast<uint32_t *>(base + kBarOff + 384); }
    __device__ volatile int *abort_flag() const { return reinterpret_cast<volatile int *>(base + kBarOff + 392); }
    __device__ float *amax(int parity) const { return reinterpret_cast<float *>(base + kAmaxOff) + parity * 8 * kMaxWidth; }
    __device__ uint8_t *out_stage(int set) const { return base + kOutOff + set * kOutSet; }
};
static_assert((2 * kPMaxStages + 2 * kPSfBufs + 6) * 8 <= 384, "barriers of the pair fp8 GEMM");
static_assert(PSmem::kDynBytes <= 227 * 1024, "shared memory of the pair fp8 GEMM");

struct alignas(64) PArgs {
    CUtensorMap w;         // [G * N, K] fp8: 2-D, 128-row boxes; SwiGLU epilogues: 5-D, boxes of alternate 16-row runs
    CUtensorMap x[3];      // [rows, K] fp8: boxes of 16, 32 and 64 rows
    const float *x_scale;  // [rows, K/128]
    const float *w_scale;  // [G, N/128, K/128]  (N in ORIGINAL row order: for EPI 1/3 gate rows then up rows)
    const int *row_off;    // [G + 1] device
    int G, N, K;
    int max_rows;
    void *out;             // EPI 0/1: bf16; EPI 3: e4m3 bytes
    int64_t ldo;           // elements per output row
    float *out_scale;      // EPI 3: [rows, N/256]
    int *status;
    Team team;             // EPI 2
    const int4 *recv_info;
    uint64_t comb_off;
    int topk;
    uint32_t *done_count;  // EPI 2, optional: local counter of finished CTAs, zero between launches
    uint64_t flag_off;     // EPI 2: slot offset of the flag row that the last CTA raises to `epoch` on every peer
    uint32_t epoch;        // flag value of this call (grows by one per call)
};

__device__ __forceinline__ void p_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// The same barrier, and whether `ok` held for all its threads: what follows a wait that may give up has to be the same for all of them.
__device__ __forceinline__ bool p_bar_all(int id, int threads, bool ok)
{
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %3, 0;\n\t"
        "bar.red.and.pred p, %1, %2, q;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(all)
        : "r"(id), "r"(threads), "r"(ok ? 1 : 0)
        : "memory");
    return all != 0;
}

__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t v) { return *reinterpret_cast<const __nv_bfloat162 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) { return as_u32(__floats2bfloat162_rn(lo, hi)); }

// silu(gate) * up as every other SwiGLU epilogue of the library has it, with its division: the same activations round to the same bytes whichever
// kernel takes a layer's shape.
__device__ __forceinline__ float swiglu(float gate, float up) { return gate / (1.f + __expf(-gate)) * up; }

// The same value for |gate| < 80, where the divisor lies in [1, 2^116) and nothing overflows, without the branches that the general division has:
// a reciprocal with one Newton step, a quotient, and the quotient corrected by its exact remainder, which rounds it as the division
// does (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, 1990). The quotient depends on the gate alone and
// has been compared with the division for every float (mf_swiglu_debug_probe). A warp divides where one of its gates is out of the range.
// Re-quantising epilogue, 32 experts of about 512 rows, N 4096, us, division / so / approximate reciprocal: K 512 140 / 110 / 104, 2048 163 / 143 /
// 141, 4096 258 / 252 / 251 (tiles of 128 x 256 rows on single CTAs: 110, 147, 261).
__device__ __forceinline__ bool swiglu_in_range(float gate) { return fabsf(gate) < 80.f; }
__device__ __forceinline__ float swiglu_fast(float gate, float up)
{
    const float d = 1.f + __expf(-gate);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = __fmaf_rn(__fmaf_rn(-d, r, 1.f), r, r);
    const float q = __fmul_rn(gate, r);
    return __fmaf_rn(-__fmaf_rn(d, q, -gate), r, q) * up;  // the remainder as d * q - gate: a gate of -0 keeps its sign
}

// Debug aid: counts the gates among `count` bit patterns from `first` on whose two quotients differ.
__global__ void k_swiglu_probe(uint32_t first, uint64_t count, unsigned long long *differ)
{
    unsigned long long bad = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        const float gate = __uint_as_float(first + (uint32_t)i);
        if (swiglu_in_range(gate) && __float_as_uint(swiglu_fast(gate, 1.f)) != __float_as_uint(swiglu(gate, 1.f))) bad++;
    }
    if (bad != 0) atomicAdd(differ, bad);
}

// The first `have` (at most four) of the scales at s as they lie in memory, 1.0 for the others. `vec`: s is 16-byte aligned and `have` a multiple of
// four. Predicated loads: with a branch around each, the next one waited for the one in front of it.
__device__ __forceinline__ void load_scales(const float *s, int have, bool vec, uint32_t (&f)[4])
{
    asm volatile(
        "{\n\t.reg .pred v, p0, p1, p2, p3;\n\t.reg .b32 m;\n\t"
        "mov.b32 %0, 0x3f800000;\n\tmov.b32 %1, 0x3f800000;\n\tmov.b32 %2, 0x3f800000;\n\tmov.b32 %3, 0x3f800000;\n\t"
        "setp.ne.s32 v, %6, 0;\n\t"
        "setp.gt.and.s32 p0, %5, 0, v;\n\t"
        "@p0 ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n\t"
        "selp.b32 m, 0, %5, v;\n\t"
        "setp.gt.s32 p0, m, 0;\n\t"
        "setp.gt.s32 p1, m, 1;\n\t"
        "setp.gt.s32 p2, m, 2;\n\t"
        "setp.gt.s32 p3, m, 3;\n\t"
        "@p0 ld.global.b32 %0, [%4];\n\t"
        "@p1 ld.global.b32 %1, [%4 + 4];\n\t"
        "@p2 ld.global.b32 %2, [%4 + 8];\n\t"
        "@p3 ld.global.b32 %3, [%4 + 12];\n\t}"
        : "=&r"(f[0]), "=&r"(f[1]), "=&r"(f[2]), "=&r"(f[3])
        : "l"(s), "r"(have), "r"((int)vec)
        : "memory");
}

// The exponent bytes (UE8M0) of four floats.
__device__ __forceinline__ uint32_t exponents(const uint32_t (&f)[4])
{
    return __byte_perm(__byte_perm(f[0] << 1, f[1] << 1, 0x0073), __byte_perm(f[2] << 1, f[3] << 1, 0x0073), 0x5410);
}

// Ring position for a number of slots known at run time.
struct RingState {
    int slot = 0;
    uint32_t phase = 0;
    __device__ void advance(int slots)
    {
        if (++slot == slots) {
            slot = 0;
            phase ^= 1;
        }
    }
};

// Cut of a group's `steps` runs of 32 rows into `cnt` tiles whose widths differ by one run at most: tile mi starts at run `first` and is `gran`
// runs wide. No product of a tile's number and the runs: in 32 bits that overflows at 3.9 M rows.
__host__ __device__ inline void p_tile_cut(int steps, int cnt, int mi, int &first, int &gran)
{
    const int each = steps / cnt, wider = steps - each * cnt;
    first = mi * each + (mi < wider ? mi : wider);
    gran = each + (mi < wider ? 1 : 0);
}

struct PTile {
    int grp = 0;    // walks forward with the tiles
    int row0, row_end, gran, nt;
};

template <int EPI> __global__ void __launch_bounds__(kPThreads, 1) k_grouped_fp8_mx(const __grid_constant__ PArgs g)
{
    constexpr bool kSwiGLU = EPI == 1 || EPI == 3;
    extern __shared__ uint8_t smem_raw[];
    PSmem sm(smem_raw);
    __shared__ int tile_start[kPMaxGroups + 1];
    __shared__ int s_row_off[kPMaxGroups + 1];
    __shared__ int s_gran;  // widest tile of this launch is at most this many steps
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const int walker = (int)(blockIdx.x >> 1), walkers = (int)(gridDim.x >> 1);
    const int n_tiles = g.N / kPTileN;
    const int k_blocks = g.K / 128;
    const int sf_spans = (k_blocks + kSfSpan - 1) / kSfSpan;
    AbortCtl ac{sm.abort_flag(), g.status};

    if (threadIdx.x == 0) {
        *sm.abort_flag() = 0;
        for (int s = 0; s < kPMaxStages; s++) {
            mbar_init(sm.full(s), 1);
            mbar_init(sm.empty(s), 1);
        }
        for (int i = 0; i < kPSfBufs; i++) {
            mbar_init(sm.sf_full(i), 4);   // the scale producers of both CTAs (counted in the leader)
            mbar_init(sm.sf_empty(i), 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(sm.tfull(i), 1);
            mbar_init(sm.tempty(i), 16);   // the epilogue warps of both CTAs (counted in the leader)
            mbar_init(sm.amax_full(i), 16);  // the epilogue warps of both CTAs, and the bytes that the peer's send
        }
        mbar_fence_init();
        tma_prefetch_desc(&g.w);
        for (int i = 0; i < 3; i++) tma_prefetch_desc(&g.x[i]);
    }
    if (warp == 1) {
        tmem_alloc_pair(sm.tmem_slot(), kPTmemCols);
        tmem_relinquish_pair();
    }
    // Barriers, tensor memory and descriptors were set up under the kernel in front of this one. The kernel behind it gets no early
    // start, which costs (its CTAs would take SMs in the order in which these become free; presumably neighbouring tiles then share less
    // in the L2). MoE layer, early start / none, us: 128 tokens 272 / 268, 512: 328 / 317, 1024: 508 / 498, 4096: 1363 / 1330.
    after_predecessor();
    if (warp == 2) {
        for (int i = lane; i <= g.G; i += 32) s_row_off[i] = min(g.row_off[i], g.max_rows);
        __syncwarp();
        // Width of the tiles: at most m steps for one m of the launch, the one whose rounds of tiles over the pairs take least. A tile
        // of w rows takes w + 64 units: 64 is what fetching 256 rows of W costs when it outlasts the MMAs. The widest one is taken unless
        // another is 2 % better. With many experts that is nearly always the answer; it is the dense expert of few rows that gains. One expert, us,
        // seven steps always / so: 4096 x 7168 (EPI 3) 512 rows 22.5 / 21.3, 1024 40.5 / 33.5, 2048 54.7 / 53.5; 7168 x 2048 (EPI 0) 512 rows 14.7 / 14.1.
        // Lane m weighs m: in a loop over m the search took 1.3 us of every launch.
        const int st0 = lane < g.G ? max(0, (s_row_off[lane + 1] - s_row_off[lane] + kGran - 1) / kGran) : 0;
        const int st1 = lane + 32 < g.G ? max(0, (s_row_off[lane + 33] - s_row_off[lane + 32] + kGran - 1) / kGran) : 0;
        int steps = 0, tiles = 0, widest = 1;
#pragma unroll
        for (int m = 1; m <= kMaxGran; m++) {
            const int n = __reduce_add_sync(0xffffffffu, (st0 + m - 1) / m + (st1 + m - 1) / m);
            if (m == 1) steps = n;
            if (lane == m) tiles = n;
        }
        float cost = 3.4e38f;
        if (tiles > 0) {
            const int rounds = (tiles * n_tiles + walkers - 1) / walkers;
            cost = (float)rounds * ((float)steps * (float)kGran / (float)tiles + 64.f) * (lane == kMaxGran ? 0.98f : 1.f);
        }
        const uint32_t least = __reduce_min_sync(0xffffffffu, __float_as_uint(cost));  // positive floats are ordered as their bits
        const int best_m = 31 - __clz((int)__ballot_sync(0xffffffffu, lane >= 1 && lane <= kMaxGran && __float_as_uint(cost) == least));
        int run = 0;
        for (int h = 0; h * 32 < g.G; h++) {
            const int st = h == 0 ? st0 : st1;
            const int n = (st + best_m - 1) / best_m;
            widest = max(widest, n > 0 ? (st + n - 1) / n : 0);
            int upto = n * n_tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += below;
            }
            if (h * 32 + lane < g.G) tile_start[h * 32 + lane] = run + upto - n * n_tiles;
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        widest = __reduce_max_sync(0xffffffffu, widest);
        if (lane == 0) {
            tile_start[g.G] = run;
            s_gran = widest;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers are initialised and both halves of the tensor memory are allocated
    tc_fence_after();
    const uint32_t tmem_base = *sm.tmem_slot();
    const int total = tile_start[g.G];
    sm.stage_bytes = PSmem::kABytes + s_gran * PSmem::kBStep;
    sm.stages = min(kPMaxStages, PSmem::kRing / sm.stage_bytes);

    // linear tile -> group, rows, 256 rows of W; inside a group the rows vary fastest. Calls come with growing t.
    auto locate = [&](int t, PTile &p) {
        while (tile_start[p.grp + 1] <= t) p.grp++;
        const int lo = s_row_off[p.grp], hi = s_row_off[p.grp + 1];
        const int local = t - tile_start[p.grp];
        const int cnt = (tile_start[p.grp + 1] - tile_start[p.grp]) / n_tiles;
        const int steps = (hi - lo + kGran - 1) / kGran;
        p.nt = local / cnt;
        const int mi = local - p.nt * cnt;
        int first;
        p_tile_cut(steps, cnt, mi, first, p.gran);
        p.row0 = lo + first * kGran;
        p.row_end = hi;
    };

    if (warp == 0) {
        if (elect_one()) {
            RingState ps;
            PTile p;
            bool fine = true;
            for (int t = walker; t < total && fine; t += walkers) {
                locate(t, p);
                const uint32_t bytes = 2u * (uint32_t)(PSmem::kABytes + p.gran * PSmem::kBStep);
                const int xrow = p.row0 + (int)crank * p.gran * (kGran / 2);
                for (int kb = 0; kb < k_blocks; kb++) {
                    fine = mbar_wait(sm.empty(ps.slot), ps.phase ^ 1, ac, 0x602);
                    if (!fine) break;
                    // both CTAs' bytes are counted on the leader's barrier
                    if (crank == 0) mbar_expect_tx(sm.full(ps.slot), bytes);
                    const uint32_t lead = mapa_u32(smem_u32(sm.full(ps.slot)), 0);
                    if (kSwiGLU) tma_load_5d_pair(sm.a(ps.slot), &g.w, kb * 128, 0, 0, 4 * (int)crank, p.grp * n_tiles + p.nt, lead);
                    else tma_load_2d_pair(sm.a(ps.slot), &g.w, kb * 128, p.grp * g.N + p.nt * kPTileN + (int)crank * BM, lead);
                    uint8_t *dst = sm.b(ps.slot);
                    int row = xrow;
#pragma unroll
                    for (int i = 2; i >= 0; i--) {
                        if (p.gran & (1 << i)) {
                            tma_load_2d_pair(dst, &g.x[i], kb * 128, row, lead);
                            dst += PSmem::kBStep << i;
                            row += (kGran / 2) << i;
                        }
                    }
                    ps.advance(sm.stages);
                }
            }
        }
    } else if (warp == 1) {
        if (crank == 0 && elect_one()) {
            RingState ps, sf;
            PTile p;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool fine = true;
            const uint32_t sfa = tmem_base + kPSfaCol, sfb = tmem_base + kPSfbCol;
            for (int t = walker; t < total && fine; t += walkers) {
                locate(t, p);
                fine = mbar_wait<true>(sm.tempty(acc), acc_phase ^ 1, ac, 0x603);  // both CTAs' epilogues have taken this accumulator out of TMEM
                if (!fine) break;
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(acc * kMaxWidth);
                const uint32_t width = (uint32_t)(p.gran * kGran);
                for (int kb = 0; kb < k_blocks; kb++) {
                    if (kb % kSfSpan == 0) {
                        fine = mbar_wait<true>(sm.sf_full(sf.slot), sf.phase, ac, 0x606);
                        if (!fine) break;
                        tc_fence_after();
                    }
                    if ((kb & 3) == 0) {
                        const uint8_t *chunk = sm.sf(sf.slot) + (kb % kSfSpan) / 4 * PSmem::kSfChunk;
                        tmem_cp_sf_pair(sfa, umma_desc_sf(chunk));
                        tmem_cp_sf_pair(sfb, umma_desc_sf(chunk + 512));
                        if (width > 128) tmem_cp_sf_pair(sfb + 4, umma_desc_sf(chunk + 1024));
                    }
                    fine = mbar_wait(sm.full(ps.slot), ps.phase, ac, 0x604);
                    if (!fine) break;
                    tc_fence_after();
                    const uint64_t da = umma_desc_sw128(sm.a(ps.slot));
                    const uint64_t db = umma_desc_sw128(sm.b(ps.slot));
                    const uint32_t idesc = umma_idesc_bs(2 * BM, width, (uint32_t)(kb & 3), (uint32_t)(kb & 3));
#pragma unroll
                    for (int k = 0; k < 4; k++)  // 32 bytes = 32 fp8 = one UMMA K step
                        umma_fp8_bs_pair(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb | k) != 0, sfa, sfb);
                    const uint32_t e = smem_u32(sm.empty(ps.slot));
                    umma_commit_pair(e);  // the stage is free in both CTAs once these MMAs have read it
                    umma_commit_pair(mapa_u32(e, 1));
                    ps.advance(sm.stages);
                    if (kb % kSfSpan == kSfSpan - 1 || kb == k_blocks - 1) {
                        const uint32_t se = smem_u32(sm.sf_empty(sf.slot));
                        umma_commit_pair(se);  // the scales have been copied and their MMAs are done
                        umma_commit_pair(mapa_u32(se, 1));
                        sf.advance(kPSfBufs);
                    }
                }
                if (!fine) break;
                const uint32_t f = smem_u32(sm.tfull(acc));
                umma_commit_pair(f);
                umma_commit_pair(mapa_u32(f, 1));
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else if (warp < 4) {
        // scale producers: one 32-bit word of four K-block scale bytes per operand row; the two warps take alternate words. Lane l writes the
        // 16 bytes of rows l, l + 32, l + 64, l + 96 of a chunk: this CTA's 128 rows of W, and all rows of X. The scales of 16 K blocks go
        // over at once. Each CTA's tensor core copies its own chunks, but the leader has both do it, so the other CTA's bytes are
        // released to the cluster: the proxy fence, then a release of shared memory alone. A full release waits for the SM's outstanding
        // loads as well: 32 experts of about 32 rows, 4096 x 7168: 161 us with it, 149.4 so (148.4 without any order), 227 with a full release
        // per four K blocks.
        // A tile of few K blocks takes as long as its scales: two warps, and all loads of a span issued before the first is used, without
        // branches between them. 32 experts of about 512 rows, N 4096, EPI 0, us, one warp that branches between aligned and single loads /
        // so: K 128 77 / 49, 384 87 / 52, 512 56 / 54, 768 120 / 66, 1024 79 / 78 (tiles of 128 x 256 on single CTAs: 56, 61, 62, 73, 86).
        const int part = warp - 2;
        RingState sf;
        PTile p;
        const int nblocks = g.N / 128;
        const bool vec = (k_blocks & 3) == 0 && ((reinterpret_cast<uintptr_t>(g.x_scale) | reinterpret_cast<uintptr_t>(g.w_scale)) & 15) == 0;
        bool fine = true;
        for (int t = walker; t < total && fine; t += walkers) {
            locate(t, p);
            // the 128-row block of W: SwiGLU: gate rows nt * 128 .. in lanes 0-15, up rows N/2 + nt * 128 .. in lanes 16-31
            const int nb = kSwiGLU ? (lane < 16 ? p.nt : nblocks / 2 + p.nt) : 2 * p.nt + (int)crank;
            const float *ws = g.w_scale + ((int64_t)p.grp * nblocks + nb) * k_blocks;
            const float *xs[kMaxGran];
#pragma unroll
            for (int i = 0; i < kMaxGran; i++) xs[i] = g.x_scale + (int64_t)min(p.row0 + i * kGran + lane, g.max_rows - 1) * k_blocks;
            for (int sp = 0; sp < sf_spans; sp++) {
                uint32_t raw[kSfSpan / 8][kMaxGran + 1][4], wrd[kSfSpan / 8][kMaxGran + 1];  // [..][kMaxGran]: W
#pragma unroll
                for (int h = 0; h < kSfSpan / 8; h++) {
                    const int kb = sp * kSfSpan + (2 * h + part) * 4;
#pragma unroll
                    for (int i = 0; i <= kMaxGran; i++) load_scales((i < kMaxGran ? xs[i] : ws) + kb, i < kMaxGran && i >= p.gran ? 0 : k_blocks - kb, vec, raw[h][i]);
                }
#pragma unroll
                for (int h = 0; h < kSfSpan / 8; h++)
#pragma unroll
                    for (int i = 0; i <= kMaxGran; i++) wrd[h][i] = exponents(raw[h][i]);
                int ok = 1;
                if (lane == 0) ok = mbar_wait(sm.sf_empty(sf.slot), sf.phase ^ 1, ac, 0x607) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                __syncwarp();  // what lane 0 has waited for holds for all lanes
                if (!ok) {
                    fine = false;
                    break;
                }
#pragma unroll
                for (int h = 0; h < kSfSpan / 8; h++) {
                    uint8_t *chunk = sm.sf(sf.slot) + (2 * h + part) * PSmem::kSfChunk;
                    const uint32_t w = wrd[h][kMaxGran];
                    *reinterpret_cast<uint4 *>(chunk + lane * 16) = make_uint4(w, w, w, w);
                    *reinterpret_cast<uint4 *>(chunk + 512 + lane * 16) = make_uint4(wrd[h][0], wrd[h][1], wrd[h][2], wrd[h][3]);
                    *reinterpret_cast<uint4 *>(chunk + 1024 + lane * 16) = make_uint4(wrd[h][4], wrd[h][5], wrd[h][6], 0x7f7f7f7fu);
                }
                fence_proxy_async_smem();  // the tensor core's copy unit reads these bytes through the async proxy
                __syncwarp();
                if (lane == 0) {
                    if (crank == 0) mbar_arrive(sm.sf_full(sf.slot));
                    else mbar_arrive_cluster_smem(mapa_u32(smem_u32(sm.sf_full(sf.slot)), 0));
                }
                sf.advance(kPSfBufs);
            }
        }
    } else if (warp >= 4) {
        // eight epilogue warps: warp w reads TMEM lane quadrant w % 4 (the hardware's rule); the two sets of four take alternate
        // chunks of 32 rows of X
        const int quad = warp & 3;
        const int set = (warp - 4) >> 2;
        constexpr int kChunks = (kMaxGran + 1) / 2;
        PTile p;
        int acc = 0;
        uint32_t acc_phase = 0;
        int flip = 0;  // EPI 3: which half of the staging buffer
        uint8_t *stg = sm.out_stage(set);
        for (int t = walker; t < total; t += walkers) {
            locate(t, p);
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * kMaxWidth);
            // lane = row of a chunk: where it goes (0: nowhere)
            unsigned long long dst[kChunks];
            float wgt[kChunks];
#pragma unroll
            for (int i = 0; i < kChunks; i++) {
                const int row = p.row0 + (set + 2 * i) * kGran + lane;
                dst[i] = 0;
                wgt[i] = 1.f;
                if (set + 2 * i < p.gran && row < p.row_end) {
                    if (EPI == 2) {
                        const int4 info = g.recv_info[row];
                        wgt[i] = __int_as_float(info.w);
                        dst[i] = reinterpret_cast<unsigned long long>(reinterpret_cast<__nv_bfloat16 *>(peer_ptr(g.team, (uint32_t)info.x, g.comb_off)) +
                                                                      ((int64_t)info.y * g.topk + info.z) * g.N + p.nt * kPTileN + (int)crank * 128);
                    } else if (EPI == 0) {
                        dst[i] = reinterpret_cast<unsigned long long>(static_cast<__nv_bfloat16 *>(g.out) + (int64_t)row * g.ldo + p.nt * kPTileN + (int)crank * 128);
                    } else if (EPI == 1) {
                        dst[i] = reinterpret_cast<unsigned long long>(static_cast<__nv_bfloat16 *>(g.out) + (int64_t)row * g.ldo + p.nt * 128 + (int)crank * 64);
                    } else {
                        dst[i] = reinterpret_cast<unsigned long long>(static_cast<uint8_t *>(g.out) + (int64_t)row * g.ldo + p.nt * 128 + (int)crank * 64);
                    }
                }
            }
            if (!p_bar_all(1 + set, 128, mbar_wait(sm.tfull(acc), acc_phase, ac, 0x605))) break;
            tc_fence_after();
            auto release = [&]() {  // this warp has read its part of the accumulator
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (crank == 0) mbar_arrive(sm.tempty(acc));
                    else mbar_arrive_cluster_smem(mapa_u32(smem_u32(sm.tempty(acc)), 0));
                }
            };
            const int last = p.gran > set ? (p.gran - 1 - set) / 2 : -1;  // index of this set's last chunk
            if (last < 0) release();
            // A chunk arrives as fragments of 8 x 8 matrices (thread: columns of the output lane / 4 and lane / 4 + 8 of a 16-lane half, rows
            // 8i + 2 (lane % 4) + e of the chunk), so that stmatrix can turn it around.
            if (!kSwiGLU) {
#pragma unroll
                for (int i = 0; i < kChunks; i++) {
                    if (i > last) continue;
                    uint32_t v[2][16];
                    tmem_ld_frag(taddr + (uint32_t)((set + 2 * i) * kGran), v[0]);
                    tmem_ld_frag(taddr + (16u << 16) + (uint32_t)((set + 2 * i) * kGran), v[1]);
                    tmem_ld_wait();
                    if (i == last) release();
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        float w[2] = {1.f, 1.f};
                        if (EPI == 2) {
                            w[0] = __shfl_sync(0xffffffffu, wgt[i], 8 * c + 2 * (lane & 3));
                            w[1] = __shfl_sync(0xffffffffu, wgt[i], 8 * c + 2 * (lane & 3) + 1);
                        }
                        uint32_t h[4];  // columns 0-7, 8-15, 16-23, 24-31 of this warp's 32
#pragma unroll
                        for (int m = 0; m < 4; m++)
                            h[m] = pack_bf16(__uint_as_float(v[m >> 1][4 * c + 2 * (m & 1)]) * w[0], __uint_as_float(v[m >> 1][4 * c + 2 * (m & 1) + 1]) * w[1]);
                        stmatrix_x4_trans(stg + (8 * c + (lane & 7)) * PSmem::kOutRowB + (quad * 32 + (lane >> 3) * 8) * 2, h[0], h[1], h[2], h[3]);
                    }
                    p_bar_sync(1 + set, 128);
                    // 2 rows x 256 contiguous bytes per instruction: over NVLink a write carries up to 256 bytes of payload
#pragma unroll
                    for (int it = 0; it < 4; it++) {
                        const int r = quad * 8 + it * 2 + (lane >> 4);
                        const unsigned long long d = __shfl_sync(0xffffffffu, dst[i], r);
                        const uint4 val = *reinterpret_cast<const uint4 *>(stg + r * PSmem::kOutRowB + (lane & 15) * 16);
                        if (d != 0) *reinterpret_cast<uint4 *>(d + (unsigned long long)((lane & 15) * 16)) = val;
                    }
                    p_bar_sync(1 + set, 128);
                }
            } else {
                uint32_t ob[kChunks][8];  // this thread's outputs as bf16: [2c + h] rows 8c + 2 (lane % 4), + 1 of the chunk, column quad * 16 + lane / 4 + 8h
#pragma unroll
                for (int i = 0; i < kChunks; i++) {
                    if (i > last) continue;
                    uint32_t gt[16], up[16];
                    tmem_ld_frag(taddr + (uint32_t)((set + 2 * i) * kGran), gt);
                    tmem_ld_frag(taddr + (16u << 16) + (uint32_t)((set + 2 * i) * kGran), up);
                    tmem_ld_wait();
                    if (i == last) release();
                    bool in_range = true;
#pragma unroll
                    for (int j = 0; j < 16; j++) in_range = in_range && swiglu_in_range(__uint_as_float(gt[j]));
                    if (__all_sync(0xffffffffu, in_range)) {
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            ob[i][j] = pack_bf16(swiglu_fast(__uint_as_float(gt[2 * j]), __uint_as_float(up[2 * j])),
                                                 swiglu_fast(__uint_as_float(gt[2 * j + 1]), __uint_as_float(up[2 * j + 1])));
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            ob[i][j] = pack_bf16(swiglu(__uint_as_float(gt[2 * j]), __uint_as_float(up[2 * j])),
                                                 swiglu(__uint_as_float(gt[2 * j + 1]), __uint_as_float(up[2 * j + 1])));
                    }
                    if (EPI == 1) {
#pragma unroll
                        for (int c = 0; c < 4; c += 2)
                            stmatrix_x4_trans(stg + (8 * (c + (lane >> 4)) + (lane & 7)) * 144 + (quad * 16 + ((lane >> 3) & 1) * 8) * 2, ob[i][2 * c],
                                              ob[i][2 * c + 1], ob[i][2 * c + 2], ob[i][2 * c + 3]);
                        p_bar_sync(1 + set, 128);
#pragma unroll
                        for (int it = 0; it < 2; it++) {
                            const int r = quad * 8 + it * 4 + (lane >> 3);
                            const unsigned long long d = __shfl_sync(0xffffffffu, dst[i], r);
                            const uint4 val = *reinterpret_cast<const uint4 *>(stg + r * 144 + (lane & 7) * 16);
                            if (d != 0) *reinterpret_cast<uint4 *>(d + (unsigned long long)((lane & 7) * 16)) = val;
                        }
                        p_bar_sync(1 + set, 128);
                    } else {
                        // maxima over this warp's 16 columns: two in the thread, then over lane / 4, two rows at a time
                        __nv_bfloat162 m[4];
#pragma unroll
                        for (int c = 0; c < 4; c++) m[c] = __hmax2(__habs2(as_bf162(ob[i][2 * c])), __habs2(as_bf162(ob[i][2 * c + 1])));
                        const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0;
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            const __nv_bfloat162 got = as_bf162(__shfl_xor_sync(0xffffffffu, as_u32(b4 ? m[c] : m[c + 2]), 16));
                            m[c] = __hmax2(b4 ? m[c + 2] : m[c], got);
                        }
                        m[0] = __hmax2(b3 ? m[1] : m[0], as_bf162(__shfl_xor_sync(0xffffffffu, as_u32(b3 ? m[0] : m[1]), 8)));
                        m[0] = __hmax2(m[0], as_bf162(__shfl_xor_sync(0xffffffffu, as_u32(m[0]), 4)));
                        const float2 both = __bfloat1622float2(m[0]);
                        const float part = fmaxf((lane & 4) != 0 ? both.y : both.x, 0.f);  // a NaN counts as nothing
                        const int row = (b4 ? 16 : 0) + (b3 ? 8 : 0) + 2 * (lane & 3) + ((lane >> 2) & 1);
                        float *slot = sm.amax(acc) + (int)(crank * 4 + quad) * kMaxWidth + (set + 2 * i) * kGran + row;
                        *slot = part;
                        st_async_f32(mapa_u32(smem_u32(slot), crank ^ 1), part, mapa_u32(smem_u32(sm.amax_full(acc)), crank ^ 1));
                    }
                }
                if (EPI == 3) {
                    // the eight partial maxima of every row of the tile: this CTA's and the peer's warps
                    __syncwarp();
                    if (lane == 0) {
                        // four floats (a lane quadrant each) for every row come from the peer
                        if (set == 0 && quad == 0) mbar_expect_tx(sm.amax_full(acc), (uint32_t)(p.gran * kGran * 16));
                        else mbar_arrive(sm.amax_full(acc));
                        mbar_arrive_cluster_smem(mapa_u32(smem_u32(sm.amax_full(acc)), crank ^ 1));
                    }
                    if (!p_bar_all(1 + set, 128, mbar_wait<true>(sm.amax_full(acc), acc_phase, ac, 0x60A))) break;
                    // The buffer of this parity is written again for the tile after the next, by warps that have passed the next tile's barrier:
                    // every warp of the pair has contributed to that one after it has read this tile's maxima.
#pragma unroll
                    for (int i = 0; i < kChunks; i++) {
                        if (i > last) continue;
                        const float *col = sm.amax(acc) + (set + 2 * i) * kGran + lane;
                        float amax = 0.f;
#pragma unroll
                        for (int q = 0; q < 8; q++) amax = fmaxf(amax, col[q * kMaxWidth]);
                        const float scale = pow2_scale_e4m3(amax);
                        const float inv = 1.f / scale;  // exact: a power of two
                        if (crank == 0 && quad == 0 && dst[i] != 0)
                            g.out_scale[(int64_t)(p.row0 + (set + 2 * i) * kGran + lane) * n_tiles + p.nt] = scale;
                        uint8_t *buf = stg + flip * (kGran * 80);
                        flip ^= 1;
                        uint8_t *mine = buf + 2 * (lane & 3) * 80 + quad * 16 + (lane >> 2);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const float m0 = __shfl_sync(0xffffffffu, inv, 8 * c + 2 * (lane & 3)), m1 = __shfl_sync(0xffffffffu, inv, 8 * c + 2 * (lane & 3) + 1);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const float2 f = __bfloat1622float2(as_bf162(ob[i][2 * c + h]));
                                const __nv_fp8x2_storage_t q = __nv_cvt_float2_to_fp8x2(make_float2(f.x * m0, f.y * m1), __NV_SATFINITE, __NV_E4M3);
                                mine[8 * c * 80 + 8 * h] = (uint8_t)q;
                                mine[(8 * c + 1) * 80 + 8 * h] = (uint8_t)(q >> 8);
                            }
                        }
                        p_bar_sync(1 + set, 128);  // two halves take turns: one barrier per chunk
                        const int r = quad * 8 + (lane >> 2);
                        const unsigned long long d = __shfl_sync(0xffffffffu, dst[i], r);
                        const uint4 val = *reinterpret_cast<const uint4 *>(buf + r * 80 + (lane & 3) * 16);
                        if (d != 0) *reinterpret_cast<uint4 *>(d + (unsigned long long)((lane & 3) * 16)) = val;
                    }
                }
            }
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // nobody signals a barrier of a CTA that has left, and both halves of the tensor memory are freed together
    if (EPI == 2) {
        // The CTA that finishes last tells every rank that all of this rank's rows are home: the CTA barrier orders the CTA's stores before thread 0, whose fence
        // and count hand them to the last CTA's, whose system fence covers all of them; the flags need no order of their own.
        if (threadIdx.x == 0 && g.done_count != nullptr) {
            __threadfence();
            if (atomicAdd(g.done_count, 1u) + 1 == gridDim.x) {
                *g.done_count = 0;
                fence_group(g.team);
                for (uint32_t r = 0; r < g.team.world; r++)
                    asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(reinterpret_cast<uint32_t *>(peer_ptr(g.team, r, g.flag_off)) + g.team.rank), "r"(g.epoch)
                                 : "memory");
            }
        }
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, kPTmemCols);
    }
}

}  // namespace mfk

using namespace mfk;

namespace {
template <int EPI> int launch_pairs(const PArgs &g, int sms, cudaStream_t s)
{
    auto kern = k_grouped_fp8_mx<EPI>;
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PSmem::kDynBytes) != cudaSuccess) {
            (void)cudaGetLastError();
            return -2;
        }
        attr_set = true;
    }
    const unsigned grid = sms < 2 ? 2u : (unsigned)sms & ~1u;  // whole clusters
    const cudaError_t e = launch_overlapped(kern, dim3(grid), dim3(kPThreads), PSmem::kDynBytes, s, 2, g);
    return e == cudaSuccess ? 0 : (int)e;
}
}  // namespace

extern "C" {

// 1 when the block-scaled kernels take this shape (the caller guarantees power-of-two scales).
int mf_grouped_gemm_fp8_mx_supported(int G, int N, int K, int epi)
{
    if (G <= 0 || G > kPMaxGroups || N <= 0 || K <= 0 || (N % kPTileN) != 0 || (K % 128) != 0) return 0;
    return epi >= 0 && epi <= 3;
}

// The cut of a group's rows into tiles, as the kernels make it: tile `mi` of `cnt` starts at run `*first` of 32 rows and takes `*gran` of them.
void mf_grouped_gemm_fp8_mx_cut(int steps, int cnt, int mi, int *first, int *gran) { p_tile_cut(steps, cnt, mi, *first, *gran); }

// Debug aid: how many of `count` floats, by their bits from `first` on, get another quotient from the SwiGLU epilogue's own division than from the
// general one; `differ` is a device word that the count is added to.
int mf_swiglu_debug_probe(uint32_t first, uint64_t count, void *differ, void *stream)
{
    k_swiglu_probe<<<1184, 256, 0, (cudaStream_t)stream>>>(first, count, static_cast<unsigned long long *>(differ));
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// epi: 0 plain (out bf16 [rows, N]), 1 SwiGLU (out bf16 [rows, N/2]), 2 weighted push into the combine slots of the
// tokens' home ranks, 3 SwiGLU + fp8 re-quantisation (out e4m3 [rows, N/2], out_scale fp32 [rows, N/256]).
// epi 2 with a done_count (a device word, zero between launches): the kernel's last CTA raises this rank's flag in row `which` of
// the flag area at `flags` of every slot to `epoch`, as mf_moe_signal_all does.
int mf_grouped_gemm_fp8_mx_signal(const void *A, const float *a_scale, int max_rows, const void *B, const float *b_scale, const int *row_off, int G,
                                  int N, int K, void *out, int64_t ldo, float *out_scale, int epi, const Team *team, const void *recv_info,
                                  uint64_t comb_off, int topk, uint32_t *done_count, uint64_t flags, int which, uint32_t epoch, int *status,
                                  int sms, void *stream)
{
    if (!mf_grouped_gemm_fp8_mx_supported(G, N, K, epi) || max_rows <= 0) return -1;
    if (epi == 2 && (team == nullptr || recv_info == nullptr)) return -1;
    if (epi == 3 && (out_scale == nullptr || (ldo & 15) != 0)) return -1;
    PArgs g{};
    int rc = epi == 1 || epi == 3 ? make_tmap_runs16(&g.w, B, (uint64_t)G * N, (uint64_t)K)
                                  : make_tmap_2d(&g.w, B, 1, (uint64_t)G * N, (uint64_t)K, (uint64_t)K, BM, true);
    for (int i = 0; i < 3 && rc == 0; i++)
        rc = make_tmap_2d(&g.x[i], A, 1, (uint64_t)max_rows, (uint64_t)K, (uint64_t)K, (uint32_t)(kGran / 2) << i, true);
    if (rc != 0) return rc;
    g.x_scale = a_scale;
    g.w_scale = b_scale;
    g.row_off = row_off;
    g.G = G;
    g.N = N;
    g.K = K;
    g.max_rows = max_rows;
    g.out = out;
    g.ldo = ldo;
    g.out_scale = out_scale;
    g.status = status;
    if (team != nullptr) g.team = *team;
    g.recv_info = static_cast<const int4 *>(recv_info);
    g.comb_off = comb_off;
    g.topk = topk;
    g.done_count = done_count;
    g.flag_off = flags + (uint64_t)which * kMaxRanks * sizeof(uint32_t);
    g.epoch = epoch;
    cudaStream_t s = (cudaStream_t)stream;
    switch (epi) {
        case 0: return launch_pairs<0>(g, sms, s);
        case 1: return launch_pairs<1>(g, sms, s);
        case 2: return launch_pairs<2>(g, sms, s);
        case 3: return launch_pairs<3>(g, sms, s);
        default: return -1;
    }
}

int mf_grouped_gemm_fp8_mx(const void *A, const float *a_scale, int max_rows, const void *B, const float *b_scale, const int *row_off, int G,
                           int N, int K, void *out, int64_t ldo, float *out_scale, int epi, const Team *team, const void *recv_info,
                           uint64_t comb_off, int topk, int *status, int sms, void *stream)
{
    return mf_grouped_gemm_fp8_mx_signal(A, a_scale, max_rows, B, b_scale, row_off, G, N, K, out, ldo, out_scale, epi, team, recv_info, comb_off,
                                         topk, nullptr, 0, 0, 0, status, sms, stream);
}

}  // extern "C"
