// The two tensor-parallel fusions in fp8 e4m3, whose block scales are applied by the tensor core itself
// (tcgen05.mma kind::mxf8f6f4.block_scale): the whole K loop of a tile accumulates in ONE TMEM buffer and
// nothing is pulled out of TMEM per K block. (The grouped expert GEMM is in mf_gemm_fp8_pair.cu.)
//   activations A [rows, K] fp8, one power-of-two fp32 scale per row per 128 elements of K      (1 x 128)
//   weights     B [N, K] fp8, one power-of-two fp32 scale per 128 x 128 block                   (128 x 128)
// The scales must be powers of two (every quantiser of this library produces such scales): a producer
// warp turns them into UE8M0 bytes (the fp32 exponent) in the tensor core's scale layout in shared
// memory, four K blocks per 32-bit word; the MMA thread copies a group of them into TMEM (tcgen05.cp)
// and picks the byte of the current K block through the instruction descriptor.
// Tile 128 x 256 per CTA; the two CTAs of a pair (PAIR, tcgen05 cta_group::2) have neighbouring row tiles and share the weights' rows: each
// fetches half of them, the leader issues the MMAs for both, everything behind the accumulator is a CTA's own. Operands from THIS GPU's memory
// only, no multicast.
// Warps: 0 TMA, 1 MMA (+ TMEM allocation), 2 scale producer, 4..11 epilogue (two per TMEM lane quadrant).
// The epilogue warps first move their part of the accumulator into registers and hand TMEM back, so the
// next tile's MMAs overlap the epilogue arithmetic and stores.
// Epilogues:
//   EPI 0  plain            : bf16 rows (MODE 2: to the owner's landing zone)
//   EPI 1  gate/up + SwiGLU : B is tile-interleaved (128 gate rows, 128 up rows per 256); out[row, 128 cols] bf16
//   EPI 3  gate/up + SwiGLU + re-quantisation: the 128 outputs of a tile row are one 1 x 128 block of the next
//                             GEMM's fp8 input: amax, power-of-two scale, e4m3 bytes and the scale are written
//                             here, so the activation never exists in bf16 in memory
// Modes:
//   MODE 1  all-gather -> GEMM : warps 3..11 of every CTA quantise its rows of this rank's bf16 sequence shard to
//                                fp8 + 1 x 128 scales into the rank's own gather buffer (first, so the first
//                                tiles can start), then warp 3 copies those bytes into every peer's gather buffer,
//                                nearest consumer first; the TMA and scale warps wait for a shard's flag
//                                before they touch its rows. Operands are read from THIS GPU's buffer only.
//   MODE 2  GEMM -> reduce-scatter : the epilogue stores each partial tile (bf16) into the landing zone of the
//                                rank that owns the rows and counts it there; after its tiles a CTA adds up
//                                the landed partials of the tiles it owns.
#include <cuda_bf16.h>

#include "mf_fp8.cuh"
#include "mf_gemm.cuh"
#include "mf_launch.cuh"
#include "mf_team.cuh"

namespace mfk {

constexpr int XBN = 256;
constexpr int XSFBUFS = 4;
constexpr int kXThreads = 384;
constexpr int kXTmemCols = 512;
constexpr uint32_t kXSfaCol = 256;  // TMEM columns [256, 260): scales of A; [260, 268): scales of B
constexpr uint32_t kXSfbCol = 260;

template <bool PAIR> struct XSmem {
    static constexpr int XSTAGES = PAIR ? 6 : 4;
    static constexpr int kABytes = BM * 128;
    static constexpr int kBBytes = (PAIR ? XBN / 2 : XBN) * 128;  // a CTA of a pair fetches half of the weights' rows
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kSfOff = XSTAGES * kStageBytes;
    static constexpr int kSfBufBytes = 512 + 1024;  // A chunk, two B chunks
    static constexpr int kBarOff = kSfOff + XSFBUFS * kSfBufBytes;
    static constexpr int kAmaxOff = kBarOff + 512;
    static constexpr int kOutOff = kBarOff + 512 + 2048;
    static constexpr int kOutRowB = 80;
    static constexpr int kOutBytes = 8 * 32 * kOutRowB;
    static constexpr int kTotal = kOutOff + kOutBytes;
    static constexpr int kDynBytes = kTotal + 1024;
    uint8_t *base;
    __device__ explicit XSmem(uint8_t *raw) : base(reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023)) {}
    __device__ uint8_t *a(int s) const { return base + s * kStageBytes; }
    __device__ uint8_t *b(int s) const { return base + s * kStageBytes + kABytes; }
    __device__ uint8_t *sf(int i) const { return base + kSfOff + i * kSfBufBytes; }
    __device__ uint64_t *bar(int i) const { return reinterpret_cast<uint64_t *>(base + kBarOff) + i; }
    __device__ uint64_t *full(int s) const { return bar(s); }
    __device__ uint64_t *empty(int s) const { return bar(XSTAGES + s); }
    __device__ uint64_t *sf_full(int i) const { return bar(2 * XSTAGES + i); }
    __device__ uint64_t *sf_empty(int i) const { return bar(2 * XSTAGES + XSFBUFS + i); }
    __device__ uint64_t *tfull() const { return bar(2 * XSTAGES + 2 * XSFBUFS); }
    __device__ uint64_t *tempty() const { return bar(2 * XSTAGES + 2 * XSFBUFS + 1); }
    __device__ uint32_t *tmem_slot() const { return reinterpret_cast<uint32_t *>(base + kBarOff + 256); }
    __device__ volatile int *abort_flag() const { return reinterpret_cast<volatile int *>(base + kBarOff + 264); }
    __device__ uint32_t *stored(int parity) const { return reinterpret_cast<uint32_t *>(base + kBarOff + 272) + parity; }  // MODE 2: warps that have stored a tile
    __device__ float *amax(int parity) const { return reinterpret_cast<float *>(base + kAmaxOff) + parity * 256; }
    __device__ uint8_t *out_stage(int epi_warp) const { return base + kOutOff + epi_warp * 32 * kOutRowB; }
};
static_assert(XSmem<false>::kDynBytes <= 227 * 1024 && XSmem<true>::kDynBytes <= 227 * 1024, "shared memory of the block-scaled fp8 GEMM");

struct XArgs {
    TmaPair tm;            // A: [rows, K] fp8; B: [N, K] fp8
    const float *a_scale;  // [rows, K/128]
    const float *b_scale;  // [N/128, K/128]  (N in ORIGINAL row order: for EPI 1/3 gate rows then up rows)
    int N, K;
    int max_rows;
    void *out;             // EPI 0/1: bf16; EPI 3: e4m3 bytes
    int64_t ldo;           // elements per output row
    float *out_scale;      // EPI 3: [rows, N/256]
    int *status;
    Team team;
    uint32_t epoch;        // flag value of this call (grows by one per call)
    uint32_t seq;          // MODE 1: number of fused calls so far on these counters, including this one
    // MODE 1
    const __nv_bfloat16 *x_local;  // this rank's shard [shard_rows, K] bf16
    int64_t ldx;
    int shard_rows;
    uint64_t ag_buf_off;     // slot offset of the gather buffer [W * shard_rows, K] e4m3
    uint64_t ag_scale_off;   // slot offset of its scales [W * shard_rows, K / 128] fp32
    uint64_t ag_ready_off;   // slot offset of W ready flags (u32)
    uint32_t *push_count;    // local device counters [W], monotonic
    // MODE 2
    uint64_t rs_land_off;    // slot offset of the landing zone [W][rows_per_rank][N] bf16
    uint64_t rs_count_off;   // slot offset of per-owned-tile arrival counters (u32), monotonic
    uint32_t *tile_uses;     // local: calls that had each owned tile so far, written by this kernel
    int rows_per_rank;
    __nv_bfloat16 *y_out;    // [rows_per_rank, N]
    int64_t ldy;
    float scale;
};

__device__ __forceinline__ void named_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// All-gather side, first pass: this CTA's rows of the rank's bf16 shard -> e4m3 + one power-of-two scale per 128 elements,
// into the rank's OWN gather buffer. Nine warps share it (the epilogue warps have nothing else to do until the first tile is
// finished, and no tile can start before the shard is complete): a unit is 2048 elements of a row (lane = 16 elements, 8
// lanes = one 128-group, four steps of 512). The next unit's loads are on their way while a unit's four steps, side by side, are
// worked on: with nine warps nothing else hides the latencies of either. 4096 rows of 8192: one warp per SM held the first tile back by more
// than 100 us, nine warps with two units at a time, loads and arithmetic in turns, by 45, so by 35 (copying the rows alone takes 25: nine warps).
// One 16-byte load per lane and run of 256, whole lines but more shuffles: 38; a third unit on its way: no difference.
constexpr int kQuantUnit = 2048;
struct QuantUnit {
    uint4 raw[4][2];
    int row, col;  // first row of the shard and column; row < 0: nothing to do
};
__device__ __forceinline__ void quant_load(const XArgs &g, QuantUnit &u, int row, int col, int r1, int lane)
{
    u.row = row < r1 ? row : -1;
    u.col = col;
    if (row >= r1) return;  // uniform over the warp
    const __nv_bfloat16 *src = g.x_local + (int64_t)row * g.ldx;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int c = min(col + v * 512, g.K - 512) + lane * 16;  // K is a multiple of 512: a step is there or not, for the whole warp
        u.raw[v][0] = __ldcg(reinterpret_cast<const uint4 *>(src + c));
        u.raw[v][1] = __ldcg(reinterpret_cast<const uint4 *>(src + c) + 1);
    }
}
__device__ __forceinline__ void quant_store(const QuantUnit &u, int K, uint8_t *own_q, float *own_s, int lane)
{
    if (u.row < 0) return;
    __nv_bfloat162 m[4];
    float scale[4];
#pragma unroll
    for (int v = 0; v < 4; v++) m[v] = __hmax2(amax_bf16(u.raw[v][0]), amax_bf16(u.raw[v][1]));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int v = 0; v < 4; v++) m[v] = __hmax2(m[v], shfl_xor_bf162(m[v], o));
#pragma unroll
    for (int v = 0; v < 4; v++) scale[v] = pow2_scale_e4m3(amax_of(m[v]));
    uint8_t *q = own_q + (int64_t)u.row * K + u.col + lane * 16;
    float *s = own_s + (int64_t)u.row * (K / 128) + u.col / 128 + lane / 8;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const __nv_bfloat162 mul = inverse_bf162(scale[v]);
        const uint2 lo = pack8_e4m3(u.raw[v][0], mul), hi = pack8_e4m3(u.raw[v][1], mul);
        if (u.col + v * 512 < K) {
            *reinterpret_cast<uint4 *>(q + v * 512) = make_uint4(lo.x, lo.y, hi.x, hi.y);
            if ((lane & 7) == 0) s[v * 4] = scale[v];
        }
    }
}
__device__ __noinline__ void ag_quant_rows(const XArgs &g, uint32_t me, int wq, int lane)
{
    constexpr int kWarps = 9;
    const int per = (g.shard_rows + (int)gridDim.x - 1) / (int)gridDim.x;
    const int r0 = min(g.shard_rows, (int)blockIdx.x * per), r1 = min(g.shard_rows, r0 + per);
    const int K = g.K, per_row = (K + kQuantUnit - 1) / kQuantUnit;
    uint8_t *own_q = peer_ptr(g.team, me, g.ag_buf_off) + (int64_t)me * g.shard_rows * K;
    float *own_s = reinterpret_cast<float *>(peer_ptr(g.team, me, g.ag_scale_off)) + (int64_t)me * g.shard_rows * (K / 128);
    const int rows_on = kWarps / per_row, parts_on = kWarps - rows_on * per_row;  // from a warp's unit to its next
    int row = r0 + wq / per_row, part = wq % per_row;
    auto next = [&](QuantUnit &u) {
        quant_load(g, u, row, part * kQuantUnit, r1, lane);
        row += rows_on;
        part += parts_on;
        if (part >= per_row) {
            part -= per_row;
            row++;
        }
    };
    QuantUnit a, b;
    next(a);
    while (a.row >= 0) {
        next(b);
        quant_store(a, K, own_q, own_s, lane);
        next(a);
        quant_store(b, K, own_q, own_s, lane);
    }
}

template <int MODE, int EPI, bool PAIR> __global__ void __launch_bounds__(kXThreads, 1) k_tp_fp8_mx(const __grid_constant__ XArgs g)
{
    using Smem = XSmem<PAIR>;
    constexpr int XSTAGES = Smem::XSTAGES;
    extern __shared__ uint8_t smem_raw[];
    Smem sm(smem_raw);
    const uint32_t crank = PAIR ? cluster_ctarank() : 0;
    const int walker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, walkers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    constexpr int kTileRows = PAIR ? 2 * BM : BM;  // of a pair or a single CTA
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int n_tiles = g.N / XBN;
    const int k_blocks = g.K / 128;
    const int sf_groups = (k_blocks + 3) / 4;
    AbortCtl ac{sm.abort_flag(), g.status};

    if (threadIdx.x == 0) {
        *sm.abort_flag() = 0;
        *sm.stored(0) = *sm.stored(1) = 0;
        for (int s = 0; s < XSTAGES; s++) {
            mbar_init(sm.full(s), 1);
            mbar_init(sm.empty(s), 1);
        }
        for (int i = 0; i < XSFBUFS; i++) {
            mbar_init(sm.sf_full(i), PAIR ? 2 : 1);  // the scale producers (of a pair: counted in the leader)
            mbar_init(sm.sf_empty(i), 1);
        }
        mbar_init(sm.tfull(), 1);
        mbar_init(sm.tempty(), PAIR ? 16 : 8);  // the epilogue warps (of a pair: counted in the leader)
        mbar_fence_init();
        tma_prefetch_desc(&g.tm.a);
        tma_prefetch_desc(&g.tm.b);
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(sm.tmem_slot(), kXTmemCols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(sm.tmem_slot(), kXTmemCols);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // both CTAs' barriers are initialised and both halves of the tensor memory are allocated
    tc_fence_after();
    const uint32_t tmem_base = *sm.tmem_slot();
    const int total = (g.max_rows / kTileRows) * n_tiles;
    const uint32_t me = g.team.rank;
    // MODE 2 by one rank: there are no partials to wait for, so a tile's epilogue writes its rows of y itself, under the next tile's MMAs. Adding up behind the
    // last tile read 67 MB back and wrote as much with the tensor cores idle: 4096 x 8192 outputs, K 3584, 126 us, so (and without a second fence
    // for the system per tile) 101; 1024 rows 43.2 / 36.0, 128 rows 23.3 / 20.0. With more ranks the loads of the other partials would hold the epilogue up.
    // The tiles are stored in the landing zone and counted all the same, as by every number of ranks, though only y is read behind the call.
    const bool alone = g.team.world == 1;

    after_predecessor();  // one rank's launch may start under the kernel in front of it; else this returns at once
    if (alone) start_successor();

    // linear tile -> (first row, column tile): blocks of rows owned by one rank, visited starting with this rank (MODE 1: the order in
    // which the shards arrive) or with the next rank (MODE 2: remote owners first, own rows last); inside a block the row tile varies fastest
    auto locate = [&](int t, int &row0, int &nt) {
        const int rows = MODE == 1 ? g.shard_rows : g.rows_per_rank;
        const int mt_per = rows / kTileRows;
        const int per_block = mt_per * n_tiles;
        const int i = t / per_block;
        const int owner = (int)((me + (MODE == 2 ? 1 : 0) + i) % g.team.world);
        const int r = t - i * per_block;
        nt = r / mt_per;
        row0 = (owner * mt_per + r % mt_per) * kTileRows + (int)crank * BM;  // of this CTA
    };

    if (MODE == 1 && warp >= 3) {
        ag_quant_rows(g, me, warp - 3, lane);
        named_bar_sync(10, 9 * 32);  // the CTA's rows are in this rank's gather buffer; warp 3 publishes them
    }

    if (warp == 0) {
        if (elect_one()) {
            PipeState ps;
            bool fine = true;
            auto load_b = [&](int stage, int kb, int nt) {
                if (PAIR) tma_load_2d_pair(sm.b(stage), &g.tm.b, kb * 128, nt * XBN + (int)crank * (XBN / 2), mapa_u32(smem_u32(sm.full(stage)), 0));
                else tma_load_2d(sm.b(stage), &g.tm.b, kb * 128, nt * XBN, sm.full(stage));
            };
            auto expect = [&](int stage) {  // of a pair both CTAs' bytes are counted on the leader's barrier
                if (!PAIR) mbar_expect_tx(sm.full(stage), Smem::kStageBytes);
                else if (crank == 0) mbar_expect_tx(sm.full(stage), 2 * Smem::kStageBytes);
            };
            // the weights of the first stages do not wait for any shard
            const int ahead = MODE == 1 && walker < total ? min(XSTAGES, k_blocks) : 0;
            for (int kb = 0; kb < ahead; kb++) {
                int row0, nt;
                locate(walker, row0, nt);
                expect(kb);
                load_b(kb, kb, nt);
            }
            for (int t = walker; t < total && fine; t += walkers) {
                int row0, nt;
                locate(t, row0, nt);
                if (MODE == 1) {
                    // the shard holding this tile's rows must have landed in this GPU's gather buffer
                    const uint32_t *ready = reinterpret_cast<const uint32_t *>(peer_ptr(g.team, me, g.ag_ready_off)) + row0 / g.shard_rows;
                    if (!wait_flag(ready, g.epoch, g.team.spin_limit)) {
                        *ac.abort_smem = 1;
                        atomicCAS(g.status, 0, 0x601);
                        break;
                    }
                    asm volatile("fence.proxy.async.global;" ::: "memory");  // peers' generic-proxy stores before our TMA reads
                }
                for (int kb = 0; kb < k_blocks; kb++) {
                    if (t != walker || kb >= ahead) {
                        fine = mbar_wait(sm.empty(ps.stage), ps.phase ^ 1, ac, 0x602);
                        if (!fine) break;
                        expect(ps.stage);
                        load_b(ps.stage, kb, nt);
                    }
                    if (PAIR) tma_load_2d_pair(sm.a(ps.stage), &g.tm.a, kb * 128, row0, mapa_u32(smem_u32(sm.full(ps.stage)), 0));
                    else tma_load_2d(sm.a(ps.stage), &g.tm.a, kb * 128, row0, sm.full(ps.stage));
                    ps.advance<XSTAGES>();
                }
            }
        }
    } else if (warp == 1) {
        if (crank == 0 && elect_one()) {
            // of a pair the leader issues for both: a commit that the other CTA waits for as well goes to both CTAs' barriers
            auto commit = [&](uint64_t *bar) {
                if (PAIR) {
                    umma_commit_pair(smem_u32(bar));
                    umma_commit_pair(mapa_u32(smem_u32(bar), 1));
                } else {
                    umma_commit(bar);
                }
            };
            PipeState ps, sf;
            uint32_t tphase = 0;
            bool fine = true;
            const uint32_t sfa = tmem_base + kXSfaCol, sfb = tmem_base + kXSfbCol;
            for (int t = walker; t < total && fine; t += walkers) {
                fine = mbar_wait<PAIR>(sm.tempty(), tphase ^ 1, ac, 0x603);  // the epilogue has taken the previous tile out of TMEM
                if (!fine) break;
                tc_fence_after();
                tphase ^= 1;
                for (int kb = 0; kb < k_blocks; kb++) {
                    if ((kb & 3) == 0) {
                        fine = mbar_wait<PAIR>(sm.sf_full(sf.stage), sf.phase, ac, 0x606);
                        if (!fine) break;
                        tc_fence_after();
                        const uint8_t *chunk = sm.sf(sf.stage);
                        if (PAIR) {
                            tmem_cp_sf_pair(sfa, umma_desc_sf(chunk));
                            tmem_cp_sf_pair(sfb, umma_desc_sf(chunk + 512));
                            tmem_cp_sf_pair(sfb + 4, umma_desc_sf(chunk + 1024));
                        } else {
                            tmem_cp_sf(sfa, umma_desc_sf(chunk));
                            tmem_cp_sf(sfb, umma_desc_sf(chunk + 512));
                            tmem_cp_sf(sfb + 4, umma_desc_sf(chunk + 1024));
                        }
                    }
                    fine = mbar_wait(sm.full(ps.stage), ps.phase, ac, 0x604);
                    if (!fine) break;
                    tc_fence_after();
                    const uint64_t da = umma_desc_sw128(sm.a(ps.stage));
                    const uint64_t db = umma_desc_sw128(sm.b(ps.stage));
                    const uint32_t idesc = umma_idesc_bs(kTileRows, XBN, (uint32_t)(kb & 3), (uint32_t)(kb & 3));
#pragma unroll
                    for (int k = 0; k < 4; k++) {  // 32 bytes = 32 fp8 = one UMMA K step
                        if (PAIR) umma_fp8_bs_pair(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb | k) != 0, sfa, sfb);
                        else umma_fp8_bs(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb | k) != 0, sfa, sfb);
                    }
                    commit(sm.empty(ps.stage));
                    ps.advance<XSTAGES>();
                    if ((kb & 3) == 3 || kb == k_blocks - 1) {
                        commit(sm.sf_empty(sf.stage));  // the scale chunk has been copied and its MMAs are done
                        sf.advance<XSFBUFS>();
                    }
                }
                if (fine) commit(sm.tfull());
            }
        }
    } else if (warp == 2) {
        // scale producer: lane l writes the 16 bytes of rows l, l + 32, l + 64, l + 96 (one 32-bit word of four
        // K-block scale bytes per row) and its share of the two B chunks
        PipeState sf;
        const int nblocks = g.N / 128;
        bool fine = true;
        for (int t = walker; t < total && fine; t += walkers) {
            int row0, nt;
            locate(t, row0, nt);
            int nb0, nb1;
            if (EPI == 1 || EPI == 3) {
                nb0 = nt;                  // gate rows nt * 128 .. + 128
                nb1 = nblocks / 2 + nt;    // up rows N/2 + nt * 128 .. + 128
            } else {
                nb0 = 2 * nt;
                nb1 = 2 * nt + 1;
            }
            const float *bs0 = g.b_scale + (int64_t)nb0 * k_blocks;
            const float *bs1 = g.b_scale + (int64_t)nb1 * k_blocks;
            if (MODE == 1) {
                // the scales of a shard arrive with its rows
                int ok = 1;
                if (lane == 0) {
                    const uint32_t *ready = reinterpret_cast<const uint32_t *>(peer_ptr(g.team, me, g.ag_ready_off)) + row0 / g.shard_rows;
                    ok = wait_flag(ready, g.epoch, g.team.spin_limit) ? 1 : 0;
                    if (!ok) {
                        *ac.abort_smem = 1;
                        atomicCAS(g.status, 0, 0x608);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    fine = false;
                    break;
                }
            }
            for (int gq = 0; gq < sf_groups; gq++) {
                int ok = 1;
                if (lane == 0) ok = mbar_wait(sm.sf_empty(sf.stage), sf.phase ^ 1, ac, 0x607) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    fine = false;
                    break;
                }
                uint32_t wa[4], wb0 = 0, wb1 = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int kb = gq * 4 + j;
                    const bool on = kb < k_blocks;
                    wb0 |= (on ? ue8m0_byte(bs0[kb]) : 127u) << (8 * j);
                    wb1 |= (on ? ue8m0_byte(bs1[kb]) : 127u) << (8 * j);
                }
#pragma unroll
                for (int r1 = 0; r1 < 4; r1++) {
                    const int row = min(row0 + r1 * 32 + lane, g.max_rows - 1);
                    const float *as = g.a_scale + (int64_t)row * k_blocks;
                    uint32_t w = 0;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int kb = gq * 4 + j;
                        // MODE 1: written by peers during this kernel, so past L1
                        w |= (kb < k_blocks ? ue8m0_byte(MODE == 1 ? __ldcg(as + kb) : as[kb]) : 127u) << (8 * j);
                    }
                    wa[r1] = w;
                }
                uint8_t *chunk = sm.sf(sf.stage);
                *reinterpret_cast<uint4 *>(chunk + lane * 16) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
                *reinterpret_cast<uint4 *>(chunk + 512 + lane * 16) = make_uint4(wb0, wb0, wb0, wb0);
                *reinterpret_cast<uint4 *>(chunk + 1024 + lane * 16) = make_uint4(wb1, wb1, wb1, wb1);
                fence_proxy_async_smem();  // the tensor core's copy unit reads these bytes through the async proxy
                __syncwarp();
                if (lane == 0) {
                    // each CTA's tensor core copies its own chunks, but the leader has both do it: the other CTA's bytes are released to the cluster
                    if (crank == 0) mbar_arrive(sm.sf_full(sf.stage));
                    else mbar_arrive_cluster_smem(mapa_u32(smem_u32(sm.sf_full(sf.stage)), 0));
                }
                sf.advance<XSFBUFS>();
            }
        }
    } else if (warp >= 4) {
        // eight epilogue warps: warp w reads TMEM lane quadrant w % 4 (the hardware's rule); the two warps of a
        // quadrant split the tile's 256 columns
        const int quad = warp & 3;
        const int half = (warp - 4) >> 2;
        uint32_t tphase = 0;
        uint8_t *stg = sm.out_stage(warp - 4);
        constexpr int kRowB = Smem::kOutRowB;
        for (int t = walker; t < total; t += walkers) {
            int row0, nt;
            locate(t, row0, nt);
            const int row = row0 + quad * 32 + lane;
            const bool row_ok = row < g.max_rows;
            if (!__all_sync(0xffffffffu, mbar_wait(sm.tfull(), tphase, ac, 0x605))) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
            uint32_t v[4][32];
            if (EPI == 1 || EPI == 3) {
                // a gate column and its up column in the same thread: half h owns gate [64h, 64h + 64), up [128 + 64h, ...)
                tmem_ld32(taddr + (uint32_t)(64 * half), v[0]);
                tmem_ld32(taddr + (uint32_t)(64 * half + 32), v[1]);
                tmem_ld32(taddr + (uint32_t)(128 + 64 * half), v[2]);
                tmem_ld32(taddr + (uint32_t)(128 + 64 * half + 32), v[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) tmem_ld32(taddr + (uint32_t)(128 * half + 32 * c), v[c]);
            }
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {  // the accumulator is in registers: the next tile may start
                if (crank == 0) mbar_arrive(sm.tempty());
                else mbar_arrive_cluster_smem(mapa_u32(smem_u32(sm.tempty()), 0));
            }
            if (EPI == 1 || EPI == 3) {
                float o[64];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const float gt = __uint_as_float(v[c][j]), up = __uint_as_float(v[2 + c][j]);
                        o[c * 32 + j] = gt / (1.f + __expf(-gt)) * up;
                    }
                if (EPI == 1) {
                    if (row_ok) {
                        __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(g.out) + (int64_t)row * g.ldo + nt * 128 + half * 64;
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            uint4 pk;
                            __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                            for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(o[q * 8 + 2 * e], o[q * 8 + 2 * e + 1]);
                            *reinterpret_cast<uint4 *>(dst + q * 8) = pk;
                        }
                    }
                } else {
                    // the activation is rounded to bf16 first (the precision it would have had in memory), then
                    // quantised: the two warps of a quadrant exchange their maxima through shared memory
                    float amax = 0.f;
#pragma unroll
                    for (int j = 0; j < 64; j++) {
                        o[j] = __bfloat162float(__float2bfloat16_rn(o[j]));
                        amax = fmaxf(amax, fabsf(o[j]));
                    }
                    float *ex = sm.amax((int)tphase);
                    ex[(quad * 2 + half) * 32 + lane] = amax;
                    named_bar_sync(1 + quad, 64);
                    amax = fmaxf(amax, ex[(quad * 2 + (half ^ 1)) * 32 + lane]);
                    const float scale = pow2_scale_e4m3(amax);
                    const float mul = 1.f / scale;  // exact: a power of two
                    if (row_ok) {
                        uint8_t *dst = static_cast<uint8_t *>(g.out) + (int64_t)row * g.ldo + nt * 128 + half * 64;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            uint4 pk;
                            pk.x = pack4_e4m3(o[q * 16 + 0], o[q * 16 + 1], o[q * 16 + 2], o[q * 16 + 3], mul);
                            pk.y = pack4_e4m3(o[q * 16 + 4], o[q * 16 + 5], o[q * 16 + 6], o[q * 16 + 7], mul);
                            pk.z = pack4_e4m3(o[q * 16 + 8], o[q * 16 + 9], o[q * 16 + 10], o[q * 16 + 11], mul);
                            pk.w = pack4_e4m3(o[q * 16 + 12], o[q * 16 + 13], o[q * 16 + 14], o[q * 16 + 15], mul);
                            *reinterpret_cast<uint4 *>(dst + q * 16) = pk;
                        }
                        if (half == 0) g.out_scale[(int64_t)row * (g.N / XBN) + nt] = scale;
                    }
                }
            } else {
                // rows leave through shared memory: lane = row on the way in, 16 lanes x 16 bytes per row on the way out
                unsigned long long dst = 0;
                if (row_ok) {
                    if (MODE == 2) {
                        // the partial tile goes to the landing zone of the rank that owns these rows
                        const int owner = row0 / g.rows_per_rank;
                        dst = reinterpret_cast<unsigned long long>(reinterpret_cast<__nv_bfloat16 *>(peer_ptr(g.team, (uint32_t)owner, g.rs_land_off)) +
                                                                   ((int64_t)me * g.rows_per_rank + (row - owner * g.rows_per_rank)) * g.N + nt * XBN + half * 128);
                    } else {
                        dst = reinterpret_cast<unsigned long long>(static_cast<__nv_bfloat16 *>(g.out) + (int64_t)row * g.ldo + nt * XBN + half * 128);
                    }
                }
                // Eight rows at a time: the lanes that own them write their whole 256-byte row segments (this warp's 128
                // columns) into the staging buffer, then the warp stores them 2 rows x 256 contiguous bytes per instruction
                // (16 lanes x 16 bytes per row). Over NVLink a write carries up to 256 bytes of payload: 64-byte pieces spent
                // almost half of the link on packet overhead.
                constexpr int kWideRowB = 272;  // 256 + 16: both the row writes and the 16-lanes-per-row reads stay conflict-free
                static_assert(8 * kWideRowB <= 32 * kRowB, "staging buffer of an epilogue warp");
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    if ((lane >> 3) == p) {
                        uint8_t *mine = stg + (lane & 7) * kWideRowB;
#pragma unroll
                        for (int c = 0; c < 4; c++) {
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                uint4 pk;
                                __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                    h[e] = __floats2bfloat162_rn(__uint_as_float(v[c][q * 8 + 2 * e]), __uint_as_float(v[c][q * 8 + 2 * e + 1]));
                                *reinterpret_cast<uint4 *>(mine + c * 64 + q * 16) = pk;
                            }
                        }
                    }
                    __syncwarp();
#pragma unroll
                    for (int it = 0; it < 4; it++) {
                        const int r = it * 2 + (lane >> 4);
                        const unsigned long long d = __shfl_sync(0xffffffffu, dst, p * 8 + r);
                        const uint4 val = *reinterpret_cast<const uint4 *>(stg + r * kWideRowB + (lane & 15) * 16);
                        if (d != 0) *reinterpret_cast<uint4 *>(d + (unsigned long long)((lane & 15) * 16)) = val;
                        if (MODE == 2 && alone) {
                            // the only partial there is, rounded as it would be read back
                            uint4 pk;
                            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&val);
                            __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const float2 f = __bfloat1622float2(h[e]);
                                o[e] = __floats2bfloat162_rn(f.x * g.scale, f.y * g.scale);
                            }
                            *reinterpret_cast<uint4 *>(g.y_out + (int64_t)(row0 + quad * 32 + p * 8 + r) * g.ldy + nt * XBN + half * 128 + (lane & 15) * 8) = pk;
                        }
                    }
                    __syncwarp();
                }
                if (MODE == 2) {
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(sm.stored((int)tphase))) : "memory");
                }
            }
            tphase ^= 1;
        }
    } else if (MODE == 2 && warp == 3) {
        // Counts every tile at its owner once all eight epilogue warps have stored their part. The release waits until a tile's stores have been
        // performed at the owner (4 to 5 us after the burst of a round's tiles): in the epilogue it held the next tile up, and K = 3584 was
        // bound by it (10.4 us a tile for 8.7 of MMAs; 4096 x 8192 outputs 89.5 us, so 78). One counter per parity: no warp is two tiles ahead of another, because a tile's MMAs start
        // when all of them have taken the previous accumulator out.
        if (lane == 0) {
            int it = 0;
            for (int t = walker; t < total; t += walkers, it++) {
                int row0, nt;
                locate(t, row0, nt);
                const uint32_t want = 8u * (uint32_t)(it / 2 + 1), at = smem_u32(sm.stored(it & 1));
                uint32_t have = 0;
                for (uint32_t i = 0; i < kMbarSpinLimit && !*ac.abort_smem; i++) {
                    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(have) : "r"(at) : "memory");
                    if (have >= want) break;
                    __nanosleep(64);
                }
                if (have < want) break;
                const int owner = row0 / g.rows_per_rank;
                const int ltile = ((row0 - owner * g.rows_per_rank) / BM) * n_tiles + nt;
                uint32_t *cnt = reinterpret_cast<uint32_t *>(peer_ptr(g.team, (uint32_t)owner, g.rs_count_off)) + ltile;
                if (alone) {
                    g.tile_uses[ltile]++;
                    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");  // nobody waits for it
                } else {
                    asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
                }
            }
        }
    } else if (MODE == 1 && warp == 3) {
        // all-gather side, after every warp's part of the quantisation: this CTA's rows and scales to every peer, nearest
        // consumer first.
        const int K = g.K, kg = K / 128;
        const int64_t shard_q = (int64_t)me * g.shard_rows * K, shard_s = (int64_t)me * g.shard_rows * kg;
        uint8_t *own_q = peer_ptr(g.team, me, g.ag_buf_off) + shard_q;
        float *own_s = reinterpret_cast<float *>(peer_ptr(g.team, me, g.ag_scale_off)) + shard_s;
        const int per = (g.shard_rows + (int)gridDim.x - 1) / (int)gridDim.x;
        const int r0 = min(g.shard_rows, (int)blockIdx.x * per), r1 = min(g.shard_rows, r0 + per);
        auto raise = [&](uint32_t p) {
            // The CTA that completes this rank's shard in the buffer of rank p raises the flag there: every CTA's fence and count hand its stores to that one,
            // whose fence for the system covers all of them. A fence for the system takes about 3 us, and three of them in a row stood in front of the first
            // tile of a call (N 7168, K 8192, SwiGLU, us, before / so: 128 rows 44.2 / 40.7, 1024 85.1 / 81.6, 4096 236 / 230).
            __syncwarp();
            if (lane == 0) {
                __threadfence();  // covers the stores ordered before it by the barriers of the warp and of the quantising warps
                const uint32_t done = atomicAdd(g.push_count + p, 1u) + 1;
                if (done == gridDim.x * g.seq) {
                    if (p == me) __threadfence();  // read by this GPU only
                    else fence_sys();
                    asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(reinterpret_cast<uint32_t *>(peer_ptr(g.team, p, g.ag_ready_off)) + me), "r"(g.epoch)
                                 : "memory");
                }
            }
            __syncwarp();
        };
        raise(me);
        const int64_t nq = (int64_t)(r1 - r0) * K / 16, ns = (int64_t)(r1 - r0) * kg;
        const uint4 *from_q = reinterpret_cast<const uint4 *>(own_q + (int64_t)r0 * K);
        const float *from_s = own_s + (int64_t)r0 * kg;
        for (uint32_t i = 1; i < g.team.world; i++) {
            const uint32_t p = (me + g.team.world - i) % g.team.world;
            uint4 *to_q = reinterpret_cast<uint4 *>(peer_ptr(g.team, p, g.ag_buf_off) + shard_q + (int64_t)r0 * K);
            float *to_s = reinterpret_cast<float *>(peer_ptr(g.team, p, g.ag_scale_off)) + shard_s + (int64_t)r0 * kg;
            int64_t v = lane;
            for (; v + 7 * 32 < nq; v += 8 * 32) {  // eight independent 16-byte loads in flight per lane, then eight peer stores
                uint4 val[8];
#pragma unroll
                for (int u = 0; u < 8; u++) val[u] = __ldcg(from_q + v + u * 32);
#pragma unroll
                for (int u = 0; u < 8; u++) to_q[v + u * 32] = val[u];
            }
            for (; v < nq; v += 32) to_q[v] = __ldcg(from_q + v);
            for (int64_t e = lane; e < ns; e += 32) to_s[e] = __ldcg(from_s + e);
            raise(p);
        }
    }
    // MODE 2, thread 0: calls that had this CTA's first owned tile so far. Every tile counts its own: smaller calls leave some out.
    uint32_t uses = 0;
    if (MODE == 2 && !alone && threadIdx.x == 0 && (int)blockIdx.x < (g.rows_per_rank / BM) * n_tiles) uses = g.tile_uses[blockIdx.x];
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // nobody signals a barrier of a CTA that has left, and both halves of the tensor memory are freed together
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, kXTmemCols);
        else tmem_dealloc(tmem_base, kXTmemCols);
    }
    if (MODE == 2 && !alone) {
        // add up the W partial tiles of every tile whose rows this rank owns
        __shared__ int ok_sh;
        const int own_tiles = (g.rows_per_rank / BM) * n_tiles;
        const uint32_t *cnt = reinterpret_cast<const uint32_t *>(peer_ptr(g.team, me, g.rs_count_off));
        const __nv_bfloat16 *land = reinterpret_cast<const __nv_bfloat16 *>(peer_ptr(g.team, me, g.rs_land_off));
        bool in_time = true;
        for (int t = blockIdx.x; t < own_tiles; t += gridDim.x) {
            if (threadIdx.x == 0) {
                g.tile_uses[t] = ++uses;
                in_time = in_time && !*ac.abort_smem && wait_flag(cnt + t, g.team.world * uses, g.team.spin_limit);
                if (!in_time) atomicCAS(g.status, 0, 0x609);
                ok_sh = in_time ? 1 : 0;
                if (t + (int)gridDim.x < own_tiles) uses = g.tile_uses[t + gridDim.x];  // arrives while this tile is added up
            }
            __syncthreads();
            if (ok_sh) {
                const int ml = t / n_tiles, nt = t % n_tiles;
                const int64_t at = (int64_t)ml * BM * g.N + nt * XBN;
                add_partials(land + at, (int64_t)g.rows_per_rank * g.N, g.N, XBN / 8, (int)g.team.world, g.scale,
                             g.y_out + (int64_t)ml * BM * g.ldy + nt * XBN, g.ldy);
            }
            __syncthreads();
        }
    }
}

}  // namespace mfk

using namespace mfk;

namespace {
template <int MODE, int EPI, bool PAIR> int launch_mx_as(const XArgs &g, int grid, cudaStream_t s)
{
    auto kern = k_tp_fp8_mx<MODE, EPI, PAIR>;
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, XSmem<PAIR>::kDynBytes) != cudaSuccess) {
            (void)cudaGetLastError();
            return -2;
        }
        attr_set = true;
    }
    // a grid whose CTAs wait for the peers' starts when the kernel in front of it has left the SMs; one rank waits for nobody (4 us of every call)
    if (g.team.world == 1) {
        const cudaError_t e = launch_overlapped(kern, dim3((unsigned)grid), dim3(kXThreads), XSmem<PAIR>::kDynBytes, s, PAIR ? 2 : 1, g);
        return e == cudaSuccess ? 0 : (int)e;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kXThreads);
    cfg.dynamicSmemBytes = XSmem<PAIR>::kDynBytes;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = PAIR ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, g);
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

// `rows`: of a rank's block. Whole 256-row tiles go to CTA pairs: a CTA fetches 32 KiB per 128 of K for what takes 48 KiB alone, which an SM's path from the
// L2 does not deliver under the MMAs (512 clocks). One rank, N 7168 / K 8192 (SwiGLU, fp8 out) and N 8192 / K 3584, us, single CTAs / pairs: 256 rows 46 / 40
// and 25 / 20, 512 50 / 46 and 26 / 21, 1024 81.6 / 76 and 36 / 33.5, 2048 138 / 137 and 62 / 55, 4096 230 / 229 and 101 / 89.5.
template <int MODE, int EPI> int launch_mx(XArgs &g, const void *b, int rows, int sms, cudaStream_t s)
{
    const bool pair = rows % (2 * BM) == 0 && (sms & 1) == 0 && sms >= 2;  // the same grid either way: the flags' counters count its CTAs
    const int rc = make_tmap_2d(&g.tm.b, b, 1, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.K, pair ? XBN / 2 : XBN, true);
    if (rc != 0) return rc;
    return pair ? launch_mx_as<MODE, EPI, true>(g, sms, s) : launch_mx_as<MODE, EPI, false>(g, sms, s);
}
}  // namespace

extern "C" {

int mf_grouped_gemm_fp8_mx_supported(int G, int N, int K, int epi);  // mf_gemm_fp8_pair.cu

// All-gather -> GEMM in fp8. x_local [shard_rows, K] bf16 is this rank's sequence shard; it is quantised (e4m3, one
// power-of-two scale per 128 elements) on its way into the gather buffers ([world * shard_rows, K] bytes at ag_buf_off,
// scales [world * shard_rows, K / 128] fp32 at ag_scale_off of every slot). B [N, K] e4m3 with b_scale [N/128, K/128].
// epi 0: out bf16 [world * shard_rows, N]; 1: SwiGLU, out bf16 [.., N/2] (B interleaved per 128 rows); 3: SwiGLU +
// re-quantisation, out e4m3 [.., N/2] with out_scale [.., N/256].
int mf_ag_gemm_fp8(const Team *team, const void *x_local, int64_t ldx, int shard_rows, const void *B, const float *b_scale, void *out, int64_t ldo,
                   float *out_scale, int N, int K, uint64_t ag_buf_off, uint64_t ag_scale_off, uint64_t ag_ready_off, uint32_t *push_count,
                   uint32_t epoch, uint32_t seq, int *status, int sms, int epi, void *stream)
{
    if (team == nullptr || team->emu || shard_rows <= 0 || (shard_rows % BM) != 0 || (K % 512) != 0 || (ldx & 7) != 0 ||
        !mf_grouped_gemm_fp8_mx_supported(1, N, K, epi) || epi == 2)
        return -1;
    if (epi == 3 && (out_scale == nullptr || (ldo & 15) != 0)) return -1;
    XArgs g{};
    const int M = shard_rows * (int)team->world;
    const uint64_t slot = team->heap_base + (uint64_t)team->rank * team->stride;
    int rc = make_tmap_2d(&g.tm.a, reinterpret_cast<const void *>(slot + ag_buf_off), 1, (uint64_t)M, (uint64_t)K, (uint64_t)K, BM, true);
    if (rc != 0) return rc;
    g.a_scale = reinterpret_cast<const float *>(slot + ag_scale_off);
    g.b_scale = b_scale;
    g.N = N;
    g.K = K;
    g.max_rows = M;
    g.out = out;
    g.ldo = ldo;
    g.out_scale = out_scale;
    g.status = status;
    g.team = *team;
    g.epoch = epoch;
    g.seq = seq;
    g.x_local = static_cast<const __nv_bfloat16 *>(x_local);
    g.ldx = ldx;
    g.shard_rows = shard_rows;
    g.ag_buf_off = ag_buf_off;
    g.ag_scale_off = ag_scale_off;
    g.ag_ready_off = ag_ready_off;
    g.push_count = push_count;
    cudaStream_t s = (cudaStream_t)stream;
    // every CTA carries a copy warp whose work peers wait for: the grid must be fully resident (one CTA per SM)
    switch (epi) {
        case 0: return launch_mx<1, 0>(g, B, shard_rows, sms, s);
        case 1: return launch_mx<1, 1>(g, B, shard_rows, sms, s);
        case 3: return launch_mx<1, 3>(g, B, shard_rows, sms, s);
        default: return -1;
    }
}

// GEMM -> reduce-scatter in fp8. A [M, K] e4m3 (M = world * rows_per_rank) with a_scale [M, K/128], B [N, K] e4m3 with
// b_scale [N/128, K/128]; y_out [rows_per_rank, N] bf16 = scale * sum over ranks of A . B^T.
int mf_gemm_rs_fp8(const Team *team, const void *A, const float *a_scale, const void *B, const float *b_scale, void *y_out, int64_t ldy,
                   int rows_per_rank, int N, int K, uint64_t rs_land_off, uint64_t rs_count_off, uint32_t *tile_uses, uint32_t epoch,
                   float scale, int *status, int sms, void *stream)
{
    if (team == nullptr || team->emu || rows_per_rank <= 0 || (rows_per_rank % BM) != 0 || (ldy & 7) != 0 || tile_uses == nullptr ||
        !mf_grouped_gemm_fp8_mx_supported(1, N, K, 0))
        return -1;
    XArgs g{};
    const int M = rows_per_rank * (int)team->world;
    int rc = make_tmap_2d(&g.tm.a, A, 1, (uint64_t)M, (uint64_t)K, (uint64_t)K, BM, true);
    if (rc != 0) return rc;
    g.a_scale = a_scale;
    g.b_scale = b_scale;
    g.N = N;
    g.K = K;
    g.max_rows = M;
    g.status = status;
    g.team = *team;
    g.epoch = epoch;
    g.tile_uses = tile_uses;
    g.rs_land_off = rs_land_off;
    g.rs_count_off = rs_count_off;
    g.rows_per_rank = rows_per_rank;
    g.y_out = static_cast<__nv_bfloat16 *>(y_out);
    g.ldy = ldy;
    g.scale = scale;
    return launch_mx<2, 0>(g, B, rows_per_rank, sms, (cudaStream_t)stream);
}

}  // extern "C"
