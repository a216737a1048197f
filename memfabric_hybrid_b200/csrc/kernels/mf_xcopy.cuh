// sm_100a copy kernels of the data-operation layer ("xcopy"): every byte that moves between two
// device-visible addresses (local HBM, a peer's HBM mapped over NVLink, pinned pooled DRAM) goes
// through these, issued from inside the kernel as 16-byte vector loads and stores.
//   mf_xcopy_batch_kernel : list of (src, dst, len) work chunks in a pinned, device-visible ring
//   mf_xcopy_bulk_kernel  : the same list where every address is a multiple of 16, through the copy unit
//   mf_xcopy_span_kernel  : pieces at any alignment, a share of equal weight per CTA
//   mf_xcopy_quant_kernel : bf16/fp16 -> int8 (per-unit scale) or fp8 e4m3 (1x128 scale) while pushing
// Parity of role: src/hybm/csrc/copy_extend/hybm_copy_kernel.cpp:53-90 (contiguous), :114-136 (batch),
// :163-235 (quantising batch).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "mf_shift.cuh"

namespace mfk {

struct CopyItem {
    uint64_t src;
    uint64_t dst;
    uint64_t len;
};

struct QuantItem {
    uint64_t src;
    uint64_t dst;
    uint64_t scale;
    uint64_t elems;
};

// Debug aid (MF_XCOPY_DEBUG=1): the pool's address window as the copy kernels check it. An address inside the window must
// lie, with its whole length, in the part of a rank's slot that is mapped here; addresses outside the window are the
// caller's own buffers and are taken as given. A descriptor that fails is skipped (nothing is read or written) and
// reported through the status word. The host validates every item before it builds descriptors; this second check
// sits in front of the first access of the kernel itself, where a sanitizer would otherwise be the only witness.
struct CopyWindow {
    uint64_t base;        // 0: no window, nothing is checked
    uint64_t slot;        // bytes between consecutive ranks' slots
    uint32_t ranks;
    uint32_t pad;
    uint64_t mapped[64];  // bytes mapped of every rank's slot
};
constexpr uint32_t kCopyBadDescriptor = 0x7D1u;

__device__ __forceinline__ bool xc_in_window(const CopyWindow *w, uint64_t a, uint64_t len)
{
    if (w == nullptr || w->base == 0 || a < w->base || a >= w->base + w->slot * w->ranks) return true;
    const uint64_t rel = a - w->base;
    const uint32_t r = (uint32_t)(rel / w->slot);
    const uint64_t off = rel - (uint64_t)r * w->slot;
    const uint64_t m = r < 64 ? w->mapped[r] : 0;
    return len <= m && off <= m - len;
}
__device__ __forceinline__ bool xc_check(const CopyWindow *w, const uint64_t src, const uint64_t dst, const uint64_t len, uint32_t *status)
{
    if (xc_in_window(w, src, len) && xc_in_window(w, dst, len)) return true;
    *reinterpret_cast<volatile uint32_t *>(status) = kCopyBadDescriptor;
    __threadfence_system();
    return false;
}

constexpr int kCopyThreads = 512;
constexpr int kCopyUnroll = 4;
constexpr uint32_t kCopyList = 32;  // descriptors that a CTA fetches at once

// Copies `len` bytes with all threads of the CTA. Fast path: both ends 16-byte aligned relative to
// each other; the unaligned head and tail go byte-wise.
__device__ __forceinline__ void cta_copy(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, uint64_t len)
{
    const int tid = threadIdx.x;
    const int nt = blockDim.x;
    if (((reinterpret_cast<uint64_t>(src) ^ reinterpret_cast<uint64_t>(dst)) & 15) != 0) {
        cta_copy_shifted<true>(src, dst, len);
        return;
    }
    uint64_t head = (16 - (reinterpret_cast<uint64_t>(src) & 15)) & 15;
    if (head > len) head = len;
    if (tid < head) dst[tid] = src[tid];
    const uint64_t body = (len - head) & ~15ULL;
    const uint4 *s = reinterpret_cast<const uint4 *>(src + head);
    uint4 *d = reinterpret_cast<uint4 *>(dst + head);
    const uint64_t n16 = body >> 4;
    uint64_t i = tid;
    // main loop: kCopyUnroll independent 16-byte loads in flight per thread before the first store
    for (; i + (uint64_t)(kCopyUnroll - 1) * nt < n16; i += (uint64_t)kCopyUnroll * nt) {
        uint4 v[kCopyUnroll];
#pragma unroll
        for (int u = 0; u < kCopyUnroll; u++) v[u] = __ldcs(s + i + (uint64_t)u * nt);
#pragma unroll
        for (int u = 0; u < kCopyUnroll; u++) __stcs(d + i + (uint64_t)u * nt, v[u]);
    }
    for (; i < n16; i += nt) __stcs(d + i, __ldcs(s + i));
    const uint64_t tail = len - head - body;
    if (tid < tail) dst[head + body + tid] = src[head + body + tid];
}

// A CTA fetches the descriptors of its next 32 chunks together (they lie in pinned host memory: a PCIe read of more than a microsecond),
// and nothing but the list's end holds its warps back: a warp that has no vectors left in one chunk is already in the next. With a
// descriptor and a barrier per chunk (one descriptor ahead), us before / now: 700 pieces of 256 B - 512 KiB at 2-byte offsets 26.2 / 24.5,
// 1500 of up to 16 KiB at any offset 15.0 / 12.2. (Large batches between device addresses go to mf_xcopy_span_kernel; batches with a leg in pinned host
// memory, and all of them where the copy unit is switched off, come here.) Where no CTA has more than one chunk a list
// and its barriers are in the way: replayed from a graph, one piece of up to 1 KiB takes 2.4 us with the single descriptor, 2.7 to 2.9 with a
// list; 20 pieces of up to 16 KiB 3.8 and 4.2, 100 of them 4.1 and 4.4.
__global__ void __launch_bounds__(kCopyThreads) mf_xcopy_batch_kernel(const CopyItem *__restrict__ items, uint32_t count,
                                                                      const CopyWindow *__restrict__ window, uint32_t *status)
{
    __shared__ uint64_t list[kCopyList * 3];
    static_assert(sizeof(CopyItem) == 3 * sizeof(uint64_t) && kCopyList * 3 <= kCopyThreads, "a thread per word of the list");
    const uint32_t slot = threadIdx.x / 3, word = threadIdx.x % 3;
    const uint64_t round = (uint64_t)gridDim.x * kCopyList;
    auto fetch = [&](uint64_t first) -> uint64_t {
        const uint64_t i = first + (uint64_t)slot * gridDim.x;
        return slot < kCopyList && i < count ? reinterpret_cast<const uint64_t *>(items + i)[word] : 0;
    };
    if (blockIdx.x >= count) return;
    if (count <= gridDim.x) {
        const CopyItem it = items[blockIdx.x];
        if (window == nullptr || xc_check(window, it.src, it.dst, it.len, status))
            cta_copy(reinterpret_cast<const uint8_t *>(it.src), reinterpret_cast<uint8_t *>(it.dst), it.len);
        return;
    }
    uint64_t next = fetch(blockIdx.x);
    for (uint64_t first = blockIdx.x; first < count; first += round) {
        if (first != blockIdx.x) __syncthreads();  // the previous list is no longer read
        if (slot < kCopyList) list[threadIdx.x] = next;
        __syncthreads();
        next = fetch(first + round);  // arrives while this list's chunks are copied
        for (uint32_t l = 0; l < kCopyList && first + (uint64_t)l * gridDim.x < count; l++) {
            const uint64_t src = list[3 * l], dst = list[3 * l + 1], len = list[3 * l + 2];
            if (window == nullptr || xc_check(window, src, dst, len, status))
                cta_copy(reinterpret_cast<const uint8_t *>(src), reinterpret_cast<uint8_t *>(dst), len);
        }
    }
}

// ---- bulk-copy engine variant ---------------------------------------------------------------------
// The same descriptor list, moved by the TMA unit instead of by registers: one lane per pipeline issues
// `cp.async.bulk` loads of `piece` bytes from the source into a ring of shared-memory stages and, as each
// lands (mbarrier), a `cp.async.bulk` store from that stage to the destination. No multicast; source and
// destination may be local HBM or a peer's mapped HBM. A pipeline keeps (stages - 2) loads and up to two
// stores in flight and runs on across chunk boundaries, so neither a CTA barrier nor a drain separates
// two items. Needs every chunk's source, destination and length to be multiples of 16 bytes (the host
// checks that and otherwise launches mf_xcopy_batch_kernel).
// A wait that runs out stores its code into *status (pinned host memory) and the pipeline stops after
// the copies it has in flight.
constexpr uint64_t kBulkWaitNs = 2000000000ull;  // a load that has not landed after 2 s is given up
constexpr int kBulkMaxStages = 8;

__device__ __forceinline__ uint32_t xc_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__global__ void __launch_bounds__(128) mf_xcopy_bulk_kernel(const CopyItem *__restrict__ items, uint32_t count, uint32_t stages,
                                                            uint32_t piece, uint32_t *status, const CopyWindow *__restrict__ window)
{
    extern __shared__ __align__(128) uint8_t xc_smem[];
    __shared__ __align__(8) uint64_t full[4][kBulkMaxStages];
    __shared__ uint64_t st_dst[4][kBulkMaxStages];
    __shared__ uint32_t st_len[4][kBulkMaxStages];
    if ((threadIdx.x & 31) != 0) return;
    const uint32_t w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const uint32_t pipe = blockIdx.x * W + w, pipes = gridDim.x * W;
    if (pipe >= count) return;
    uint8_t *ring = xc_smem + (size_t)w * stages * piece;
    for (uint32_t s = 0; s < stages; s++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(xc_smem_u32(&full[w][s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the initialised barriers as the copy unit sees them

    const uint32_t look = stages - 2;  // loads issued ahead of the store front
    uint32_t ci = pipe;                // chunk whose pieces are being loaded
    CopyItem cur = items[ci];
    CopyItem nxt = ci + pipes < count ? items[ci + pipes] : CopyItem{0, 0, 0};
    uint64_t off = 0;
    bool more = true, fine = true;
    // debug window: a chunk that fails the check is emptied (its pieces are never issued)
    if (window != nullptr && !xc_check(window, cur.src, cur.dst, cur.len, status)) off = cur.len;
    if (off >= cur.len) {
        // walk on to the first chunk of this pipeline that has bytes to move
        while (more && off >= cur.len) {
            ci += pipes;
            if (ci < count) {
                cur = nxt;
                off = (window != nullptr && !xc_check(window, cur.src, cur.dst, cur.len, status)) ? cur.len : 0;
                if (ci + pipes < count) nxt = items[ci + pipes];
            } else {
                more = false;
            }
        }
    }
    uint32_t loaded = 0, stored = 0;
    while (fine && (more || stored < loaded)) {
        if (more) {
            const uint32_t s = loaded % stages;
            // the store that last read this stage is at least two store groups back
            asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            const uint64_t left = cur.len - off;
            const uint32_t n = left < piece ? (uint32_t)left : piece;
            const uint32_t bar = xc_smem_u32(&full[w][s]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             xc_smem_u32(ring + (size_t)s * piece)),
                         "l"(cur.src + off), "r"(n), "r"(bar)
                         : "memory");
            st_dst[w][s] = cur.dst + off;
            st_len[w][s] = n;
            loaded++;
            off += n;
            while (more && off >= cur.len) {
                ci += pipes;
                if (ci < count) {
                    cur = nxt;
                    off = (window != nullptr && !xc_check(window, cur.src, cur.dst, cur.len, status)) ? cur.len : 0;
                    if (ci + pipes < count) nxt = items[ci + pipes];
                } else {
                    more = false;
                }
            }
        }
        if (loaded >= stored + look + 1 || (!more && stored < loaded)) {
            const uint32_t s = stored % stages, parity = (stored / stages) & 1;
            const uint32_t bar = xc_smem_u32(&full[w][s]);
            uint32_t ok = 0;
            uint64_t t0 = 0;
            for (uint32_t spin = 0; !ok; spin++) {
                asm volatile(
                    "{\n\t.reg .pred P;\n\t"
                    "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
                    "selp.b32 %0, 1, 0, P;\n\t}"
                    : "=r"(ok)
                    : "r"(bar), "r"(parity)
                    : "memory");
                if (!ok && (spin & 255u) == 255u) {  // time limit, not an iteration count: a try_wait may suspend for a while
                    uint64_t now;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > kBulkWaitNs) break;
                }
            }
            if (!ok) {
                *reinterpret_cast<volatile uint32_t *>(status) = 0x701u;
                __threadfence_system();
                fine = false;
                break;
            }
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(st_dst[w][s]),
                         "r"(xc_smem_u32(ring + (size_t)s * piece)), "r"(st_len[w][s])
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            stored++;
        }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- pieces at any alignment, cut into a share per CTA ---------------------------------------------
// A large batch whose addresses are not all multiples of 16: the host has cut it into shares of equal weight (see SpanCutter), and CTA i copies
// descriptors start[i] .. start[i + 1] - 1, which lie together in host memory; the shares travel with the launch. One thread walks the pieces and
// has the copy unit load their whole granules into a ring of shared-memory stages, eight warps cut the destination's vectors out of
// neighbouring granules and store them, one warp copies the few bytes in front of the first vector and behind the last. The loads of the next
// pieces are on their way whatever the warps wait for, so that short pieces and the ends of long ones cost no latency of their own.
// What bounds it: memory in large batches, latencies and the list's way from host memory in small ones. 700 pieces of 256 B - 512 KiB at 2-byte offsets (53
// MB) took 28.9 us with register copies of chunks dealt out one by one, 28.2 with equal shares alone, 21.7 so (4.9 TB/s); 1500 of up to 512 KiB at 4-byte
// offsets 51 / 41 (5.2 TB/s); 200 at 8-byte offsets 11.8 / 7.8; 1500 of up to 16 KiB at any offset 12.4 / 10.9 with half as many shares, 9.3 with all: a
// share costs the host 5 ns, and such a batch waits for the host.
struct SpanStarts {
    uint32_t start[601];
};
constexpr int kSpanConsumers = 8, kSpanThreads = (kSpanConsumers + 2) * 32, kSpanStages = 6;
constexpr uint32_t kSpanVecs = 1024, kSpanStageBytes = (kSpanVecs + 1) * 16, kSpanSmem = kSpanStages * kSpanStageBytes;

// `head` bytes one by one, `vecs` destination vectors, the rest one by one; granules are loaded from src + head - shift on.
__device__ __forceinline__ ShiftPlan span_plan(uint64_t src, uint64_t dst, uint64_t len)
{
    if (((src ^ dst) & 15) != 0) return shift_plan(src, dst, len);
    ShiftPlan p;
    p.head = (16 - (dst & 15)) & 15;
    if (p.head > len) p.head = len;
    p.vecs = (len - p.head) >> 4;
    p.shift = 0;
    return p;
}

enum XcWait : int { kXcArrived, kXcToldToQuit, kXcRanOut };
__device__ __forceinline__ XcWait xc_wait(uint64_t *bar, uint32_t parity, volatile int *quit, uint64_t limit_ns)
{
    uint64_t t0 = 0;
    for (uint32_t spin = 0;; spin++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred P;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P;\n\t}"
            : "=r"(ok)
            : "r"(xc_smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return kXcArrived;
        if ((spin & 255u) == 255u) {  // time limit, not an iteration count: a try_wait may suspend for a while
            if (quit != nullptr && *quit) return kXcToldToQuit;
            uint64_t now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) return kXcRanOut;
        }
    }
}
// The wait of a role whose CTA goes as soon as one of its waits runs out. Loader and storers wait for the same stage with the same limit, so either may be
// the first: whoever runs out reports it, before the others learn of it.
constexpr uint32_t kSpanLoadMissing = 0x702, kSpanStageMissing = 0x703;
__device__ __forceinline__ bool span_wait(uint64_t *bar, uint32_t parity, volatile int *quit, uint32_t *status, uint32_t code, uint64_t limit_ns = kBulkWaitNs)
{
    const XcWait w = xc_wait(bar, parity, quit, limit_ns);
    if (w == kXcRanOut) {
        *reinterpret_cast<volatile uint32_t *>(status) = code;
        *quit = 1;
    }
    return w == kXcArrived;
}

template <int Q> __device__ __forceinline__ void span_cut(const uint4 *g, uint4 *d, uint32_t vecs, uint32_t bits)
{
#pragma unroll
    for (uint32_t u = 0; u < kSpanVecs / (kSpanConsumers * 32); u++) {
        const uint32_t i = threadIdx.x + u * kSpanConsumers * 32;
        if (i < vecs) __stcs(d + i, cut16<Q>(g[i], g[i + 1], bits));
    }
}

__global__ void __launch_bounds__(kSpanThreads, 2) mf_xcopy_span_kernel(const CopyItem *__restrict__ items, const __grid_constant__ SpanStarts spans,
                                                                        const CopyWindow *__restrict__ window, uint32_t *status)
{
    extern __shared__ __align__(128) uint8_t xc_smem[];
    __shared__ __align__(8) uint64_t full[kSpanStages], empty[kSpanStages];
    __shared__ uint64_t list[kCopyList * 3];
    __shared__ int quit_sh;
    volatile int *quit = &quit_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t beg = spans.start[blockIdx.x], end = spans.start[blockIdx.x + 1];
    const uint64_t *words = reinterpret_cast<const uint64_t *>(items);
    auto fetch = [&](uint32_t first) -> uint64_t {
        return threadIdx.x < kCopyList * 3 && first + threadIdx.x / 3 < end ? words[(uint64_t)first * 3 + threadIdx.x] : 0;
    };
    uint64_t next = fetch(beg);
    if (threadIdx.x == 0) {
        quit_sh = 0;
        for (int s = 0; s < kSpanStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(xc_smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(xc_smem_u32(&empty[s])), "r"(kSpanConsumers));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the initialised barriers as the copy unit sees them
    }
    uint32_t slot = 0, phase = 0;  // of the role's next stage
    auto advance = [&]() {
        if (++slot == kSpanStages) {
            slot = 0;
            phase ^= 1;
        }
    };
    for (uint32_t first = beg; first < end; first += kCopyList) {
        __syncthreads();  // the barriers are initialised; the previous list is no longer read
        if (*quit) break;
        if (threadIdx.x < kCopyList * 3) list[threadIdx.x] = next;
        __syncthreads();
        next = fetch(first + kCopyList);  // arrives while this list's pieces are copied
        const uint32_t n = min(kCopyList, end - first);
        if (window != nullptr) {
            if (threadIdx.x < n && !xc_check(window, list[3 * threadIdx.x], list[3 * threadIdx.x + 1], list[3 * threadIdx.x + 2], status)) list[3 * threadIdx.x + 2] = 0;
            __syncthreads();
        }
        if (warp == kSpanConsumers) {
            if (lane != 0) continue;
            for (uint32_t l = 0; l < n && !*quit; l++) {
                const uint64_t src = list[3 * l];
                const ShiftPlan p = span_plan(src, list[3 * l + 1], list[3 * l + 2]);
                for (uint64_t v = 0; v < p.vecs; v += kSpanVecs) {
                    const uint32_t bytes = ((uint32_t)min((uint64_t)kSpanVecs, p.vecs - v) + (p.shift != 0 ? 1 : 0)) * 16;
                    if (!span_wait(&empty[slot], phase ^ 1, quit, status, kSpanStageMissing)) break;
                    const uint32_t bar = xc_smem_u32(&full[slot]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     xc_smem_u32(xc_smem + slot * kSpanStageBytes)),
                                 "l"(src + p.head - p.shift + v * 16), "r"(bytes), "r"(bar)
                                 : "memory");
                    advance();
                }
            }
        } else if (warp > kSpanConsumers) {
            constexpr uint32_t kAtOnce = 4;
            for (uint32_t l0 = 0; l0 < n; l0 += kAtOnce) {
                uint8_t b[kAtOnce][2];
                uint8_t *to[kAtOnce][2];
#pragma unroll
                for (uint32_t j = 0; j < kAtOnce; j++) {
                    const uint32_t l = min(l0 + j, n - 1);
                    const uint64_t src = list[3 * l], dst = list[3 * l + 1], len = list[3 * l + 2];
                    const ShiftPlan p = span_plan(src, dst, len);
                    const uint64_t edge = len - p.vecs * 16;  // at most 62: a head of up to 31 bytes and as many behind the vectors
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t e = lane + 32 * h;
                        const uint64_t at = e < p.head ? e : e + p.vecs * 16;
                        to[j][h] = nullptr;
                        if (e < edge && l0 + j < n) {
                            b[j][h] = *reinterpret_cast<const uint8_t *>(src + at);
                            to[j][h] = reinterpret_cast<uint8_t *>(dst + at);
                        }
                    }
                }
#pragma unroll
                for (uint32_t j = 0; j < kAtOnce; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (to[j][h] != nullptr) *to[j][h] = b[j][h];
            }
        } else {
            for (uint32_t l = 0; l < n && !*quit; l++) {
                const uint64_t dst = list[3 * l + 1];
                const ShiftPlan p = span_plan(list[3 * l], dst, list[3 * l + 2]);
                uint4 *d = reinterpret_cast<uint4 *>(dst + p.head);
                const uint32_t bits = (p.shift & 3) * 8;
                for (uint64_t v = 0; v < p.vecs; v += kSpanVecs) {
                    if (!span_wait(&full[slot], phase, quit, status, kSpanLoadMissing)) break;
                    const uint4 *g = reinterpret_cast<const uint4 *>(xc_smem + slot * kSpanStageBytes);
                    const uint32_t m = (uint32_t)min((uint64_t)kSpanVecs, p.vecs - v);
                    if (p.shift == 0) {
#pragma unroll
                        for (uint32_t u = 0; u < kSpanVecs / (kSpanConsumers * 32); u++) {
                            const uint32_t i = threadIdx.x + u * kSpanConsumers * 32;
                            if (i < m) __stcs(d + v + i, g[i]);
                        }
                    } else {
                        switch (p.shift >> 2) {  // uniform over the CTA
                            case 0: span_cut<0>(g, d + v, m, bits); break;
                            case 1: span_cut<1>(g, d + v, m, bits); break;
                            case 2: span_cut<2>(g, d + v, m, bits); break;
                            default: span_cut<3>(g, d + v, m, bits); break;
                        }
                    }
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(xc_smem_u32(&empty[slot])) : "memory");
                    advance();
                }
            }
        }
    }
    __syncthreads();
    // a load that did not land in time: once more as long for what the copy unit still has in flight, then the CTA goes
    if (*quit && warp == kSpanConsumers && lane == 0)
        for (int s = 0; s < kSpanStages; s++) {
            const uint32_t done = slot > (uint32_t)s ? phase : phase ^ 1;  // parity of the stage's last load
            xc_wait(&full[s], done, nullptr, kBulkWaitNs);
        }
}

// The two roles on stages of their own that nothing ever fills or frees, each with a limit of its own: word 0 of `status` is what is reported, word 1 counts
// the roles that have left.
__global__ void __launch_bounds__(64) mf_xcopy_wait_probe_kernel(uint32_t *status, uint64_t loader_ns, uint64_t storer_ns)
{
    __shared__ __align__(8) uint64_t full, empty;
    __shared__ int quit_sh;
    if (threadIdx.x == 0) {
        quit_sh = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(xc_smem_u32(&full)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(xc_smem_u32(&empty)));
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        const bool loader = threadIdx.x == 0;
        if (!span_wait(loader ? &empty : &full, 0, &quit_sh, status, loader ? kSpanStageMissing : kSpanLoadMissing, loader ? loader_ns : storer_ns))
            atomicAdd_system(status + 1, 1u);
    }
}

// One WARP per (item, unit); a CTA of 8 warps walks the units of its item. The unit is read once when it fits in
// the lanes' registers (unit <= 512 elements with 16-byte loads), else twice (the second pass hits L1 / L2):
// absolute maximum by warp shuffles, then scale + round + 8-byte stores to the (peer) destination.
// mode 0: int8, q = rint(x * 127 / amax), dequant factor amax / 127 written to scale[unitIndex]
// mode 1: fp8 e4m3 (satfinite), q = x * 448 / amax, dequant factor amax / 448
// Vector path: source 16-byte aligned, destination 8-byte aligned, unit a multiple of 8; anything else takes
// the element-wise path of the same warp layout.
template <typename In> __device__ __forceinline__ float to_f32(In v);
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename In> __device__ __forceinline__ void unpack8(const uint4 &raw, float *f)
{
    const In *h = reinterpret_cast<const In *>(&raw);
#pragma unroll
    for (int k = 0; k < 8; k++) f[k] = to_f32<In>(h[k]);
}

// int8: adding 1.5 * 2^23 rounds to an integer (to nearest, ties to even, as rintf) and leaves it in the low bits of the sum; the clamp, whose
// bounds are integers, comes first and takes a NaN to -127. Round and convert instructions run at a quarter of the rate: 512 items
// of 128 Ki fp16 elements, units of 128, took 54.2 us with them, 41.8 so.
__device__ __forceinline__ uint32_t round_int8(float x, float mul)
{
    return __float_as_uint(fminf(127.f, fmaxf(-127.f, x * mul)) + 12582912.f);  // the low byte
}

template <int MODE> __device__ __forceinline__ uint8_t quant1(float x, float mul)
{
    if (MODE == 0) return (uint8_t)round_int8(x, mul);
    return (uint8_t)__nv_cvt_float_to_fp8(x * mul, __NV_SATFINITE, __NV_E4M3);
}

template <int MODE> __device__ __forceinline__ uint2 quant8(const float *f, float mul)
{
    uint32_t lo = 0, hi = 0;
    if (MODE == 1) {
        // two values per conversion instruction (cvt.rn.satfinite.e4m3x2.f32)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            lo |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[2 * k] * mul, f[2 * k + 1] * mul), __NV_SATFINITE, __NV_E4M3) << (16 * k);
            hi |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[4 + 2 * k] * mul, f[5 + 2 * k] * mul), __NV_SATFINITE, __NV_E4M3) << (16 * k);
        }
        return make_uint2(lo, hi);
    }
    // the low bytes of four sums in three byte permutations
    auto four = [&](const float *g) {
        return __byte_perm(__byte_perm(round_int8(g[0], mul), round_int8(g[1], mul), 0x0040),
                           __byte_perm(round_int8(g[2], mul), round_int8(g[3], mul), 0x0040), 0x5410);
    };
    return make_uint2(four(f), four(f + 4));
}

template <typename In, int MODE>
__global__ void __launch_bounds__(256) mf_xcopy_quant_kernel(const QuantItem *__restrict__ items, uint32_t unit)
{
    __shared__ QuantItem it;
    if (threadIdx.x == 0) it = items[blockIdx.y];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t units = (it.elems + unit - 1) / unit;
    const In *src = reinterpret_cast<const In *>(it.src);
    uint8_t *dst = reinterpret_cast<uint8_t *>(it.dst);
    float *scales = reinterpret_cast<float *>(it.scale);
    const float qmax = MODE == 0 ? 127.f : 448.f;
    const bool vec = (unit % 8) == 0 && (it.src & 15) == 0 && (it.dst & 7) == 0;
    // Lanes per unit: a unit of up to 128 elements is 16 vectors, so two units share a warp. Each group of lanes
    // works on J units per step, all loads issued before the first reduction (latency hiding).
    const uint32_t W = (vec && unit <= 128) ? 16u : 32u;
    const uint32_t upw = 32u / W, sub = lane / W, sl = lane % W;
    constexpr int J = 2;
    const uint64_t per_cta = 8ull * upw * J;
    for (uint64_t base = (uint64_t)blockIdx.x * per_cta + (uint64_t)warp * upw * J; base < units; base += (uint64_t)gridDim.x * per_cta) {
        uint64_t ub[J], ue[J], nv[J];
        uint4 keep[J][2];
        float amax[J], f[8];
#pragma unroll
        for (int j = 0; j < J; j++) {
            const uint64_t u = base + (uint64_t)j * upw + sub;
            const bool on = u < units;
            ub[j] = on ? u * unit : 0;
            ue[j] = on ? min(it.elems, ub[j] + (uint64_t)unit) : 0;   // off: an empty range, the lanes only take part in the shuffles
            nv[j] = vec ? (ue[j] - ub[j]) / 8 : 0;                     // whole 8-element vectors of this unit
            const uint4 *src16 = reinterpret_cast<const uint4 *>(src + ub[j]);
            amax[j] = 0.f;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint64_t v = sl + (uint64_t)W * i;
                if (v < nv[j]) {
                    keep[j][i] = __ldg(src16 + v);
                    unpack8<In>(keep[j][i], f);
#pragma unroll
                    for (int k = 0; k < 8; k++) amax[j] = fmaxf(amax[j], fabsf(f[k]));
                }
            }
            for (uint64_t v = sl + 2ull * W; v < nv[j]; v += W) {
                unpack8<In>(__ldg(src16 + v), f);
#pragma unroll
                for (int k = 0; k < 8; k++) amax[j] = fmaxf(amax[j], fabsf(f[k]));
            }
            for (uint64_t k = ub[j] + nv[j] * 8 + sl; k < ue[j]; k += W) amax[j] = fmaxf(amax[j], fabsf(to_f32<In>(src[k])));
        }
#pragma unroll
        for (int j = 0; j < J; j++)
            for (uint32_t o = W / 2; o > 0; o >>= 1) amax[j] = fmaxf(amax[j], __shfl_xor_sync(0xffffffffu, amax[j], o));
#pragma unroll
        for (int j = 0; j < J; j++) {
            const float mul = amax[j] > 0.f ? qmax / amax[j] : 1.f;
            if (sl == 0 && ue[j] > ub[j]) scales[ub[j] / unit] = amax[j] > 0.f ? amax[j] / qmax : 1.f;
            const uint4 *src16 = reinterpret_cast<const uint4 *>(src + ub[j]);
            uint2 *dst8 = reinterpret_cast<uint2 *>(dst + ub[j]);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint64_t v = sl + (uint64_t)W * i;
                if (v < nv[j]) {
                    unpack8<In>(keep[j][i], f);
                    dst8[v] = quant8<MODE>(f, mul);
                }
            }
            for (uint64_t v = sl + 2ull * W; v < nv[j]; v += W) {
                unpack8<In>(__ldg(src16 + v), f);
                dst8[v] = quant8<MODE>(f, mul);
            }
            for (uint64_t k = ub[j] + nv[j] * 8 + sl; k < ue[j]; k += W) dst[k] = quant1<MODE>(to_f32<In>(src[k]), mul);
        }
    }
}

// Fast path of the quantising copy: units that are whole 16-byte vectors of the source, whole units per item; source 16-byte,
// destination 8-byte aligned. W lanes share a unit, R vectors each, and take J consecutive units per step: J x R (eight or nine)
// independent loads per lane are in flight before the first reduction, and a unit is read once. Few lanes per unit: what they hold
// is reduced without shuffles, and fewer lanes repeat a unit's divisions. The kernel above keeps two loads per lane in flight and is bound
// by the latency of each step, and reads a unit of more than 512 elements twice; here memory and the latencies of the arithmetic are about
// even. 512 items of 128 Ki 16-bit values (201 MB), us, before / now: units of 128 -> fp8 39.7 / 35.6 (5.6 TB/s; 16 lanes per unit that
// traded units while they reduced, 2 lanes: 47.9), -> int8 40.0 / 36.1; -> int8 by the kernel above / here: 64 198 / 40.5, 192 145 / 40.6,
// 256 112 / 36.8, 576 95 / 39.3, 1024 75 / 38.2, 2048 86 / 35.6. (Loads of the next steps by cp.async into shared memory, two CTAs
// per SM: 48.9 for 38.4; the warps that hide the arithmetic are worth more.)
//
// Blocks are dealt out over a grid that fits the GPU at once: block v takes steps v % parts, v % parts + parts, .. of item
// v / parts, a step being the units that a CTA converts at once. The descriptors sit in pinned host memory (a PCIe
// read of more than a microsecond), so a CTA fetches those of its next 32 blocks together and its warps then run through these
// blocks without another barrier.
template <typename In> struct PairOf;
template <> struct PairOf<__nv_bfloat16> { using type = __nv_bfloat162; };
template <> struct PairOf<__half> { using type = __half2; };
template <typename In> struct Pair16 {  // two 16-bit values in a register
    using type = typename PairOf<In>::type;
    __device__ static type of(uint32_t w) { return *reinterpret_cast<const type *>(&w); }
    __device__ static type max2(type a, type b) { return __hmax2(a, b); }
    __device__ static type absmax(const uint4 &v) { return max2(max2(__habs2(of(v.x)), __habs2(of(v.y))), max2(__habs2(of(v.z)), __habs2(of(v.w)))); }
    __device__ static type xchg(type a, int lane_mask) { return __shfl_xor_sync(0xffffffffu, a, lane_mask); }
    __device__ static float fold(type a) { return fmaxf(__low2float(a), __high2float(a)); }
};
constexpr uint32_t kQuantList = 32;
constexpr int kQuantCtasPerSm = 3;             // 80 registers a thread, 96 KB of loads in flight per SM
// Units that the 8 warps of a CTA take at once.
template <int W, int J> constexpr uint32_t quant_step() { return 8u * (32u / W) * J; }

// V: 16-byte vectors per unit, 0: unit_vecs of them, at most W * R
template <typename In, int MODE, int W, int R, int J, int V>
__global__ void __launch_bounds__(256, kQuantCtasPerSm) mf_xcopy_quant_units_kernel(const QuantItem *__restrict__ items, uint32_t count, uint32_t parts,
                                                                                    uint32_t unit_vecs)
{
    const uint32_t vecs = V > 0 ? (uint32_t)V : unit_vecs;
    __shared__ QuantItem list[kQuantList];
    constexpr uint32_t kStep = quant_step<W, J>();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sub = lane / W, sl = lane % W;
    const float qmax = MODE == 0 ? 127.f : 448.f;
    const uint32_t blocks = count * parts;  // the launch keeps this far below 2^32
    for (uint32_t v0 = blockIdx.x; v0 < blocks; v0 += gridDim.x * kQuantList) {
        __syncthreads();  // the previous list is no longer read
        if (threadIdx.x < kQuantList * 4) {
            const uint32_t v = v0 + (threadIdx.x >> 2) * gridDim.x;
            if (v < blocks)
                reinterpret_cast<uint64_t *>(list)[threadIdx.x] = reinterpret_cast<const uint64_t *>(items + v / parts)[threadIdx.x & 3];
        }
        __syncthreads();
        for (uint32_t l = 0; l < kQuantList; l++) {
            const uint32_t v = v0 + l * gridDim.x;
            if (v >= blocks) break;
            const QuantItem it = list[l];
            const uint64_t units = it.elems / 8 / vecs;
            const uint4 *src = reinterpret_cast<const uint4 *>(it.src);
            uint2 *dst = reinterpret_cast<uint2 *>(it.dst);
            float *scales = reinterpret_cast<float *>(it.scale);
            // the loop bounds are the same for the whole warp (the shuffles below), its last lanes may have fewer units left
            for (uint64_t step = (uint64_t)(v % parts) * kStep + warp * (32 / W) * J; step < units; step += (uint64_t)parts * kStep) {
                const uint64_t base = step + sub * J;
                uint4 raw[J][R];
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int r = 0; r < R; r++)
                        raw[j][r] = base + j < units && sl + r * W < vecs ? __ldcs(src + (base + j) * vecs + sl + r * W) : make_uint4(0, 0, 0, 0);
                // Largest magnitude of each unit, two 16-bit values per register (a maximum needs no rounding).
                typename Pair16<In>::type m[J];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    m[j] = Pair16<In>::absmax(raw[j][0]);
#pragma unroll
                    for (int r = 1; r < R; r++) m[j] = Pair16<In>::max2(m[j], Pair16<In>::absmax(raw[j][r]));
                }
                float mul[J];
#pragma unroll
                for (int j = 0; j < J; j++) {
#pragma unroll
                    for (int o = W / 2; o >= 1; o /= 2) m[j] = Pair16<In>::max2(m[j], Pair16<In>::xchg(m[j], o));
                    const float amax = Pair16<In>::fold(m[j]);
                    mul[j] = amax > 0.f ? qmax / amax : 1.f;
                    if (sl == 0 && base + j < units) scales[base + j] = amax > 0.f ? amax / qmax : 1.f;
                }
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int r = 0; r < R; r++)
                        if (base + j < units && sl + r * W < vecs) {
                            float f[8];
                            unpack8<In>(raw[j][r], f);
                            __stcs(dst + (base + j) * vecs + sl + r * W, quant8<MODE>(f, mul[j]));
                        }
            }
        }
    }
}

// Units of more vectors than a warp holds, up to 1024: the CTA shares a unit, four vectors per thread, and has the warps that takes
// (quant_wide_threads); the next unit's vectors are on their way while this one is reduced and stored.
// 512 items of 128 Ki bf16 values to int8, us, general kernel / 256 threads for every unit / so: 2056 100 / 126 / 62, 3072 101 / 105 / 50,
// 4096 97 / 88 / 46, 5120 115 / 72 / 50, 7168 131 / 53 / 48, 8192 142 / 49 / 46.
constexpr uint32_t kQuantWideVecs = 4;
inline uint32_t quant_wide_threads(uint32_t vecs) { return (vecs + 32 * kQuantWideVecs - 1) / (32 * kQuantWideVecs) * 32; }

template <typename In>
__global__ void __launch_bounds__(256, 4) mf_xcopy_quant_wide_kernel(const QuantItem *__restrict__ items, uint32_t count, uint32_t parts, uint32_t vecs)
{
    __shared__ QuantItem list[kQuantList];
    __shared__ float top[2][8];
    constexpr int R = kQuantWideVecs;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t blocks = count * parts;
    uint32_t parity = 0;
    for (uint32_t v0 = blockIdx.x; v0 < blocks; v0 += gridDim.x * kQuantList) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kQuantList * 4; i += blockDim.x) {
            const uint32_t v = v0 + (i >> 2) * gridDim.x;
            if (v < blocks) reinterpret_cast<uint64_t *>(list)[i] = reinterpret_cast<const uint64_t *>(items + v / parts)[i & 3];
        }
        __syncthreads();
        const uint32_t have = min(kQuantList, (blocks - v0 + gridDim.x - 1) / gridDim.x);
        // unit u of block l of the list; behind the last unit of a block comes the next block that has one
        uint32_t l = 0;
        uint64_t u = 0;
        auto settle = [&]() {
            for (; l < have; l++) {
                u = (v0 + l * gridDim.x) % parts;
                if (u < list[l].elems / 8 / vecs) return;
            }
        };
        auto load = [&](uint4 (&raw)[R]) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t at = threadIdx.x + r * blockDim.x;
                raw[r] = l < have && at < vecs ? __ldcs(reinterpret_cast<const uint4 *>(list[l].src) + u * vecs + at) : make_uint4(0, 0, 0, 0);
            }
        };
        settle();
        uint4 next[R];
        load(next);
        while (l < have) {
            uint4 raw[R];
#pragma unroll
            for (int r = 0; r < R; r++) raw[r] = next[r];
            uint2 *dst = reinterpret_cast<uint2 *>(list[l].dst) + u * vecs;
            float *scale = reinterpret_cast<float *>(list[l].scale) + u;
            u += parts;
            if (u >= list[l].elems / 8 / vecs) {
                l++;
                settle();
            }
            load(next);
            typename Pair16<In>::type m = Pair16<In>::absmax(raw[0]);
#pragma unroll
            for (int r = 1; r < R; r++) m = Pair16<In>::max2(m, Pair16<In>::absmax(raw[r]));
#pragma unroll
            for (int o = 16; o >= 1; o /= 2) m = Pair16<In>::max2(m, Pair16<In>::xchg(m, o));
            if (lane == 0) top[parity][warp] = fmaxf(Pair16<In>::fold(m), 0.f);
            __syncthreads();  // the other half of top is written by warps that have passed the next barrier
            float amax = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++)
                if (w < (int)(blockDim.x >> 5)) amax = fmaxf(amax, top[parity][w]);
            parity ^= 1;
            const float mul = amax > 0.f ? 127.f / amax : 1.f;
            if (threadIdx.x == 0) *scale = amax > 0.f ? amax / 127.f : 1.f;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t at = threadIdx.x + r * blockDim.x;
                if (at < vecs) {
                    float f[8];
                    unpack8<In>(raw[r], f);
                    __stcs(dst + at, quant8<0>(f, mul));
                }
            }
        }
    }
}

}  // namespace mfk
