"""GPU tests of the pooled-HBM copy paths (bit-exact against the source data).

Two processes on ONE device are a valid test of the inter-process mapping (VMM export over the fd
channel, peer mapping, batched kernel) because the copy kernels never wait on one another."""
import zlib

import numpy as np
import pytest

from conftest import free_port
from mp_util import run_ranks

pytestmark = pytest.mark.gpu
MiB = 1 << 20


def test_smoke_single_rank():
    from memfabric_hybrid_b200 import smoke
    smoke.run()


def _two_ranks(rank, world, url, sync):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    ndev = torch.cuda.device_count()
    dev_id = rank % ndev
    torch.cuda.set_device(dev_id)
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = rank
    cfg.start_store = rank == 0
    cfg.operation_timeout = 60
    assert bm.initialize(url, world, dev_id, cfg) == 0, mf.get_last_err_msg()
    h = bm.create2(id=1, local_dram_size=32 * MiB, max_dram_size=32 * MiB, local_hbm_size=128 * MiB, max_hbm_size=128 * MiB)
    assert h.join() == 0, mf.get_last_err_msg()
    sync.wait(120)
    peer = 1 - rank
    g = torch.Generator("cuda").manual_seed(100 + rank)
    x = torch.randint(0, 255, (64 * MiB,), dtype=torch.uint8, device="cuda", generator=g)
    pdev = h.peer_rank_ptr(peer, bm.BmMemType.DEVICE)
    mdev = h.peer_rank_ptr(rank, bm.BmMemType.DEVICE)
    # The pool's internal stream is not ordered with PyTorch's: tensors that a PyTorch kernel fills must be
    # complete before a copy that runs there reads or overwrites them.
    torch.cuda.synchronize()
    # D2RD: odd sizes and offsets on purpose (head/tail paths), plus big aligned segments
    segs = [(0, 1 * MiB), (1 * MiB + 3, 4097), (2 * MiB + 16, 16 * 1024), (3 * MiB, 8 * MiB), (12 * MiB + 1, 777), (16 * MiB, 32 * MiB)]
    srcs = [x.data_ptr() + o for o, _ in segs]
    dsts = [pdev + o for o, _ in segs]
    sizes = [s for _, s in segs]
    assert h.copy_data_batch(srcs, dsts, sizes, len(segs), bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
    sync.wait(120)
    # what the peer pushed into OUR slice
    gp = torch.Generator("cuda").manual_seed(100 + peer)
    want = torch.randint(0, 255, (64 * MiB,), dtype=torch.uint8, device="cuda", generator=gp)
    got = torch.zeros(64 * MiB, dtype=torch.uint8, device="cuda")
    pulled = torch.zeros(8 * MiB, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert h.copy_data_batch([mdev + o for o, _ in segs], [got.data_ptr() + o for o, _ in segs], sizes, len(segs),
                             bm.BmCopyType.G2L, 0) == 0, mf.get_last_err_msg()
    for o, s in segs:
        assert torch.equal(got[o:o + s], want[o:o + s]), f"segment at {o} (+{s}) differs"
    # RD2D pull from the peer's slice (it holds OUR data) and a D2H leg into the pooled DRAM, then GH2H
    assert h.copy_data(pdev + 3 * MiB, pulled.data_ptr(), 8 * MiB, bm.BmCopyType.G2L, 0) == 0, mf.get_last_err_msg()
    assert torch.equal(pulled, x[3 * MiB:11 * MiB])
    mhost = h.peer_rank_ptr(rank, bm.BmMemType.HOST)
    assert h.copy_data(x.data_ptr(), mhost, 8 * MiB, bm.BmCopyType.L2GH, 0) == 0, mf.get_last_err_msg()
    back = np.empty(8 * MiB, dtype=np.uint8)
    assert h.copy_data(mhost, back.ctypes.data, 8 * MiB, bm.BmCopyType.GH2H, 0) == 0
    assert zlib.crc32(back.tobytes()) == zlib.crc32(x[:8 * MiB].cpu().numpy().tobytes())
    # async + wait on the internal stream
    assert h.copy_data(x.data_ptr(), pdev + 48 * MiB, 16 * MiB, bm.BmCopyType.L2G, bm.ASYNC_COPY_FLAG) == 0
    assert h.wait() == 0
    # per-item results: one bad item out of three
    rc, res = h.copy_data_batch_partial_succeed([x.data_ptr(), x.data_ptr(), x.data_ptr()],
                                                [pdev, pdev + 1024 * MiB, pdev + MiB], [4096, 4096, 4096], 3, bm.BmCopyType.L2G, 0)
    assert rc == -2012 and res[0] == 0 and res[1] != 0 and res[2] == 0, (rc, res)
    mf.get_and_clear_last_err_msg()
    st = h.copy_stats()
    sync.wait(120)
    assert h.leave() == 0
    sync.wait(120)  # rank 0 hosts the config store: no teardown while the peer is still leaving
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return st["kernel_launches"]


def test_two_process_hbm_pool():
    url = f"tcp://127.0.0.1:{free_port()}"
    launches = run_ranks(_two_ranks, 2, (url,), timeout=300, with_barrier=True)
    assert all(l > 0 for l in launches), f"SM copy kernel did not run: {launches}"


@pytest.mark.parametrize("bulk", [0, 1])
def test_copy_kernels_refuse_descriptors_outside_the_mapped_window(bulk):
    """The debug window of the copy kernels (MF_XCOPY_DEBUG=1 publishes the pool's window; here it is handed in directly):
    a descriptor whose pooled side runs past the mapped part of a slot is skipped before its first access and reported;
    its neighbours are copied."""
    import ctypes as C
    import torch
    from memfabric_hybrid_b200 import _native as N
    cu = N.cuda()
    cu.mf_xcopy_debug_probe.restype = C.c_int
    cu.mf_xcopy_debug_probe.argtypes = [C.POINTER(C.c_uint64), C.c_uint32, C.c_uint64, C.c_uint64, C.c_uint32, C.POINTER(C.c_uint64), C.c_int]
    n = 64 << 10
    src = torch.arange(n, device="cuda", dtype=torch.int32)
    pool = torch.zeros(4 * n, device="cuda", dtype=torch.int32)       # stands for a window of 4 slots of n ints, 3/4 of each mapped
    other = torch.zeros(n, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    slot = n * 4
    base = pool.data_ptr()
    mapped = (C.c_uint64 * 4)(*[slot * 3 // 4] * 4)
    half = n * 2                                                      # bytes of half a slot
    trip = [src.data_ptr(), base, half,                               # into the mapped part of slot 0
            src.data_ptr(), base + slot + slot // 2, half,            # slot 1: starts inside, ends past the mapped 3/4: refused
            src.data_ptr(), other.data_ptr(), half,                   # neither side in the window: taken as given
            src.data_ptr(), base + 4 * slot - 4096, 4096 * 2]         # runs out of the window's last slot: refused
    arr = (C.c_uint64 * len(trip))(*trip)
    rc = cu.mf_xcopy_debug_probe(arr, len(trip) // 3, base, slot, 4, mapped, bulk)
    assert rc == 0x7D1, hex(rc & 0xFFFFFFFF)
    torch.cuda.synchronize()
    q = n // 2
    assert torch.equal(pool[:q], src[:q]) and torch.equal(other[:q], src[:q])
    assert int(pool[n + q:2 * n].abs().max()) == 0 and int(pool[4 * n - 1024:].abs().max()) == 0   # the refused ones wrote nothing
    # all descriptors fine: status 0
    ok = (C.c_uint64 * 3)(src.data_ptr(), base + 2 * slot, half)
    assert cu.mf_xcopy_debug_probe(ok, 1, base, slot, 4, mapped, bulk) == 0
    torch.cuda.synchronize()
    assert torch.equal(pool[2 * n:2 * n + q], src[:q])


def _prepared_rank(rank, world, url):
    import numpy as np
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    from memfabric_hybrid_b200.utils import benchutil as bu
    torch.cuda.set_device(0)
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.auto_ranking = False
    cfg.rank_id, cfg.start_store = 0, True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    blocks = 4
    nbytes = blocks * bu.KV_BLOCK_BYTES
    pool = (nbytes + (4 << 20)) // (2 << 20) * (2 << 20)
    h = bm.create2(id=0, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    src = torch.randint(0, 255, (nbytes,), dtype=torch.uint8, device="cuda")
    back = torch.zeros_like(src)
    segs = bu.kv_block_segments(blocks)
    offs = np.array([o for o, _ in segs], dtype=np.uint64)
    sizes = np.array([s for _, s in segs], dtype=np.uint64)
    put = h.create_batch(offs + np.uint64(src.data_ptr()), offs + np.uint64(base), sizes, bm.BmCopyType.L2G)
    get = h.create_batch(offs + np.uint64(base), offs + np.uint64(back.data_ptr()), sizes, bm.BmCopyType.G2L)
    assert put.nbytes == nbytes and get.nbytes == nbytes
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    # eager: two launches in stream order
    assert put.launch(s.cuda_stream) == 0 and get.launch(s.cuda_stream) == 0, mf.get_last_err_msg()
    s.synchronize()
    eager_ok = bool(torch.equal(back, src))
    # recorded into a CUDA graph and replayed on new data: submission writes nothing on the host
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        assert put.launch(torch.cuda.current_stream().cuda_stream) == 0
        assert get.launch(torch.cuda.current_stream().cuda_stream) == 0
    graph_ok = True
    for seed in (1, 2):
        src.copy_(torch.randint(0, 255, (nbytes,), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)))
        back.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        graph_ok = graph_ok and bool(torch.equal(back, src))
    del g
    # a triple outside the pool is refused when the batch is built, host-to-pool types are refused
    bad = None
    try:
        h.create_batch([src.data_ptr()], [base + pool + 4096], [4096], bm.BmCopyType.L2G)
    except RuntimeError as e:
        bad = str(e)
    host = np.zeros(4096, dtype=np.uint8)
    bad2 = None
    try:
        h.create_batch([host.ctypes.data], [base], [4096], bm.BmCopyType.H2G)
    except RuntimeError as e:
        bad2 = str(e)
    mf.get_and_clear_last_err_msg()
    put.destroy()
    get.destroy()
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return eager_ok, graph_ok, bad is not None, bad2 is not None


def test_prepared_batch_launches_and_replays_in_a_cuda_graph():
    """mf_bm_batch_create / _launch: validated once, one launch per submission, capturable."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_prepared_rank, 1, (url,), timeout=180) == [(True, True, True, True)]


def _shifted_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    torch.cuda.set_device(0)
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    pool = 64 * MiB
    h = bm.create2(id=4, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    # every pair of offsets inside a 16-byte granule; lengths around the granule, the warp's run (2 KiB), the CTA's step
    # (32 KiB) and the work chunk
    lens = [1, 15, 16, 17, 31, 32, 33, 47, 48, 63, 512, 2047, 2048, 2064, 2081, 4095, 32767, 32768 + 17, 70001]
    segs, so, do = [], 0, 0
    for s in range(16):
        for d in range(16):
            n = lens[(s * 16 + d) % len(lens)]
            for ln in (n, lens[(s + d) % len(lens)]):
                segs.append((so + s, do + d, ln))
                so += (s + ln + 63) // 16 * 16
                do += (d + ln + 63) // 16 * 16
    # short pieces go element by element: bytes up to 2 KiB, words at 4-byte offsets up to 8 KiB
    for s, d in ((0, 4), (4, 0), (8, 12), (12, 4), (2, 6), (3, 0)):
        for ln in (4, 2047, 2048, 2049, 2052, 4096, 8188, 8190, 8192, 8193, 8196):
            segs.append((so + s, do + d, ln))
            so += (s + ln + 63) // 16 * 16
            do += (d + ln + 63) // 16 * 16
    g = torch.Generator("cuda").manual_seed(5)
    src = torch.randint(0, 256, (so + 64,), dtype=torch.uint8, device="cuda", generator=g)
    fill = torch.randint(0, 256, (do + 64,), dtype=torch.uint8, device="cuda", generator=g)
    torch.cuda.synchronize()
    assert h.copy_data(fill.data_ptr(), base, fill.numel(), bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
    assert h.copy_data_batch([src.data_ptr() + s for s, _, _ in segs], [base + d for _, d, _ in segs], [n for _, _, n in segs], len(segs),
                             bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
    got = torch.empty_like(fill)
    assert h.copy_data(base, got.data_ptr(), got.numel(), bm.BmCopyType.G2L, 0) == 0, mf.get_last_err_msg()
    want = fill.clone()
    for s, d, n in segs:
        want[d:d + n] = src[s:s + n]
    torch.cuda.synchronize()
    ok = bool(torch.equal(got, want))   # the bytes between the pieces included
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return ok


def _share_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    torch.cuda.set_device(0)
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    pool = 256 * MiB
    h = bm.create2(id=5, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base, bad = h.peer_rank_ptr(0, bm.BmMemType.DEVICE), []
    stage = 16384   # bytes that a CTA moves at once
    ends = [stage * k + e for k in (1, 2, 7) for e in (-17, -16, -1, 0, 1, 15, 16, 31, 33)]
    # the ends of stages, at one offset and at two; more pieces than a CTA's list holds, of a few bytes and of a few vectors; one long piece cut into all shares
    for name, lens, offs in (("stages", ends * 12, (0, 1, 4, 15)), ("tiny", [1, 5, 16, 17, 62, 63, 64] * 3000, (0, 3)), ("short", [300, 700, 1030] * 8000, (0, 8, 11)),
                             ("long", [100_000_003], (5,)), ("same offset", [40_001] * 400, (7,))):
        segs, so, do = [], 0, 0
        for i, ln in enumerate(lens):
            s, d = offs[i % len(offs)], offs[i // len(offs) % len(offs)]
            segs.append((so + s, do + d, ln))
            so += (s + ln + 31) // 16 * 16
            do += (d + ln + 47) // 16 * 16
        src = torch.randint(0, 256, (so + 64,), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(len(lens)))
        fill = torch.full((do + 64,), 77, dtype=torch.uint8, device="cuda")
        want = fill.clone()
        for s, d, n in segs:
            want[d:d + n] = src[s:s + n]
        lists = [src.data_ptr() + s for s, _, _ in segs], [base + d for _, d, _ in segs], [n for _, _, n in segs]
        got = torch.empty_like(fill)
        for prepared in (False, True):
            torch.cuda.synchronize()
            assert h.copy_data(fill.data_ptr(), base, fill.numel(), bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
            if prepared:
                b = h.create_batch(*lists, bm.BmCopyType.L2G)
                b.launch(torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                b.destroy()
            else:
                assert h.copy_data_batch(*lists, len(segs), bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
            assert h.copy_data(base, got.data_ptr(), got.numel(), bm.BmCopyType.G2L, 0) == 0, mf.get_last_err_msg()
            torch.cuda.synchronize()
            if not torch.equal(got, want):   # the bytes between the pieces included
                bad.append((name, prepared))
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


@pytest.mark.parametrize("debug", ["0", "1"], ids=["plain", "descriptors_checked"])
def test_unaligned_batches_in_shares(debug):
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_share_rank, 1, (url,), timeout=240, env={"MF_XCOPY_DEBUG": debug}) == [[]]


def test_unaligned_batches_without_the_copy_unit():
    """MF_XCOPY_BULK=0: the same batches, direct and prepared, through the register copy kernel."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_share_rank, 1, (url,), timeout=240, env={"MF_XCOPY_BULK": "0"}) == [[]]


@pytest.mark.parametrize("loader_us,storer_us,code", [(500, 500_000, 0x703), (500_000, 500, 0x702)], ids=["loader_first", "storers_first"])
def test_a_wait_of_the_span_kernel_that_runs_out_is_reported(loader_us, storer_us, code):
    """Whichever role gives up first: the status is set before the other one, which then leaves without a word, is told."""
    import ctypes as C
    from memfabric_hybrid_b200 import _native as N
    cu = N.cuda()
    cu.mf_xcopy_wait_probe.restype = C.c_int
    cu.mf_xcopy_wait_probe.argtypes = [C.c_uint32, C.c_uint32]
    assert cu.mf_xcopy_wait_probe(loader_us, storer_us) == code


def test_pieces_at_every_pair_of_byte_offsets():
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_shifted_rank, 1, (url,), timeout=180) == [True]


def _quant_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    torch.cuda.set_device(0)
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    pool = 320 * MiB
    h = bm.create2(id=5, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    # units per item: around a half-warp's eight, a CTA's step of 128, two steps; then so many items that none is cut into parts and
    # one CTA walks the three steps of an item of 257 units; then one item fewer and one more than a resident grid (148 SMs x 3)
    # takes with a step each
    plans = [[1, 2, 8, 15, 16, 17, 127, 128, 129, 255, 256, 257, 600], [257] * 7200, [300] * 148, [300] * 149]
    bad = []
    for pi, units in enumerate(plans):
        for fp8, fp16 in ((True, False), (False, True)):
            n = sum(units) * 128
            g = torch.Generator("cuda").manual_seed(pi)
            x = torch.randn(n, device="cuda", generator=g).to(torch.float16 if fp16 else torch.bfloat16)
            x[:128] = 0    # a unit without a largest value
            torch.cuda.synchronize()
            first = np.concatenate(([0], np.cumsum(units)))[:-1]
            fac = base + (n + 255) // 256 * 256 + 4 * (pi == 0)   # factors that 16-byte stores do not reach in the first plan
            assert h.quant_copy_batch([x.data_ptr() + int(f) * 256 for f in first], [base + int(f) * 128 for f in first], [u * 256 for u in units],
                                      [fac + int(f) * 4 for f in first], 128, fp8=fp8, fp16_input=fp16) == 0, mf.get_last_err_msg()
            q = torch.empty(n, dtype=torch.uint8, device="cuda")
            f = torch.empty(n // 128, device="cuda")
            assert h.copy_data(base, q.data_ptr(), n, bm.BmCopyType.G2L, 0) == 0
            assert h.copy_data(fac, f.data_ptr(), n // 32, bm.BmCopyType.G2L, 0) == 0
            top = 448.0 if fp8 else 127.0
            v = x.float().view(-1, 128)
            amax = v.abs().amax(1, keepdim=True)
            one = torch.ones_like(amax)
            top = torch.full_like(amax, top)   # tensor by tensor: a division by a Python number is a product with its reciprocal
            y = v * torch.where(amax > 0, top / amax, one)
            want = y.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else y.round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
            if not (torch.equal(q.view(-1, 128), want) and torch.equal(f.view(-1, 1), torch.where(amax > 0, amax / top, one))):
                bad.append((pi, fp8))
            del x, q, v, y, want
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


def test_quantising_copy_of_items_around_its_block_sizes():
    """The same bytes and factors as the formula in fp32 (x * (top / amax), amax / top)."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_quant_rank, 1, (url,), timeout=300) == [[]]


def _int8_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    torch.cuda.set_device(0)
    torch.zeros(1, device="cuda")
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    h = bm.create2(id=12, local_dram_size=0, max_dram_size=0, local_hbm_size=64 << 20, max_hbm_size=64 << 20)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    from memfabric_hybrid_b200.ops.heap import tensor_at
    bad = []
    for dt in (torch.bfloat16, torch.float16):
        # every 16-bit pattern (NaN, infinities and subnormal values among them), shuffled so that units mix them, and the finite ones
        # in order, so that units hold one magnitude; then values half-way between two integers
        bits = torch.arange(65536, dtype=torch.int32).to(torch.int16)
        mixed = bits[torch.randperm(65536, generator=torch.Generator().manual_seed(1))]
        half = (torch.arange(65536) % 255 - 127.5).clamp(-127, 127).to(dt).view(torch.int16)
        for pi, pattern in enumerate((mixed, bits, half)):
            for unit, off in ((128, 0), (1024, 0), (64, 0), (128, 1)):
                n = 65536 - (unit if off else 0)
                x = pattern.cuda().view(dt)[off:off + n]
                q, f = tensor_at(base, (n,), torch.uint8), tensor_at(base + (1 << 20), (n // unit,), torch.float32)
                torch.cuda.synchronize()
                assert h.quant_copy_batch([x.data_ptr()], [base], [2 * n], [base + (1 << 20)], unit, fp16_input=dt == torch.float16) == 0
                v = x.float().view(-1, unit)
                amax = torch.where(torch.isnan(v), torch.zeros_like(v), v.abs()).amax(1, keepdim=True)   # a NaN counts as nothing
                one, top = torch.ones_like(amax), torch.full_like(amax, 127.0)
                y = v * torch.where(amax > 0, top / amax, one)
                want = torch.where(torch.isnan(y), torch.full_like(y, -127.0), y.round().clamp(-127, 127)).to(torch.int8).view(torch.uint8)
                if not torch.equal(q.view(-1, unit), want) or not torch.equal(f.view(-1, 1), torch.where(amax > 0, amax / top, one)):
                    bad.append((str(dt), pi, unit, off, int((q.view(-1, unit) != want).sum())))
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


def test_int8_rounding_of_every_16_bit_value():
    """Round to nearest even and the clamp, as the formula in fp32 gives them; a NaN becomes -127. Units of the fast path and of the general one,
    source addresses on and off 16 bytes."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_int8_rank, 1, (url,), timeout=300) == [[]]


def _units_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    from memfabric_hybrid_b200.ops.heap import tensor_at
    torch.cuda.set_device(0)
    torch.zeros(1, device="cuda")
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    pool = 256 * MiB
    h = bm.create2(id=13, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    bad = []
    # units on both sides of every line of the rule, the largest of each lane layout and sizes that leave places empty; 8200 and 100
    # (not whole vectors) are the general kernel's, and so is an item whose last unit is not full (tail)
    for unit in (8, 56, 64, 72, 128, 136, 192, 200, 256, 264, 576, 584, 1024, 1032, 2048, 2056, 7168, 8192, 8200, 100):
        for units, tail in (([1, 2, 3, 7, 8, 9, 31, 64, 65], 0), ([33] * 700 if unit <= 1024 else [5] * 700, 0), ([4, 9], unit // 2)):
            dt = torch.float16 if unit % 16 == 8 else torch.bfloat16
            sizes = [u * unit + tail for u in units]
            n, nf = sum(sizes), sum(-(-e // unit) for e in sizes)
            x = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(unit)).to(dt)
            x[:unit] = 0
            first = np.concatenate(([0], np.cumsum(sizes)))
            f0 = np.concatenate(([0], np.cumsum([-(-e // unit) for e in sizes])))
            fac = base + (n + 64 + 255) // 256 * 256
            q, f = tensor_at(base, (n + 64,), torch.uint8), tensor_at(fac, (nf + 1,), torch.float32)
            q.fill_(77)
            f.fill_(-5)
            torch.cuda.synchronize()
            assert h.quant_copy_batch([x.data_ptr() + int(a) * 2 for a in first[:-1]], [base + int(a) for a in first[:-1]], [e * 2 for e in sizes],
                                      [fac + int(a) * 4 for a in f0[:-1]], unit, fp16_input=dt == torch.float16) == 0, mf.get_last_err_msg()
            if len(units) > 100 and tail == 0:
                v = x.float().view(-1, unit)
                want_amax = v.abs().amax(1)
            else:
                v, want_amax = None, torch.cat([x[a + k:min(b, a + k + unit)].float().abs().amax().view(1) for a, b in zip(first[:-1], first[1:])
                                                for k in range(0, int(b - a), unit)])
            one, top = torch.ones_like(want_amax), torch.full_like(want_amax, 127.0)
            mul = torch.where(want_amax > 0, top / want_amax, one)
            lens = torch.tensor([min(int(b - a) - k, unit) for a, b in zip(first[:-1], first[1:]) for k in range(0, int(b - a), unit)], device="cuda")
            y = x.float() * torch.repeat_interleave(mul, lens)
            want = y.round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
            if not (torch.equal(q[:n], want) and torch.equal(f[:nf], torch.where(want_amax > 0, want_amax / top, one)) and bool((q[n:] == 77).all())
                    and float(f[nf]) == -5):
                bad.append((unit, units[:2], tail, int((q[:n] != want).sum())))
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


def test_quantising_copy_of_units_of_any_size():
    """int8 bytes and factors as the formula in fp32 gives them, nothing written behind them."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_units_rank, 1, (url,), timeout=300) == [[]]


def _wide_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    from memfabric_hybrid_b200.ops.heap import tensor_at
    torch.cuda.set_device(0)
    torch.zeros(1, device="cuda")
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    pool = 256 * MiB
    h = bm.create2(id=14, local_dram_size=0, max_dram_size=0, local_hbm_size=pool, max_hbm_size=pool)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    bad = []
    # units that a CTA shares, three warps to eight, both sides of each step, in items of one, two and many units; then more items than 32 for every
    # CTA of the grid, so that a CTA fetches a second list of descriptors: 444 CTAs, 1480 of three warps, 592 of eight
    cases = [(u, per, n) for u in (2056, 3072, 3080, 4096, 4104, 5128, 6152, 7176, 8192) for per, n in ((1, 5), (2, 700), (37, 3), (400, 2))]
    cases += [(64, 1, 15000), (2056, 1, 47500), (8192, 1, 19500)]
    for unit, per, n in cases:
        dt = torch.float16 if unit % 16 == 8 else torch.bfloat16
        each = unit * per
        x = torch.randn(n * per, unit, device="cuda", generator=torch.Generator("cuda").manual_seed(unit + n)).to(dt)
        x[n * per // 2] = 0
        fac = base + (n * each + 64 + 255) // 256 * 256
        q, f = tensor_at(base, (n * each + 64,), torch.uint8), tensor_at(fac, (n * per + 1,), torch.float32)
        q.fill_(77)
        f.fill_(-5)
        torch.cuda.synchronize()
        at = range(n)
        assert h.quant_copy_batch([x.data_ptr() + i * each * 2 for i in at], [base + i * each for i in at], [each * 2] * n, [fac + i * per * 4 for i in at], unit,
                                  fp16_input=dt == torch.float16) == 0, mf.get_last_err_msg()
        amax = x.abs().amax(1).float()
        one, top = torch.ones_like(amax), torch.full_like(amax, 127.0)
        mul = torch.where(amax > 0, top / amax, one)
        ok = torch.equal(f[:n * per], torch.where(amax > 0, amax / top, one)) and bool((q[n * each:] == 77).all()) and float(f[n * per]) == -5
        got = q[:n * each].view(n * per, unit)
        for lo in range(0, n * per, 4096):   # in bands: the fp32 values of all items would be 2.5 times the pool
            want = (x[lo:lo + 4096].float() * mul[lo:lo + 4096, None]).round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
            ok = ok and torch.equal(got[lo:lo + 4096], want)
        if not ok:
            bad.append((unit, per, n))
        del x
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


def test_quantising_copy_of_wide_units_and_of_more_items_than_a_list_holds():
    """int8 bytes and factors as the formula in fp32 gives them, nothing written behind them."""
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_wide_rank, 1, (url,), timeout=300) == [[]]


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 129, 1000])
def test_register_copy_takes_one_list_of_descriptors_after_another(n):
    """Two CTAs, 32 descriptors in a list: a CTA without any, one descriptor each, part of a list, a full one, several; pieces at odd offsets, nothing
    written between them."""
    import ctypes as C
    import torch
    from memfabric_hybrid_b200 import _native as N
    cu = N.cuda()
    cu.mf_xcopy_debug_probe.restype = C.c_int
    cu.mf_xcopy_debug_probe.argtypes = [C.POINTER(C.c_uint64), C.c_uint32, C.c_uint64, C.c_uint64, C.c_uint32, C.POINTER(C.c_uint64), C.c_int]
    r = np.random.default_rng(n)
    size = r.integers(1, 3000, n)
    s_off = np.concatenate(([0], np.cumsum(size + r.integers(1, 40, n))))
    d_off = np.concatenate(([0], np.cumsum(size + r.integers(1, 40, n))))
    src = torch.randint(1, 256, (int(s_off[-1]),), dtype=torch.uint8, device="cuda")
    dst = torch.zeros(int(d_off[-1]) + 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    trip = np.stack([src.data_ptr() + s_off[:-1], dst.data_ptr() + d_off[:-1], size], 1).reshape(-1)
    assert cu.mf_xcopy_debug_probe((C.c_uint64 * (3 * n))(*map(int, trip)), n, 0, 0, 0, None, 0) == 0
    torch.cuda.synchronize()
    a, got, want = src.cpu().numpy(), dst.cpu().numpy(), np.zeros(dst.numel(), dtype=np.uint8)
    for s, d, k in zip(s_off, d_off, size):
        want[d:d + k] = a[s:s + k]
    assert np.array_equal(got, want)


def _many_pieces_rank(rank, world, url):
    import torch
    import memfabric_hybrid as mf
    from memfabric_hybrid import bm
    from memfabric_hybrid_b200.ops.heap import tensor_at
    torch.cuda.set_device(0)
    torch.zeros(1, device="cuda")
    assert mf.initialize() == 0
    cfg = bm.BmConfig()
    cfg.rank_id = 0
    cfg.start_store = True
    assert bm.initialize(url, 1, 0, cfg) == 0, mf.get_last_err_msg()
    h = bm.create2(id=15, local_dram_size=0, max_dram_size=0, local_hbm_size=64 * MiB, max_hbm_size=64 * MiB)
    assert h.join() == 0, mf.get_last_err_msg()
    base = h.peer_rank_ptr(0, bm.BmMemType.DEVICE)
    bad = []
    # the register copy's grid is 296 CTAs here: one chunk each, a second one for a few, a full list each, and a second and third list
    for n in (1, 200, 296, 297, 9472, 9473, 20000):
        r = np.random.default_rng(n)
        size = r.integers(1, 1500, n)
        s_off = np.concatenate(([1], 1 + np.cumsum(size + r.integers(1, 40, n))))
        d_off = np.concatenate(([2], 2 + np.cumsum(size + r.integers(1, 40, n))))
        src = torch.randint(1, 256, (int(s_off[-1]),), dtype=torch.uint8, device="cuda")
        pool = tensor_at(base, (int(d_off[-1]) + 64,), torch.uint8)
        pool.zero_()
        torch.cuda.synchronize()
        lists = [src.data_ptr() + s_off[:-1].astype(np.uint64), base + d_off[:-1].astype(np.uint64), size.astype(np.uint64)]
        assert h.copy_data_batch(*lists, n, bm.BmCopyType.L2G, 0) == 0, mf.get_last_err_msg()
        a, got, want = src.cpu().numpy(), pool.cpu().numpy(), np.zeros(pool.numel(), dtype=np.uint8)
        for s, d, k in zip(s_off, d_off, size):
            want[d:d + k] = a[s:s + k]
        if not np.array_equal(got, want):
            bad.append(n)
    h.leave()
    h.destroy()
    bm.uninitialize(0)
    mf.uninitialize()
    return bad


def test_batches_of_more_pieces_than_the_ctas_lists_hold():
    url = f"tcp://127.0.0.1:{free_port()}"
    assert run_ranks(_many_pieces_rank, 1, (url,), timeout=300) == [[]]
