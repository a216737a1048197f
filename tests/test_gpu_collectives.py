"""Collective kernels against a plain PyTorch fp32 reference.

Single-GPU tests emulate all ranks in ONE cooperative launch (rank = blockIdx.y); the multi-GPU test runs
real ranks as child processes over NVLink peer mappings."""
import os

import pytest
import torch

from conftest import free_port
from mp_util import run_ranks

pytestmark = pytest.mark.gpu


def _tol(dtype):
    return dict(rtol=2e-2, atol=2e-2) if dtype in (torch.bfloat16, torch.float16) else dict(rtol=1e-5, atol=1e-5)


@pytest.fixture(scope="module")
def comms():
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    out = {}
    for w in (2, 4, 8):
        heap = EmulatedHeap(w, (1 << 20) + 4 * (2 << 20) + (1 << 20))
        out[w] = Communicator(heap, stage_bytes=2 << 20)
    yield out
    for c in out.values():
        torch.cuda.synchronize()
        assert c.heap.status()[0] == 0, f"a device wait gave up: {c.heap.status()}"


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("n", [8, 1000, 4096 + 24, 300_000, 1_500_000])
def test_all_reduce(comms, world, dtype, n):
    c = comms[world]
    torch.manual_seed(n + world)
    x = torch.randn(world, n, device="cuda", dtype=torch.float32).to(dtype)
    ref = x.float().sum(0) / world
    for algo in ("oneshot", "twoshot", None):
        if algo == "oneshot" and n * x.element_size() > c.stage_bytes:
            continue
        out = c.all_reduce(x, scale=1.0 / world, algo=algo)
        torch.cuda.synchronize()
        assert out.shape == (world, n)
        for r in range(world):
            torch.testing.assert_close(out[r].float(), ref, **_tol(dtype))
        assert torch.equal(out[0], out[world - 1]), "ranks must hold bit-identical results"


@pytest.mark.parametrize("world", [2, 8])
def test_all_reduce_fused_cast_and_ops(comms, world):
    c = comms[world]
    x = torch.randn(world, 70_000, device="cuda")
    out = c.all_reduce(x, scale=1.0 / world, out_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    assert out.dtype == torch.bfloat16
    torch.testing.assert_close(out[1].float(), (x.sum(0) / world), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(c.all_reduce(x, op="max")[0], x.max(0).values)
    torch.testing.assert_close(c.all_reduce(x, op="min")[0], x.min(0).values)
    xi = torch.randint(-1000, 1000, (world, 5000), device="cuda", dtype=torch.int32)
    assert torch.equal(c.all_reduce(xi)[0], xi.sum(0).to(torch.int32))
    assert torch.equal(c.all_reduce(xi, op="max", algo="twoshot")[world - 1], xi.max(0).values)


@pytest.mark.parametrize("n", [100, 200_000])
def test_all_reduce_into_a_given_output(comms, n):
    """What is stored are values of out_dtype, or of the input's type: an output of another type of that size receives their bits. Where they would not fit the output's
    elements, values of its own type."""
    c, world = comms[4], 4
    x = torch.randn(world, n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(torch.bfloat16)
    bits = torch.zeros(world, n, dtype=torch.int16, device="cuda")
    assert c.all_reduce(x, out=bits) is bits
    want = c.all_reduce(x)
    assert torch.equal(bits.view(torch.bfloat16), want)
    y = x.float()
    words = torch.zeros(world, n, dtype=torch.int32, device="cuda")
    assert torch.equal(c.all_reduce(y, out=words).view(torch.float32), c.all_reduce(y))
    assert torch.equal(c.all_reduce(y, out=torch.empty_like(x)), want)   # the same sums, rounded once
    wide = torch.zeros(world, n, dtype=torch.float32, device="cuda")
    c.all_reduce(y, out=wide, out_dtype=torch.bfloat16)
    got = wide.view(torch.bfloat16)   # rows of the output are 2 n values apart
    assert torch.equal(got[:, :n], want) and not bool(got[:, n:].any())
    torch.cuda.synchronize()
    assert c.heap.status()[0] == 0


@pytest.mark.parametrize("world,m", [(2, 8 << 20), (4, 2 << 20), (8, 512 << 10)])
def test_all_reduce_on_both_sides_of_one_shot(world, m):
    """The largest calls of one shot and the smallest of two, in one buffer and in pieces of the staging area: the same sum in rank order, rounded once."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    for stage in (m + 4096, (m // 3 + 4095) // 4096 * 4096):
        heap = EmulatedHeap(world, (1 << 20) + 4 * stage + 4096)
        c = Communicator(heap, stage_bytes=stage)
        for n in (m // 2 - 1, m // 2, m // 2 + 1):
            x = torch.randn(world, n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(torch.bfloat16)
            acc = x[0].float()
            for r in range(1, world):
                acc = acc + x[r].float()
            assert torch.equal(c.all_reduce(x), acc.to(torch.bfloat16).expand(world, n)), (stage, n)
        torch.cuda.synchronize()
        assert heap.status()[0] == 0


@pytest.mark.parametrize("world,n", [(2, 262_145), (2, 262_143), (2, 1_000_003), (3, 262_149), (4, 700_001), (8, 147_465)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_one_shot_into_outputs_off_16_bytes(world, n, dtype):
    """Around two vectors per thread, where the sums start to go through the staging area: every offset of the output, also in place; the fp32 sum in rank order."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = EmulatedHeap(world, (1 << 20) + 4 * (3 << 20) + 4096)
    c = Communicator(heap, stage_bytes=3 << 20)
    x = torch.randn(world, n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(dtype)
    acc = x[0].float()
    for r in range(1, world):
        acc = acc + x[r].float()
    want = (acc * 0.5).to(dtype).expand(world, n)
    for off in range(8):
        room = torch.full((world * n + 16,), 7, device="cuda", dtype=dtype)
        got = room[off:off + world * n].view(world, n)
        c.all_reduce(x, out=got, scale=0.5, algo="oneshot")
        assert torch.equal(got, want) and bool((room[:off] == 7).all()) and bool((room[off + world * n:] == 7).all()), off
        got.copy_(x)
        assert torch.equal(c.all_reduce(got, out=got, scale=0.5, algo="oneshot"), want), off
    torch.cuda.synchronize()
    assert heap.status()[0] == 0


@pytest.mark.parametrize("world", [2, 3, 8])
def test_small_all_reduce_in_packets(world):
    """Sizes that change from call to call (what an earlier call left in the packet area must not count), odd ones, inputs off eight bytes, in place, an output in
    the input's memory, every type: the fp32 sum in rank order, rounded once. 76 KiB is about where the staged kernel takes over."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = EmulatedHeap(world, (1 << 20) + 4 * (1 << 20) + 4096)
    c = Communicator(heap, stage_bytes=1 << 20)
    for k, n in enumerate([1, 7, 40_000, 513, 8, 38_912, 1021, 4096, 38_913, 19_456, 19_459, 3, 2048 // world, 2048 // world + 1]):
        g = torch.Generator("cuda").manual_seed(n)
        for dtype, out_dtype in ((torch.bfloat16, None), (torch.float32, None), (torch.float32, torch.bfloat16), (torch.float16, None), (torch.int32, None)):
            if dtype == torch.int32:
                x = torch.randint(-1000, 1000, (world, n), device="cuda", generator=g, dtype=dtype)
                want = x.sum(0).to(dtype)
            else:
                x = torch.randn(world, n, device="cuda", generator=g).to(dtype)
                acc = x[0].float()
                for r in range(1, world):
                    acc = acc + x[r].float()
                want = (acc * 0.5).to(out_dtype or dtype)
            scale = 1.0 if dtype == torch.int32 else 0.5
            want = want.expand(world, n)
            room = torch.full((world * n + 16,), 7, device="cuda", dtype=out_dtype or dtype)
            off = k % 8
            got = c.all_reduce(x, out=room[off:off + world * n].view(world, n), scale=scale, out_dtype=out_dtype)
            assert torch.equal(got, want) and bool((room[:off] == 7).all()) and bool((room[off + world * n:] == 7).all()), (n, dtype, out_dtype)
            assert torch.equal(c.all_reduce(x, scale=scale, out_dtype=out_dtype), want), (n, dtype, out_dtype)
            if out_dtype is None:
                wide = torch.empty(world * n + 5, dtype=dtype, device="cuda")
                y = wide[1:1 + world * n].view(world, n)
                y.copy_(x)
                assert torch.equal(c.all_reduce(y, out=y, scale=scale), want), (n, dtype)
                if n * x.element_size() <= 16 << 10:   # within a rank any overlap is fine; across ranks the staged kernel takes over, with one CTA per rank
                    y.copy_(x)
                    assert torch.equal(c.all_reduce(y, out=wide[4:4 + world * n].view(world, n), scale=scale), want), (n, dtype)
        if n > 1 and world == 8:
            assert torch.equal(c.all_reduce(x, op="max")[0], x.max(0).values)
    torch.cuda.synchronize()
    assert heap.status()[0] == 0


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [8, 1024, 50_000, 400_000])
def test_reduce_scatter_all_gather(comms, world, dtype, m):
    c = comms[world]
    x = torch.randn(world, world * m, device="cuda").to(dtype)
    rs = c.reduce_scatter(x, scale=1.0 / world)
    torch.cuda.synchronize()
    ref = x.float().sum(0).view(world, m) / world
    for r in range(world):
        torch.testing.assert_close(rs[r].float(), ref[r], **_tol(dtype))
    shard = torch.randn(world, m, device="cuda").to(dtype)
    ag = c.all_gather(shard)
    torch.cuda.synchronize()
    for r in range(world):
        assert torch.equal(ag[r].view(world, m), shard), f"rank {r}"
    if dtype == torch.float32:
        agc = c.all_gather(shard, out_dtype=torch.bfloat16)
        assert torch.equal(agc[0].view(world, m), shard.to(torch.bfloat16))


def _rank_order_sum(x):
    """fp32 sum of the ranks' rows in rank order, rounded once: what every rank has to hold, bit for bit."""
    acc = x[0].float()
    for r in range(1, x.shape[0]):
        acc = acc + x[r].float()
    return acc.to(x.dtype)


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [8, 1001, 4096, 70_001, 1_500_001])
def test_two_shot_all_reduce_in_place_and_off_16_bytes(comms, world, dtype, n):
    """A rank's own part is read from the input behind the first exchange, where it lies on 16 bytes; odd rows put some ranks' inputs off them. The
    largest size takes several pieces."""
    c = comms[world]
    x = torch.randn(world, n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(dtype)
    want = _rank_order_sum(x).expand(world, n)
    assert torch.equal(c.all_reduce(x, algo="twoshot"), want)
    y = x.clone()
    assert c.all_reduce(y, out=y, algo="twoshot") is y and torch.equal(y, want)
    shifted = torch.empty(world * n + 3, dtype=dtype, device="cuda")[3:].view(world, n)
    shifted.copy_(x)
    assert torch.equal(c.all_reduce(shifted, out=shifted, algo="twoshot"), want)


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [8, 125, 1001, 60_001])
def test_reduce_scatter_and_all_gather_of_odd_parts(comms, world, dtype, m):
    """Parts that start on and off 16 bytes, next to outputs that nothing else may be written to."""
    c = comms[world]
    gen = torch.Generator("cuda").manual_seed(m)
    x = torch.randn(world, world * m, device="cuda", generator=gen).to(dtype)
    assert torch.equal(c.reduce_scatter(x), _rank_order_sum(x).view(world, m))
    shard = torch.randn(world, m, device="cuda", generator=gen).to(dtype)
    room = torch.full((world * world * m + 8,), 7.0, device="cuda").to(dtype)
    out = room[3:3 + world * world * m].view(world, world * m)
    c.all_gather(shard, out=out)
    assert torch.equal(out, shard.reshape(1, -1).expand(world, -1))
    assert bool((room[:3] == 7).all()) and bool((room[3 + world * world * m:] == 7).all())


@pytest.mark.parametrize("world", [2, 8])
def test_reduce_scatter_and_all_gather_whose_output_lies_in_the_input(comms, world):
    """One CTA per rank: the exchange stands between the last read of any input and the first write to any output, so that every overlap is fine,
    of another type too."""
    c = comms[world]
    m = 4096 // world // world
    x0 = torch.randn(world, world * m, device="cuda", generator=torch.Generator("cuda").manual_seed(world))
    want = _rank_order_sum(x0).view(world, m)
    for off in (0, 4, 5, m, (world - 1) * (world * m)):
        x = x0.clone()
        assert torch.equal(c.reduce_scatter(x, out=x.view(-1)[off:off + world * m].view(world, m)), want), off
        x = x0.clone()
        out = x.view(-1).view(torch.bfloat16)[off * 2:off * 2 + world * m].view(world, m)
        assert torch.equal(c.reduce_scatter(x, out=out, out_dtype=torch.bfloat16), want.to(torch.bfloat16)), off
    m = 8192 // world
    shard = torch.randn(world, m, device="cuda", generator=torch.Generator("cuda").manual_seed(world)).to(torch.bfloat16)
    for off in (0, 3, 8, m, (world - 1) * world * m):
        out = torch.zeros(world, world * m, device="cuda", dtype=torch.bfloat16)
        x = out.view(-1)[off:off + world * m].view(world, m)
        x.copy_(shard)
        c.all_gather(x, out=out)
        assert torch.equal(out, shard.reshape(1, -1).expand(world, -1)), off


@pytest.mark.parametrize("world,stage_mb", [(2, 32), (3, 21), (4, 16), (5, 14), (8, 8), (16, 6)])
def test_large_reductions_whose_parts_are_pushed_in_chunks(world, stage_mb):
    """From 60 MiB over all ranks on, the parts travel in chunks while they are reduced: ends of chunks and of CTA ranges, inputs on and off 16 bytes, an
    output in the input's memory, every rank's sum in rank order bit for bit; just below, and by other numbers of ranks than 2, 4 and 8, the two passes."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = EmulatedHeap(world, (1 << 20) + 4 * (stage_mb << 20) + (1 << 20))
    c = Communicator(heap, stage_bytes=stage_mb << 20)
    line = (60 << 20) // world // world     # bytes of a part
    for dtype, shift, more in ((torch.float32, 0, 0), (torch.float32, 1, 36), (torch.bfloat16, 0, 8), (torch.bfloat16, 5, 1000), (torch.int32, 0, 4), (torch.float32, 0, -16)):
        es = 2 if dtype == torch.bfloat16 else 4
        m = -(-line // es) // 8 * 8 + 8 + more
        g = torch.Generator("cuda").manual_seed(m)
        flat = torch.empty(world * world * m + 8, dtype=dtype, device="cuda")
        x = flat[shift:shift + world * world * m].view(world, world * m)
        if dtype == torch.int32:
            x.copy_(torch.randint(-1000, 1000, x.shape, device="cuda", dtype=dtype, generator=g))
            want = x.sum(0).to(dtype)
        else:
            x.copy_(torch.randn(x.shape, device="cuda", generator=g).to(dtype))
            want = _rank_order_sum(x)
        room = torch.full((world * m + 16,), 7, device="cuda", dtype=dtype)
        c.reduce_scatter(x, out=room[8:8 + world * m].view(world, m))
        assert torch.equal(room[8:8 + world * m], want) and bool((room[:8] == 7).all()) and bool((room[8 + world * m:] == 7).all()), (dtype, shift)
        y = x.clone()
        assert torch.equal(c.all_reduce(y, out=y, algo="twoshot"), want.expand(world, -1)), (dtype, shift)
        z = y[:, :world * m - 3].contiguous().zero_() + x[:, :world * m - 3]     # a last part that is shorter
        assert torch.equal(c.all_reduce(z), want[:world * m - 3].expand(world, -1)), (dtype, shift)
        if dtype == torch.float32:
            assert torch.equal(c.reduce_scatter(x, scale=0.5, out_dtype=torch.bfloat16).view(-1), (want * 0.5).to(torch.bfloat16))
            assert torch.equal(c.reduce_scatter(x, op="max").view(-1), x.max(0).values)
        y = x.clone()
        assert torch.equal(c.reduce_scatter(y, out=y.view(-1)[:world * m].view(world, m)).reshape(-1), want), (dtype, shift)
    torch.cuda.synchronize()
    assert heap.status()[0] == 0


@pytest.mark.parametrize("world", [2, 3])
def test_collectives_whose_peers_never_come(world):
    """One rank alone with the slots of a group: what it sends lands in slots that nobody reads, and every wait of the calls ends at its limit, is reported with where it
    gave up and with the call's number, and leaves the GPU to the next call."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    stage = 32 << 20
    heap = EmulatedHeap(world, (1 << 20) + 4 * stage + 4096)
    heap.emu, heap.spin_limit = False, 2000   # under a millisecond
    c = Communicator(heap, stage_bytes=stage)
    big = (60 << 20) // world // 4 + 24       # fp32 values from which on two ranks push their parts in chunks
    big -= big % (8 * world)
    big += 8 * world
    calls = [(0x102, lambda: c.all_reduce(torch.ones(64, device="cuda", dtype=torch.bfloat16))),            # packets, one trip
             (0x102, lambda: c.all_reduce(torch.ones(20_000, device="cuda", dtype=torch.bfloat16))),        # two trips
             (0x100, lambda: c.all_reduce(torch.ones(100_000, device="cuda", dtype=torch.bfloat16))),       # staged, one shot
             (0x110, lambda: c.all_reduce(torch.ones(100_000, device="cuda", dtype=torch.bfloat16), algo="twoshot")),
             (0x118 if world == 2 else 0x110, lambda: c.all_reduce(torch.ones(big, device="cuda"), algo="twoshot")),
             (0x128 if world == 2 else 0x120, lambda: c.reduce_scatter(torch.ones(big, device="cuda"))),
             (0x120, lambda: c.reduce_scatter(torch.ones(8 * world, device="cuda"))),
             (0x130, lambda: c.all_gather(torch.ones(1000, device="cuda")))]
    for where, call in calls:
        call()
        torch.cuda.synchronize()
        code, at, epoch, count = heap.status()
        assert (code, at, epoch) == (1, where, c._epoch) and count > 0, (hex(at), hex(where))
        heap.clear_status()
    whole = EmulatedHeap(world, (1 << 20) + 4 * (1 << 20) + 4096)
    assert bool((Communicator(whole, stage_bytes=1 << 20).all_reduce(torch.ones(world, 64, device="cuda")) == world).all())
    torch.cuda.synchronize()
    assert whole.status()[0] == 0


@pytest.mark.parametrize("world", [2, 8])
def test_broadcast_scatter_alltoallv(comms, world):
    c = comms[world]
    x = torch.randn(world, 100_003, device="cuda")
    ref = x[world - 1].clone()
    c.broadcast(x, root=world - 1)
    torch.cuda.synchronize()
    for r in range(world):
        assert torch.equal(x[r], ref)
    # all-to-all-v with uneven counts: rank s sends (s + d + 1) * 16 elements to rank d
    cnt = [[(s + d + 1) * 16 + 3 for d in range(world)] for s in range(world)]
    soff = [[sum(cnt[s][:d]) for d in range(world)] for s in range(world)]
    rcnt = [[cnt[s][d] for s in range(world)] for d in range(world)]
    roff = [[sum(rcnt[d][:s]) for s in range(world)] for d in range(world)]
    nsend = max(sum(r) for r in cnt)
    nrecv = max(sum(r) for r in rcnt)
    xs = torch.randn(world, nsend, device="cuda").to(torch.bfloat16)
    out = torch.zeros(world, nrecv, device="cuda", dtype=torch.bfloat16)
    c.all_to_all_v(xs, out, cnt, soff, rcnt, roff)
    torch.cuda.synchronize()
    for d in range(world):
        for s in range(world):
            got = out[d, roff[d][s]:roff[d][s] + rcnt[d][s]]
            want = xs[s, soff[s][d]:soff[s][d] + cnt[s][d]]
            assert torch.equal(got, want), f"{s}->{d}"


def test_barrier_and_bounded_wait():
    """A wait that nothing satisfies ends with a status word, not a hang, and the context stays usable."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = EmulatedHeap(4, 8 << 20)
    heap.spin_limit = 20_000  # a few milliseconds
    c = Communicator(heap, stage_bytes=1 << 20)
    c.barrier()
    c.barrier(channel=3)
    torch.cuda.synchronize()
    assert heap.status()[0] == 0
    flag = heap.alloc(64)
    c.wait_flag_probe(flag, epoch=7)  # nobody ever writes this flag
    torch.cuda.synchronize()
    code, where, epoch, count = heap.status()
    assert code == 1 and where == 0x1ff and epoch == 7 and count == 1
    heap.clear_status()
    x = torch.ones(4, 64, device="cuda")
    assert torch.equal(c.all_reduce(x)[0], torch.full((64,), 4.0, device="cuda"))  # still healthy


def test_device_timeline_of_a_collective(tmp_path, comms):
    import json
    from memfabric_hybrid_b200.utils import devtrace
    devtrace.enable(lanes=64, per_lane=256)
    try:
        c = comms[4]
        x = torch.randn(4, 400_000, device="cuda")
        c.all_reduce(x, algo="twoshot")
        torch.cuda.synchronize()
        assert devtrace.count() > 0
        path = tmp_path / "t.json"
        n = devtrace.dump(str(path), rank=0)
        ev = json.loads(path.read_text())["traceEvents"]
        names = {e["name"] for e in ev}
        assert n == len(ev) and {"stage_in", "sync", "reduce", "copy_out"} <= names
        assert all(e["dur"] >= 0 and e["ph"] == "X" for e in ev)
        assert devtrace.count() == 0          # dump emptied the lanes
    finally:
        devtrace.disable()


def _real_ranks(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = SymmetricHeap(url, world, rank, rank % torch.cuda.device_count(), 128 << 20)
    c = Communicator(heap, stage_bytes=8 << 20)
    if os.environ.get("MF_SHM_MULTICAST"):
        c.multicast = True      # force the multicast kernels whatever the world size (the selector prefers peer loads / stores on 2 GPUs)
    def draw(r, n):
        return torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(1000 * r + n % 997)).to(torch.bfloat16)

    for n in (64, 10_000, 3_000_000):
        x = draw(rank, n)
        out = c.all_reduce(x, scale=1.0 / world)
        ref = sum(draw(r, n).float() for r in range(world)) / world
        torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)
    x = torch.full((world * 1024,), float(rank + 1), device="cuda")
    rs = c.reduce_scatter(x)
    assert torch.equal(rs, torch.full((1024,), float(sum(range(1, world + 1))), device="cuda"))
    ag = c.all_gather(torch.full((512,), float(rank), device="cuda"))
    assert torch.equal(ag.view(world, 512)[:, 0].cpu(), torch.arange(world, dtype=torch.float32))
    # direct mode: tensors that live in the heap are read and written in place by the peers (no staging)
    n = 1_000_000
    hx = heap.view(heap.alloc(n * 2), (n,), torch.bfloat16)
    ho = heap.view(heap.alloc(n * 2), (n,), torch.bfloat16)
    hx.copy_(draw(rank, n))
    ref = sum(draw(r, n).float() for r in range(world)) / world
    c.all_reduce(hx, out=ho, scale=1.0 / world, algo="direct")
    torch.testing.assert_close(ho.float(), ref, rtol=2e-2, atol=2e-2)
    c.all_reduce(hx, out=hx, scale=1.0 / world)  # in place
    torch.testing.assert_close(hx.float(), ref, rtol=2e-2, atol=2e-2)
    m = 200_000
    fx = heap.view(heap.alloc(world * m * 4), (world * m,), torch.float32)
    fx.copy_(torch.arange(world * m, device="cuda", dtype=torch.float32) % 1000 + rank)
    rs = c.reduce_scatter(fx)
    exp = (torch.arange(rank * m, (rank + 1) * m, device="cuda", dtype=torch.float32) % 1000) * world + sum(range(world))
    torch.testing.assert_close(rs, exp, rtol=1e-6, atol=1e-3)
    rs16 = c.reduce_scatter(fx, scale=0.5, out_dtype=torch.bfloat16)   # fused scale and cast in the epilogue
    torch.testing.assert_close(rs16.float(), exp * 0.5, rtol=1e-2, atol=1e-2)
    go = heap.view(heap.alloc(world * m * 4), (world * m,), torch.float32)
    c.all_gather(torch.full((m,), float(rank), device="cuda"), out=go)
    assert torch.equal(go.view(world, m)[:, m - 1].cpu(), torch.arange(world, dtype=torch.float32))
    # ring send/recv
    msg = torch.full((100_000,), float(rank), device="cuda")
    got = torch.empty_like(msg)
    nxt, prv = (rank + 1) % world, (rank - 1) % world
    if rank % 2 == 0:
        c.send(msg, nxt)
        c.recv(got, prv)
    else:
        c.recv(got, prv)
        c.send(msg, nxt)
    torch.cuda.synchronize()
    assert torch.equal(got, torch.full_like(got, float(prv)))
    c.barrier()
    torch.cuda.synchronize()
    st = heap.status()
    mc = heap.mc_base != 0
    heap.close()
    SymmetricHeap.shutdown()
    return st[0] if not os.environ.get("MF_SHM_MULTICAST") else (st[0], mc)


@pytest.mark.multigpu
def test_real_ranks_over_nvlink():
    n = min(torch.cuda.device_count(), 4)
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_real_ranks, n, (url,), timeout=300, with_barrier=True) == [0] * n


@pytest.mark.multigpu
def test_real_ranks_with_nvlink_multicast():
    """The same scenario with the multicast alias of the heap switched on: large all-reduces of heap tensors go
    through multimem load-reduce / store. No rank leaves early (a rank that dies while bound to a multicast
    object disturbs its peers)."""
    n = min(torch.cuda.device_count(), 4)
    url = f"127.0.0.1:{free_port()}"
    res = run_ranks(_real_ranks, n, (url,), timeout=300, with_barrier=True, env={"MF_SHM_MULTICAST": "1"})
    assert [r[0] for r in res] == [0] * n
    assert len({r[1] for r in res}) == 1      # every rank took the same decision about the alias


def _busy_ranks(rank, world, url, sync):
    """An all-reduce issued while matrix multiplications on another stream keep every SM busy: the collective's CTAs may
    have to queue behind them while the peer's CTAs already poll. It must either complete correctly or end with the clean
    time-out status of a bounded wait; it must not hang, and the context must stay usable."""
    import torch
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    heap = SymmetricHeap(url, world, rank, rank % torch.cuda.device_count(), 64 << 20)
    c = Communicator(heap, stage_bytes=8 << 20)
    side = torch.cuda.Stream()
    a = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    n = 1 << 20
    hx = heap.view(heap.alloc(n * 2), (n,), torch.bfloat16)
    ho = heap.view(heap.alloc(n * 2), (n,), torch.bfloat16)
    hx.fill_(float(rank + 1))
    small = torch.full((1000,), float(rank + 1), device="cuda")
    torch.cuda.synchronize()
    heap.host_barrier()
    outcomes = []
    for it in range(3):
        with torch.cuda.stream(side):
            for _ in range(12 if rank % 2 == 0 else 4):      # ranks are busy for different lengths of time (about 10 and 3 ms)
                torch.matmul(a, b)
        out_small = c.all_reduce(small)                       # staged path
        c.all_reduce(hx, out=ho)                              # direct path, peers read and write the heap tensors in place
        torch.cuda.synchronize()
        st = heap.status()
        if st[0] == 0:
            want = float(sum(range(1, world + 1)))
            assert torch.equal(out_small, torch.full_like(out_small, want))
            assert torch.equal(ho.float(), torch.full((n,), want, device="cuda"))
            outcomes.append("ok")
        else:
            assert st[0] == 1, st                             # ST_TIMEOUT of a bounded wait, nothing else
            heap.clear_status()
            outcomes.append("timeout")
        heap.host_barrier()
    # the context is still good for an undisturbed call
    got = c.all_reduce(small)
    torch.cuda.synchronize()
    ok = heap.status()[0] == 0 and torch.equal(got, torch.full_like(got, float(sum(range(1, world + 1)))))
    heap.close()
    SymmetricHeap.shutdown()
    return outcomes, bool(ok)


@pytest.mark.multigpu
def test_collective_while_compute_occupies_the_sms():
    n = 2
    url = f"127.0.0.1:{free_port()}"
    res = run_ranks(_busy_ranks, n, (url,), timeout=300, with_barrier=True)
    for outcomes, ok in res:
        assert ok and all(o in ("ok", "timeout") for o in outcomes), res
    assert any("ok" in o for o, _ in res), res   # 10 ms of queueing is far inside the waits' budget: it completes


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [1, 7, 33, 4099, 65_537])
def test_parts_that_do_not_end_on_16_bytes(comms, world, dtype, m):
    """Rows of the staging area start on 16 bytes whatever m is; what the user's buffers hold sits at any offset."""
    c = comms[world]
    torch.manual_seed(m + world)
    x = torch.randn(world, world * m, device="cuda").to(dtype)
    part = c.reduce_scatter(x, scale=1.0 / world)
    full = c.all_gather(part)
    torch.cuda.synchronize()
    ref = (x.double().sum(0) / world).view(world, m)
    # one rounding to the type of the fp32 sum of `world` terms
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    bound = ref.abs() * eps + x.double().abs().sum(0).view(world, m) / world * 2.0 ** -22
    assert ((part.double() - ref).abs() <= bound).all()
    for r in range(world):
        assert torch.equal(full[r].view(world, m), part)


@pytest.mark.parametrize("world", [2, 3, 8])
@pytest.mark.parametrize("dtype,n", [(torch.bfloat16, n) for n in (1023, 1024, 1025, 8184, 8192, 8193, 8200)] +
                         [(torch.float32, n) for n in (1023, 1025, 4088, 4096, 4097, 9000)])
def test_copies_around_two_vectors_per_thread(world, dtype, n):
    """One CTA's range around the line between the plain and the wide copy loop (two vectors, or two elements where the
    ends do not allow vectors, per thread of 512): broadcast and all-gather are copies, bit for bit."""
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    from memfabric_hybrid_b200.ops.collectives import Communicator
    c = Communicator(EmulatedHeap(world, (1 << 20) + 4 * (1 << 20) + (1 << 20)), stage_bytes=1 << 20, max_ctas=1)
    torch.manual_seed(n + world)
    x = torch.randn(world, n, device="cuda").to(dtype)
    out = torch.zeros(world, n, device="cuda", dtype=dtype)
    c.broadcast(x, world - 1, out=out)
    full = c.all_gather(x)
    torch.cuda.synchronize()
    assert c.heap.status()[0] == 0
    assert all(torch.equal(out[r], x[world - 1]) for r in range(world))
    assert all(torch.equal(full[r], x.view(-1)) for r in range(world))
