"""Workloads of the framework's public entry points on one GPU: KV-block copies into and out of the pooled HBM, the
quantising put, collectives, the tcgen05 GEMMs, the expert-parallel MoE layer (prefill, decode, low-latency pair) and the
fp8 tensor-parallel MLP. ``listed()`` are the sizes to look at first, ``draw()`` gives others of the same ranges.

One GPU is one rank: pool copies go to the rank's own slice, the MoE and tensor-parallel layers run the slice of a model
that one GPU of an 8-GPU box holds (32 of 256 experts, 1/8 of the FFN width), and the collectives run all ranks of a group
in one cooperative launch (``EmulatedHeap``), the library's own way of running several ranks' kernels on one device."""
from __future__ import annotations

import math
import socket
import weakref

import numpy as np
import torch

H_DSV3, I_DSV3, E_LOCAL, TOPK = 7168, 2048, 32, 8      # one GPU's part of the DeepSeek-V3 MoE layer at 8 GPUs
H_LLAMA, F_LLAMA = 8192, 3584                          # one GPU's part of the Llama-3-70B MLP at 8 GPUs
KV_SEGS = (128 << 10, 16 << 10)                        # a layer of a DeepSeek-R1 KV block (61 layers in all)


# ---------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one KV block (122 segments) handed to the next stage: the smallest transfer of a disaggregated server
        {"name": "kv_put_1_block", "op": "kv", "blocks": 1, "layers": 61, "get": False},
        # 64 blocks fetched from the pool: a long prompt's cache, the size the repository's benchmark moves
        {"name": "kv_get_64_blocks", "op": "kv", "blocks": 64, "layers": 61, "get": True},
        # pieces of any length at 2-byte alignment: packed, variable-length sequences of bf16 values
        {"name": "ragged_put", "op": "ragged", "pieces": 700, "longest": 512 << 10, "align": 2, "get": False},
        # bf16 rows quantised to fp8 (1 x 128 factors) on their way into the pool
        {"name": "quant_put_fp8", "op": "quant", "items": 512, "elems": 131072, "unit": 128, "fp8": True, "fp16": False},
        # tensor-parallel decode: the sum of one small activation over 8 ranks
        {"name": "allreduce_small", "op": "allreduce", "world": 8, "n": 4 * 7168, "dtype": "bf16", "out": "bf16"},
        # sharded optimiser: mean of the gradients (fp32, cast to bf16) scattered, then the shards gathered
        {"name": "shard_step_8x30MB", "op": "shard", "world": 8, "m": 983_040, "dtype": "fp32", "out": "bf16"},
        # a large projection in prefill
        {"name": "gemm_prefill", "op": "gemm", "m": 4096, "n": 4096, "k": 7168, "swiglu": False},
        # the MLP of a decode step: 32 sequences, one token each
        {"name": "mlp_decode_32", "op": "mlp", "tokens": 32},
        # the MoE layer on a prefill batch, and on a decode batch
        {"name": "moe_prefill_4096", "op": "moe", "tokens": 4096},
        {"name": "moe_decode_128", "op": "moe", "tokens": 128},
        # the low-latency dispatch / combine pair of a decode step, replayed as a CUDA graph as a server does
        {"name": "moe_ll_128", "op": "ll", "tokens": 128},
        # the fp8 MLP of a prefill batch
        {"name": "tp_mlp_fp8_4096", "op": "tp_fp8", "tokens": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["kv", "ragged", "quant", "allreduce", "shard", "gemm", "mlp", "moe", "moe", "ll", "tp_fp8"])
    if op == "kv":
        return {"op": op, "blocks": _log(rng, 1, 64), "layers": rng.randint(16, 61), "get": rng.random() < 0.5}
    if op == "ragged":
        return {"op": op, "pieces": _log(rng, 20, 1500), "longest": _log(rng, 4 << 10, 512 << 10), "align": rng.choice([1, 2, 4, 8, 16]),
                "get": rng.random() < 0.5}
    if op == "quant":
        fp8 = rng.random() < 0.5
        unit = 128 if fp8 else rng.choice([64, 128, 192, 576, 1024, 7168])
        return {"op": op, "items": _log(rng, 4, 512), "elems": unit * max(1, _log(rng, 1024, 131072) // unit), "unit": unit, "fp8": fp8,
                "fp16": rng.random() < 0.3}
    if op == "allreduce":
        dtype = rng.choice(["bf16", "fp16", "fp32"])
        n = _log(rng, 512, 8 << 20)
        return {"op": op, "world": rng.choice([2, 4, 8]), "n": n - n % 8 if rng.random() < 0.7 else n, "dtype": dtype,
                "out": "bf16" if dtype == "fp32" and rng.random() < 0.5 else dtype}
    if op == "shard":
        m = _log(rng, 1024, 1_000_000)
        dtype = rng.choice(["bf16", "fp32"])
        return {"op": op, "world": rng.choice([2, 4, 8]), "m": m - m % 8 if rng.random() < 0.7 else m, "dtype": dtype, "out": "bf16"}
    if op == "gemm":
        swiglu = rng.random() < 0.3
        n = 256 * _log(rng, 2, 28) if swiglu else 8 * _log(rng, 32, 1024)
        return {"op": op, "m": _log(rng, 1, 4096), "n": n, "k": 64 * _log(rng, 8, 128), "swiglu": swiglu}
    if op == "mlp":
        return {"op": op, "tokens": _log(rng, 1, 512)}
    if op == "moe":
        return {"op": op, "tokens": _log(rng, 1, 4096)}
    if op == "ll":
        return {"op": op, "tokens": _log(rng, 1, 256)}
    return {"op": op, "tokens": 128 * _log(rng, 1, 32)}


# ---------------------------------------------------------------------------------------------------- what a program keeps
_POOL_BYTES = 6 << 30
_keep: dict = {}


def _port():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _pool():
    """The process's pooled HBM (one rank) and the free regions of its own slice."""
    if "pool" not in _keep:
        import memfabric_hybrid as mf
        from memfabric_hybrid import bm
        torch.zeros(1, device="cuda")
        mf.initialize()
        cfg = bm.BmConfig()
        cfg.rank_id = 0
        cfg.start_store = True
        assert bm.initialize(f"tcp://127.0.0.1:{_port()}", 1, 0, cfg) == 0, mf.get_last_err_msg()
        h = bm.create2(id=0, local_dram_size=0, max_dram_size=0, local_hbm_size=_POOL_BYTES, max_hbm_size=_POOL_BYTES,
                       data_op_type=bm.BmDataOpType.SDMA)
        assert h.join() == 0, mf.get_last_err_msg()
        _keep["pool"] = (bm, h, h.peer_rank_ptr(0, bm.BmMemType.DEVICE), [(0, _POOL_BYTES)])
        _keep["copy_stream"] = torch.cuda.Stream()
    return _keep["pool"]


def _give_back(free, off, size):
    free.append((off, size))
    free.sort()
    out = []
    for o, s in free:
        if out and out[-1][0] + out[-1][1] == o:
            out[-1] = (out[-1][0], out[-1][1] + s)
        else:
            out.append((o, s))
    free[:] = out


class _State:
    pass


def _region(st, nbytes):
    """A piece of the pool for the life of ``st``: its address and a byte tensor over it, zeroed."""
    from memfabric_hybrid_b200.ops.heap import tensor_at
    _, _, base, free = _pool()
    size = (nbytes + (2 << 20) - 1) // (2 << 20) * (2 << 20)
    for i, (o, s) in enumerate(free):
        if s >= size:
            free[i:i + 1] = [(o + size, s - size)] if s > size else []
            weakref.finalize(st, _give_back, free, o, size)
            t = tensor_at(base + o, (nbytes,), torch.uint8)
            t.zero_()
            return base + o, t
    raise torch.cuda.OutOfMemoryError("out of memory: the pool has no free region of that size")


def _heap():
    """The process's symmetric heap (one rank): the MoE and tensor-parallel communicators live in it."""
    if "heap" not in _keep:
        from memfabric_hybrid_b200.ops.heap import SymmetricHeap
        _keep["heap"] = SymmetricHeap(f"127.0.0.1:{_port()}", 1, 0, 0, 2 << 30)
    return _keep["heap"]


def _moe_comm():
    if "moe" not in _keep:
        from memfabric_hybrid_b200.ops.moe import MoEComm
        _keep["moe"] = MoEComm(_heap(), 4096, H_DSV3, E_LOCAL, TOPK, max_recv=4096 * TOPK, intermediate=I_DSV3)
    return _keep["moe"]


def _ll_comm():
    if "ll" not in _keep:
        from memfabric_hybrid_b200.ops.moe import MoEComm
        _keep["ll"] = MoEComm(_heap(), 256, H_DSV3, E_LOCAL, TOPK, max_recv=256 * TOPK)
    return _keep["ll"]


def _tp():
    if "tp" not in _keep:
        from memfabric_hybrid_b200.ops.tp import TensorParallel
        _keep["tp"] = TensorParallel(_heap(), 8192, H_LLAMA, fp8=True)
    return _keep["tp"]


def _comm(world):
    if ("comm", world) not in _keep:
        from memfabric_hybrid_b200.ops.collectives import Communicator
        from memfabric_hybrid_b200.ops.heap import EmulatedHeap
        stage = 32 << 20
        _keep["comm", world] = Communicator(EmulatedHeap(world, 4 * stage + (2 << 20)), stage_bytes=stage)
    return _keep["comm", world]


# ---------------------------------------------------------------------------------------------------- inputs
_DT = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _gen(seed, salt=0):
    return torch.Generator("cuda").manual_seed(int(seed) * 1009 + salt)


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    t = torch.randn(*shape, device="cuda", generator=g)
    if scale != 1.0:
        t *= scale
    return t.to(dtype)


def _kv_bytes(case):
    return case["blocks"] * case["layers"] * sum(KV_SEGS)


def _kv_segments(blocks, layers):
    """(offset, size) of every segment, block after block: per layer an array [blocks, 128 KiB] and one [blocks, 16 KiB]."""
    out = []
    for b in range(blocks):
        base = 0
        for _ in range(layers):
            for seg in KV_SEGS:
                out.append((base + b * seg, seg))
                base += blocks * seg
    return out


def _ragged_segments(case):
    """(source offset, destination offset, size): pieces of log-uniform length with gaps, in another order at the destination.
    One layout per case (the buffers keep their sizes); the seed fills it with other bytes."""
    r = np.random.default_rng([case["pieces"], case["longest"], case["align"]])
    al, n = case["align"], case["pieces"]
    size = np.maximum(al, (np.exp(r.uniform(math.log(256), math.log(case["longest"]), n)) // al * al)).astype(np.int64)
    gap = r.integers(1, 64, (2, n)) * al
    s_off = np.cumsum(np.concatenate(([0], (size + gap[0])[:-1]))) + gap[0][0]
    order = r.permutation(n)
    d_off = np.empty(n, np.int64)
    d_off[order] = np.cumsum(np.concatenate(([0], (size + gap[1])[order][:-1]))) + gap[1][0]
    return s_off, d_off, size, int((s_off + size).max()), int((d_off + size).max())


def _bytes(g, n):
    return torch.randint(-128, 128, (n,), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8)


def _moe_inputs(case, seed):
    g = _gen(seed, 1)
    x = _randn(g, case["tokens"], H_DSV3)
    p = torch.softmax(torch.randn(case["tokens"], E_LOCAL, device="cuda", generator=g), -1)
    w, idx = torch.topk(p, TOPK, dim=-1)
    return x, idx.to(torch.int32).contiguous(), (w / w.sum(-1, keepdim=True)).contiguous()


def _expert(seed, e):
    """bf16 master weights of expert e: gate and up rows, down rows."""
    g = _gen(seed, 100 + e)
    return _randn(g, 2 * I_DSV3, H_DSV3, scale=0.02), _randn(g, H_DSV3, I_DSV3, scale=0.02)


def _tp_inputs(case, seed):
    g = _gen(seed, 2)
    return (_randn(g, case["tokens"], H_LLAMA), _randn(g, F_LLAMA, H_LLAMA, scale=0.02), _randn(g, F_LLAMA, H_LLAMA, scale=0.02),
            _randn(g, H_LLAMA, F_LLAMA, scale=0.02))


def _ranks_inputs(case, seed):
    n = case["n"] if case["op"] == "allreduce" else case["m"] * case["world"]
    return _randn(_gen(seed, 3), case["world"], n, dtype=_DT[case["dtype"]])


def _gemm_inputs(case, seed):
    g = _gen(seed, 4)
    return _randn(g, case["m"], case["k"]), _randn(g, case["n"], case["k"], scale=0.05)


def _quant_inputs(case, seed):
    return _randn(_gen(seed, 5), case["items"], case["elems"], dtype=torch.float16 if case["fp16"] else torch.bfloat16)


# ---------------------------------------------------------------------------------------------------- one pass
def prepare(case, seed):
    st = _State()
    st.case, op = case, case["op"]
    getattr(_Prepare, op)(st, case, seed)
    torch.cuda.synchronize()
    return st


def run(st):
    return getattr(_Run, st.case["op"])(st)


class _Prepare:
    @staticmethod
    def kv(st, case, seed):
        segs = _kv_segments(case["blocks"], case["layers"])
        total = _kv_bytes(case)
        addr, pool = _region(st, total)
        mine = torch.zeros(total, dtype=torch.uint8, device="cuda")
        (pool if case["get"] else mine).copy_(_bytes(_gen(seed), total))
        st.out, st.keep = (mine, pool) if case["get"] else (pool, mine)
        a = np.array([o for o, _ in segs], dtype=np.uint64)
        _Prepare._lists(st, case, mine, addr, a, a, np.array([s for _, s in segs], dtype=np.uint64))

    @staticmethod
    def ragged(st, case, seed):
        s_off, d_off, size, s_end, d_end = _ragged_segments(case)
        g = _gen(seed)
        addr, pool = _region(st, s_end if case["get"] else d_end)
        mine = torch.zeros(d_end if case["get"] else s_end, dtype=torch.uint8, device="cuda")
        (pool if case["get"] else mine).copy_(_bytes(g, s_end))
        st.out, st.keep = (mine, pool) if case["get"] else (pool, mine)
        _Prepare._lists(st, case, mine, addr, (d_off if case["get"] else s_off).astype(np.uint64),
                        (s_off if case["get"] else d_off).astype(np.uint64), size.astype(np.uint64))

    @staticmethod
    def _lists(st, case, mine, addr, off_mine, off_pool, size):
        """The descriptor lists as a serving engine keeps them: arrays of 64-bit addresses and sizes."""
        bm, st.pool, _, _ = _pool()
        a, b = off_mine + np.uint64(mine.data_ptr()), off_pool + np.uint64(addr)
        st.src, st.dst = (b, a) if case["get"] else (a, b)
        st.size, st.count = size, len(size)
        st.kind = bm.BmCopyType.G2L if case["get"] else bm.BmCopyType.L2G
        st.flags = bm.ASYNC_COPY_FLAG | bm.FLAG_USE_EXTERNAL_STREAM
        _Prepare._events(st)

    @staticmethod
    def _events(st):
        st.stream = _keep["copy_stream"]
        st.before, st.after = torch.cuda.Event(), torch.cuda.Event()

    @staticmethod
    def quant(st, case, seed):
        st.x = _quant_inputs(case, seed)
        n, per, unit = case["items"], case["elems"], case["unit"]
        total, factors = n * per, n * (per // unit)
        pad = (total + 255) // 256 * 256
        addr, pool = _region(st, pad + factors * 4)
        st.out = {"q": pool[:total], "factor": pool[pad:pad + factors * 4].view(torch.float32)}
        _, st.pool, _, _ = _pool()
        src = st.x.data_ptr()
        st.batch = st.pool.prepare_quant_batch([src + i * per * 2 for i in range(n)], [addr + i * per for i in range(n)], [per * 2] * n,
                                               [addr + pad + i * (per // unit) * 4 for i in range(n)], unit, fp8=case["fp8"],
                                               fp16_input=case["fp16"])
        _Prepare._events(st)

    @staticmethod
    def allreduce(st, case, seed):
        st.comm, st.x, st.dtype = _comm(case["world"]), _ranks_inputs(case, seed), _DT[case["out"]]

    shard = allreduce

    @staticmethod
    def gemm(st, case, seed):
        st.a, st.b = _gemm_inputs(case, seed)

    @staticmethod
    def mlp(st, case, seed):
        from memfabric_hybrid_b200.ops.gemm import interleave_gate_up
        st.x, gate, up, st.down = _tp_inputs(case, seed)
        st.gate_up = interleave_gate_up(gate, up)

    @staticmethod
    def moe(st, case, seed):
        from memfabric_hybrid_b200.ops import moe as M
        st.comm = _moe_comm()
        st.x, st.idx, st.w = _moe_inputs(case, seed)
        parts = [[], [], [], []]
        for e in range(E_LOCAL):
            w1, w2 = _expert(seed, e)
            for out, t in zip(parts, M.quantize_weight_fp8(w1) + M.quantize_weight_fp8(w2)):
                out.append(t)
        w1q, st.w1s, st.w2q, st.w2s = (torch.stack(p) for p in parts)
        st.w1q = M.interleave_gate_up_fp8(w1q)

    @staticmethod
    def ll(st, case, seed):
        st.comm = _ll_comm()
        st.x, st.idx, st.w = _moe_inputs(case, seed)
        st.rows = case["tokens"] * TOPK
        st.out = torch.empty(case["tokens"], H_DSV3, dtype=torch.bfloat16, device="cuda")
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _ll_pass(st)
        torch.cuda.synchronize()
        st.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st.graph):
            st.row_off = _ll_pass(st)

    @staticmethod
    def tp_fp8(st, case, seed):
        from memfabric_hybrid_b200.ops import moe as M
        st.tp = _tp()
        st.x, gate, up, down = _tp_inputs(case, seed)
        q, st.s1 = M.quantize_weight_fp8(torch.cat([gate, up]))
        st.q1 = M.interleave_gate_up_fp8(q[None], 128)[0]
        st.q2, st.s2 = M.quantize_weight_fp8(down)


def _ll_pass(st):
    """Rows travel to their experts as block-scaled fp8, an expert that returns its rows as they are answers, and the
    weighted answers are summed: the output is the input rounded to fp8."""
    d = st.comm.ll_dispatch(st.x, st.idx, st.w)
    q, s = st.comm.recv_x()[:st.rows], st.comm.recv_scale()[:st.rows]
    y = (q.float().view(st.rows, H_DSV3 // 128, 128) * s.view(st.rows, H_DSV3 // 128, 1)).view(st.rows, H_DSV3).to(torch.bfloat16)
    st.comm.ll_combine(y, d, out=st.out)
    return d.row_off


class _Run:
    @staticmethod
    def kv(st):
        cur = torch.cuda.current_stream()
        st.before.record(cur)
        st.stream.wait_event(st.before)
        rc = st.pool.copy_data_batch(st.src, st.dst, st.size, st.count, st.kind, st.flags, st.stream.cuda_stream)
        if rc != 0:
            raise RuntimeError(f"copy_data_batch: {rc}")
        st.after.record(st.stream)
        cur.wait_event(st.after)
        return st.out

    ragged = kv

    @staticmethod
    def quant(st):
        cur = torch.cuda.current_stream()
        st.before.record(cur)
        st.stream.wait_event(st.before)
        rc = st.pool.quant_copy_prepared(st.batch, st.stream.cuda_stream)
        if rc != 0:
            raise RuntimeError(f"quant_copy_prepared: {rc}")
        st.after.record(st.stream)
        cur.wait_event(st.after)
        return st.out

    @staticmethod
    def allreduce(st):
        return st.comm.all_reduce(st.x, scale=1.0 / st.comm.world, out_dtype=st.dtype)

    @staticmethod
    def shard(st):
        part = st.comm.reduce_scatter(st.x, scale=1.0 / st.comm.world, out_dtype=st.dtype)
        return {"part": part, "full": st.comm.all_gather(part)}

    @staticmethod
    def gemm(st):
        from memfabric_hybrid_b200.ops.gemm import gemm_bf16
        return gemm_bf16(st.a, st.b, swiglu=st.case["swiglu"])

    @staticmethod
    def mlp(st):
        from memfabric_hybrid_b200.ops.gemm import gemm_bf16
        h = gemm_bf16(st.x, st.gate_up, swiglu=True)
        return {"h": h, "y": gemm_bf16(h, st.down)}

    @staticmethod
    def moe(st):
        d = st.comm.dispatch(st.x, st.idx, st.w)
        st.comm.expert_ffn(d, st.w1q, st.w1s, st.w2q, st.w2s)
        return {"y": st.comm.combine(d), "tokens_per_expert": d.tokens_per_expert, "row_off": d.row_off}

    @staticmethod
    def ll(st):
        st.graph.replay()
        return {"y": st.out, "row_off": st.row_off}

    @staticmethod
    def tp_fp8(st):
        hq, hs = st.tp.ag_gemm_fp8(st.x, st.q1, st.s1)
        return st.tp.gemm_rs_fp8(hq, hs, st.q2, st.s2)


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    op = case["op"]
    if op == "kv":
        return {"bytes": 2 * _kv_bytes(case), "flops": 0}
    if op == "ragged":
        mean = (case["longest"] - 256) / math.log(case["longest"] / 256)   # of a log-uniform length
        return {"bytes": int(2 * case["pieces"] * mean), "flops": 0}
    if op == "quant":
        n = case["items"] * case["elems"]
        return {"bytes": 3 * n + 4 * n // case["unit"], "flops": 0}
    size = {"bf16": 2, "fp16": 2, "fp32": 4}
    if op == "allreduce":
        n = case["world"] * case["n"]
        return {"bytes": n * (size[case["dtype"]] + size[case["out"]]), "flops": n}
    if op == "shard":
        n = case["world"] * case["m"]
        return {"bytes": n * case["world"] * (size[case["dtype"]] + size[case["out"]]) + 2 * n * size[case["out"]], "flops": n * case["world"]}
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * (n // 2 if case["swiglu"] else n)), "flops": 2 * m * n * k}
    t = case["tokens"]
    if op in ("mlp", "tp_fp8"):
        weight = 3 * F_LLAMA * H_LLAMA
        return {"bytes": weight * (2 if op == "mlp" else 1) + 2 * t * (2 * H_LLAMA + (F_LLAMA if op == "mlp" else 0)), "flops": 2 * t * weight}
    if op == "ll":
        return {"bytes": 2 * t * H_DSV3 * 2, "flops": 2 * t * TOPK * H_DSV3}
    expert = 3 * H_DSV3 * I_DSV3
    used = E_LOCAL * (1 - (1 - TOPK / E_LOCAL) ** t)   # experts that get a token
    return {"bytes": int(used * expert) + 2 * t * H_DSV3 * 2, "flops": 2 * t * TOPK * expert}


def tolerance(case):
    op = case["op"]
    if op in ("kv", "ragged"):
        return "exact"
    if op == "quant":
        # factors are fp32 quotients; a value on a rounding boundary may fall either way
        return {"rel": 1e-6, "differ": 1e-4}
    if op in ("allreduce", "shard"):
        # one rounding to the output type of an fp32 sum
        return {"rel": 1e-6} if case["out"] == "fp32" else {"rel": 1e-3, "max": 2e-2}
    if op in ("gemm", "mlp"):
        return {"rel": 4e-3, "max": 4e-2}
    if op == "ll":
        return {"rel": 4e-3, "max": 4e-2}
    # the activations between the two GEMMs are rounded to bf16 and then to fp8 (or to fp8 at once): one in about thirty
    # falls on the other side of a boundary, 1.6e-2 of the result's norm
    return {"rel": 3e-2, "max": 2e-1}


# ---------------------------------------------------------------------------------------------------- in 64 bits
def _fp8_blocks(t, dims):
    """Values after rounding to e4m3 with one power-of-two factor per block of 128 along ``dims`` of the last two axes."""
    r, c = t.shape
    br, bc = (128 if 0 in dims else 1), (128 if 1 in dims else 1)
    b = t.double().reshape(r // br, br, c // bc, bc)
    amax = b.abs().amax(dim=(1, 3), keepdim=True).clamp_min(1e-30)
    f = torch.exp2(torch.ceil(torch.log2(amax / 448.0))).clamp_min(2.0 ** -126)
    return ((b / f).to(torch.float32).to(torch.float8_e4m3fn).double() * f).reshape(r, c)


def _swiglu(g, u):
    return g * torch.sigmoid(g) * u


def exact(case, seed):
    return getattr(_Exact, case["op"])(case, seed)


class _Exact:
    @staticmethod
    def kv(case, seed):
        return _bytes(_gen(seed), _kv_bytes(case))

    @staticmethod
    def ragged(case, seed):
        s_off, d_off, size, s_end, d_end = _ragged_segments(case)
        src = _bytes(_gen(seed), s_end)
        out = torch.zeros(d_end, dtype=torch.uint8, device="cuda")
        for s, d, n in zip(s_off.tolist(), d_off.tolist(), size.tolist()):
            out[d:d + n] = src[s:s + n]
        return out

    @staticmethod
    def quant(case, seed):
        x = _quant_inputs(case, seed).double().view(-1, case["unit"])
        top = 448.0 if case["fp8"] else 127.0
        amax = x.abs().amax(1, keepdim=True)
        factor = torch.where(amax > 0, amax / top, torch.ones_like(amax))
        v = x / factor
        q = v.float().to(torch.float8_e4m3fn).view(torch.uint8) if case["fp8"] else v.round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
        return {"q": q.view(-1), "factor": factor.view(-1)}

    @staticmethod
    def allreduce(case, seed):
        x = _ranks_inputs(case, seed)
        return (x.double().sum(0, keepdim=True) / case["world"]).expand(case["world"], -1)

    @staticmethod
    def shard(case, seed):
        total = _Exact.allreduce(case, seed)[0]
        return {"part": total.view(case["world"], case["m"]), "full": total.expand(case["world"], -1)}

    @staticmethod
    def gemm(case, seed):
        a, b = (t.double() for t in _gemm_inputs(case, seed))
        c = a @ b.t()
        if case["swiglu"]:
            c = c.view(case["m"], case["n"] // 256, 2, 128)
            c = _swiglu(c[:, :, 0], c[:, :, 1]).reshape(case["m"], case["n"] // 2)
        return c

    @staticmethod
    def mlp(case, seed):
        x, gate, up, down = (t.double() for t in _tp_inputs(case, seed))
        h = _swiglu(x @ gate.t(), x @ up.t())
        return {"h": h, "y": h.float().to(torch.bfloat16).double() @ down.t()}

    @staticmethod
    def moe(case, seed):
        x, idx, w = _moe_inputs(case, seed)
        xq = _fp8_blocks(x, (1,))
        y = torch.zeros(case["tokens"], H_DSV3, dtype=torch.float64, device="cuda")
        counts = []
        for e in range(E_LOCAL):
            tok, k = (idx == e).nonzero(as_tuple=True)
            counts.append(tok.numel())
            if not counts[-1]:
                continue
            w1, w2 = (_fp8_blocks(t, (0, 1)) for t in _expert(seed, e))
            gu = xq[tok] @ w1.t()
            h = _fp8_blocks(_swiglu(gu[:, :I_DSV3], gu[:, I_DSV3:]), (1,))
            y.index_add_(0, tok, (h @ w2.t()) * w[tok, k].double()[:, None])
        n = torch.tensor(counts, dtype=torch.int32, device="cuda")
        return {"y": y, "tokens_per_expert": n, "row_off": torch.cat([n.new_zeros(1), n.cumsum(0).to(torch.int32)])}

    @staticmethod
    def ll(case, seed):
        x, idx, w = _moe_inputs(case, seed)
        n = torch.bincount(idx.view(-1).long(), minlength=E_LOCAL)
        return {"y": _fp8_blocks(x, (1,)) * w.double().sum(1, keepdim=True),
                "row_off": torch.cat([n.new_zeros(1), n.cumsum(0)]).to(torch.int32)}

    @staticmethod
    def tp_fp8(case, seed):
        x, gate, up, down = _tp_inputs(case, seed)
        gate, up, down = (_fp8_blocks(t, (0, 1)) for t in (gate, up, down))
        xq = _fp8_blocks(x, (1,))
        return _fp8_blocks(_swiglu(xq @ gate.t(), xq @ up.t()), (1,)) @ down.t()
