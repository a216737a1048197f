"""MoE expert parallelism: layout, fp8 dispatch, grouped fp8 GEMMs and combine against fp32 references."""
import pytest
import torch

from conftest import free_port
from mp_util import run_ranks

pytestmark = pytest.mark.gpu


def _deq(q, s):
    """fp8 rows [R, K] with 1x128 scales [R, K/128] -> fp32."""
    R, K = q.shape
    return (q.float().view(R, K // 128, 128) * s[:, :, None]).view(R, K)


def _deq_w(q, s):
    *lead, Nn, K = q.shape
    return (q.float().reshape(*lead, Nn // 128, 128, K // 128, 128) * s[..., :, None, :, None]).reshape(*lead, Nn, K)


def test_grouped_gemm_fp8_plain_and_swiglu():
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    torch.manual_seed(0)
    G, N, K = 4, 256, 512
    counts = [130, 0, 7, 300]
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    R = sum(counts)
    x = torch.randn(R, K, device="cuda").to(torch.bfloat16)
    xq = torch.empty(R, K, dtype=torch.uint8, device="cuda")
    xs = torch.empty(R, K // 128, dtype=torch.float32, device="cuda")
    assert cu.mf_quant_rows_fp8(x.data_ptr(), K, off[G:].data_ptr(), K, xq.data_ptr(), xs.data_ptr(), 64,
                                torch.cuda.current_stream().cuda_stream) == 0
    xd = _deq(xq.view(torch.float8_e4m3fn), xs)
    assert (xd - x.float()).abs().max() <= 0.07 * x.float().abs().max()
    w = (torch.randn(G, N, K, device="cuda") * 0.05).to(torch.bfloat16)
    wq, ws = M.quantize_weight_fp8(w)
    wd = _deq_w(wq, ws)
    out = torch.zeros(R, N, dtype=torch.bfloat16, device="cuda")
    st = gemm.status_word()
    rc = cu.mf_grouped_gemm_fp8(xq.data_ptr(), xs.data_ptr(), R, wq.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, out.data_ptr(), N, 0,
                                None, None, 0, 1, st.data_ptr(), gemm.sm_count(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    gemm.check_status()
    ref = torch.cat([xd[off[g]:off[g + 1]] @ wd[g].t() for g in range(G)])
    assert (out.float() - ref).abs().max() <= 2e-2 * ref.abs().max() + 1e-3
    # SwiGLU: B rows are [gate (N/2) | up (N/2)]; the kernel takes the tile-interleaved copy
    wi = M.interleave_gate_up_fp8(wq, tile=64)   # the 128 x 128 kernel pairs 64 gate rows with 64 up rows
    out2 = torch.zeros(R, N // 2, dtype=torch.bfloat16, device="cuda")
    rc = cu.mf_grouped_gemm_fp8(xq.data_ptr(), xs.data_ptr(), R, wi.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, out2.data_ptr(), N // 2,
                                1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    gemm.check_status()
    ref2 = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
    assert (out2.float() - ref2).abs().max() <= 3e-2 * ref2.abs().max() + 1e-3


@pytest.mark.parametrize("G,N,K,counts", [(4, 256, 512, [130, 0, 7, 300]), (3, 512, 768, [1, 257, 128]), (2, 1024, 2048, [640, 513])])
def test_grouped_gemm_fp8_block_scaled(G, N, K, counts):
    """The 128 x 256 kernel whose scales are applied by the tensor core (UE8M0 bytes in TMEM): plain, SwiGLU, and
    SwiGLU + re-quantisation epilogues against fp32 references on the dequantised operands. K = 768 has a partial
    group of K blocks (6 = 4 + 2)."""
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    torch.manual_seed(G * N + K)
    s = torch.cuda.current_stream().cuda_stream
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    R = sum(counts)
    # rows of very different magnitude, so that a wrong scale byte or a wrong row shows
    x = (torch.randn(R, K, device="cuda") * torch.logspace(-2, 2, R, device="cuda")[:, None]).to(torch.bfloat16)
    xq = torch.empty(R, K, dtype=torch.uint8, device="cuda")
    xs = torch.empty(R, K // 128, dtype=torch.float32, device="cuda")
    assert cu.mf_quant_rows_fp8(x.data_ptr(), K, off[G:].data_ptr(), K, xq.data_ptr(), xs.data_ptr(), 64, s) == 0
    assert torch.equal(xs, torch.exp2(torch.round(torch.log2(xs)))), "activation scales must be powers of two"
    xd = _deq(xq.view(torch.float8_e4m3fn), xs)
    w = (torch.randn(G, N, K, device="cuda") * 0.05 * torch.logspace(-1, 1, N // 128, device="cuda").repeat_interleave(128)[None, :, None]).to(torch.bfloat16)
    wq, ws = M.quantize_weight_fp8(w)
    assert torch.equal(ws, torch.exp2(torch.round(torch.log2(ws))))
    wd = _deq_w(wq, ws)
    ref = torch.cat([xd[off[g]:off[g + 1]] @ wd[g].t() for g in range(G)])
    st = gemm.status_word()
    assert cu.mf_grouped_gemm_fp8_mx_supported(G, N, K, 0) == 1
    out = torch.zeros(R, N, dtype=torch.bfloat16, device="cuda")
    assert cu.mf_grouped_gemm_fp8_mx(xq.data_ptr(), xs.data_ptr(), R, wq.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, out.data_ptr(), N, None, 0,
                                     None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    rowmax = ref.abs().amax(dim=1, keepdim=True)
    assert ((out.float() - ref).abs() <= 2e-2 * rowmax + 1e-5).all(), float(((out.float() - ref).abs() / (rowmax + 1e-9)).max())
    # SwiGLU (bf16 out) and SwiGLU + re-quantisation (fp8 + power-of-two scale per 128 outputs)
    wi = M.interleave_gate_up_fp8(wq, tile=128)
    ref2 = torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:]
    rowmax2 = ref2.abs().amax(dim=1, keepdim=True)
    out2 = torch.zeros(R, N // 2, dtype=torch.bfloat16, device="cuda")
    assert cu.mf_grouped_gemm_fp8_mx(xq.data_ptr(), xs.data_ptr(), R, wi.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, out2.data_ptr(), N // 2, None,
                                     1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    assert ((out2.float() - ref2).abs() <= 3e-2 * rowmax2 + 1e-5).all()
    hq = torch.zeros(R, N // 2, dtype=torch.uint8, device="cuda")
    hs = torch.zeros(R, N // 256, dtype=torch.float32, device="cuda")
    assert cu.mf_grouped_gemm_fp8_mx(xq.data_ptr(), xs.data_ptr(), R, wi.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, hq.data_ptr(), N // 2,
                                     hs.data_ptr(), 3, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    assert torch.equal(hs, torch.exp2(torch.round(torch.log2(hs))))
    hd = _deq(hq.view(torch.float8_e4m3fn), hs)
    # fp8 e4m3 keeps 3 mantissa bits: each value is within 1/16 of itself plus the block's smallest step
    blockmax = ref2.view(R, N // 256, 128).abs().amax(dim=2, keepdim=True).expand(R, N // 256, 128).reshape(R, N // 2)
    assert ((hd - ref2).abs() <= 0.07 * ref2.abs() + 0.02 * blockmax + 1e-6).all()
    # the same bytes as the stand-alone quantiser produces from the bf16 SwiGLU output of the kernel above
    hq2, hs2 = torch.empty_like(hq), torch.empty_like(hs)
    assert cu.mf_quant_rows_fp8(out2.data_ptr(), N // 2, off[G:].data_ptr(), N // 2, hq2.data_ptr(), hs2.data_ptr(), 64, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(hs, hs2) and torch.equal(hq, hq2)


@pytest.mark.parametrize("N,K,counts", [(256, 128, [1]), (256, 640, [31, 0, 32, 33, 223]), (512, 2176, [224, 225, 0, 449]), (256, 2048, [0] * 33 + [65] + [0] * 29 + [3]),
                                        (768, 512, [1000, 1, 448])])
def test_grouped_gemm_fp8_tile_widths(N, K, counts):
    """Row counts around the steps (32) and the largest width (224) of a tile, empty groups, 64 groups, K of one block, of a group of scales
    that is not full (5, 17 blocks) and of whole spans (16): plain and re-quantised results, rows behind the last one untouched, and
    a row of NaN and infinities that changes no other row."""
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    torch.manual_seed(sum(counts) + N + K)
    s = torch.cuda.current_stream().cuda_stream
    G, R, spare = len(counts), sum(counts), 40
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    x = torch.randn(R, K, device="cuda").to(torch.bfloat16)
    xq, xs = torch.zeros(R + spare, K, dtype=torch.uint8, device="cuda"), torch.ones(R + spare, K // 128, device="cuda")
    assert cu.mf_quant_rows_fp8(x.data_ptr(), K, off[G:].data_ptr(), K, xq.data_ptr(), xs.data_ptr(), 64, s) == 0
    w = (torch.randn(G, N, K, device="cuda") * 0.05).to(torch.bfloat16)
    wq, ws = M.quantize_weight_fp8(w)
    xd, wd = _deq(xq[:R].view(torch.float8_e4m3fn), xs[:R]).double(), _deq_w(wq, ws).double()
    ref = torch.cat([xd[off[g]:off[g + 1]] @ wd[g].t() for g in range(G)])
    # one rounding to bf16, and the fp32 accumulation of K terms
    bound = ref.abs() * 2.0 ** -8 + torch.cat([xd[off[g]:off[g + 1]].abs() @ wd[g].abs().t() for g in range(G)]) * K * 2.0 ** -24
    st = gemm.status_word()

    def run(epi, b, ldo, dt, scales=None):
        out = torch.full((R + spare, ldo), 7.0, device="cuda").to(dt)
        assert cu.mf_grouped_gemm_fp8_mx(xq.data_ptr(), xs.data_ptr(), R + spare, b.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, out.data_ptr(), ldo,
                                         scales.data_ptr() if scales is not None else None, epi, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
        torch.cuda.synchronize()
        gemm.check_status()
        assert bool((out[R:] == 7).all())
        return out[:R]

    out = run(0, wq, N, torch.bfloat16)
    assert bool(((out.double() - ref).abs() <= bound).all())
    wi = M.interleave_gate_up_fp8(wq, tile=128)
    h = run(1, wi, N // 2, torch.bfloat16)
    gate, up = ref[:, :N // 2], ref[:, N // 2:]
    want = torch.nn.functional.silu(gate) * up
    # silu' <= 1.1: the accumulation errors of both factors, one rounding to bf16, a few units of fp32 of the exponential and the quotient
    bg, bu = (bound - ref.abs() * 2.0 ** -8).split(N // 2, 1)
    assert bool(((h.double() - want).abs() <= want.abs() * 2.0 ** -7.9 + 1.1 * bg * up.abs() + bu * gate.abs() + 1e-6).all())
    hs, hs2, hq2 = torch.zeros(R + spare, N // 256, device="cuda"), torch.zeros(R, N // 256, device="cuda"), torch.zeros(R, N // 2, dtype=torch.uint8, device="cuda")
    hq = run(3, wi, N // 2, torch.uint8, hs)
    assert cu.mf_quant_rows_fp8(h.data_ptr(), N // 2, off[G:].data_ptr(), N // 2, hq2.data_ptr(), hs2.data_ptr(), 64, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(hq, hq2) and torch.equal(hs[:R], hs2) and bool((hs[R:] == 0).all())
    bad = R // 2
    xq[bad, ::5] = 0x7F  # NaN
    again = run(0, wq, N, torch.bfloat16)
    keep = torch.arange(R, device="cuda") != bad
    assert torch.equal(again[keep], out[keep]) and bool(torch.isnan(again[bad]).all())
    hs3 = torch.zeros_like(hs)
    hq3 = run(3, wi, N // 2, torch.uint8, hs3)
    assert torch.equal(hq3[keep], hq[keep]) and torch.equal(hs3[:R][keep], hs[:R][keep])
    assert bool((hq3[bad] & 0x7F == 0x7F).all()) and bool((hs3[bad] == 1).all())


@pytest.mark.parametrize("sms", [148, 147, 1])
@pytest.mark.parametrize("N,K,counts", [(256, 128, [1]), (256, 640, [31, 0, 32, 33, 223]), (512, 2176, [224, 225, 0, 449]), (256, 384, [0] * 33 + [65] + [0] * 29 + [3])])
def test_grouped_gemm_fp8_push_of_weighted_rows(N, K, counts, sms):
    """The combine epilogue around the steps and the largest width of a tile, with empty groups and with numbers of CTAs that are no whole pairs: every row
    times its weight in its token's slot, no other slot touched, the flag raised by the last CTA and its counter back at zero."""
    import ctypes as C
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    gen = torch.Generator("cuda").manual_seed(sum(counts) + K)
    G, R, spare, topk = len(counts), sum(counts), 40, 3
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    x = torch.randn(R + spare, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    xs = 2.0 ** torch.randint(-4, 1, (R + spare, K // 128), generator=gen, device="cuda").float()
    w = torch.randn(G, N, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    ws = 2.0 ** torch.randint(-7, -3, (G, N // 128, K // 128), generator=gen, device="cuda").float()
    xd, wd = _deq(x[:R], xs[:R]).double(), _deq_w(w, ws).double()
    ref = torch.cat([xd[off[g]:off[g + 1]] @ wd[g].t() for g in range(G)])
    room = torch.cat([xd[off[g]:off[g + 1]].abs() @ wd[g].abs().t() for g in range(G)]) * K * 2.0 ** -24
    weight = torch.rand(R + spare, generator=gen, device="cuda")
    slots = (R + spare + topk - 1) // topk * topk
    place = torch.randperm(slots, generator=gen, device="cuda")[:R + spare]   # slot token * topk + k of every row; the spare rows' slots stay as they are
    info = torch.stack([torch.zeros_like(place), place // topk, place % topk, weight.view(torch.int32).long()], 1).to(torch.int32).contiguous()
    flags_at, comb_at = 256, 4096
    heap = torch.zeros(comb_at + slots * N * 2, dtype=torch.uint8, device="cuda")
    flags, comb = heap[flags_at:flags_at + 4 * 64].view(torch.int32), heap[comb_at:].view(torch.bfloat16).view(slots, N)
    comb.fill_(7)
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    team = M.TeamC(heap.data_ptr(), heap.numel(), 0, 0, 1, 0, 1 << 20)
    st, s = gemm.status_word(), torch.cuda.current_stream().cuda_stream
    for epoch in (5, 6):
        assert cu.mf_grouped_gemm_fp8_mx_signal(x.data_ptr(), xs.data_ptr(), R + spare, w.data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K, None, 0, None, 2,
                                                C.byref(team), info.data_ptr(), comb_at, topk, done.data_ptr(), flags_at, 1, epoch, st.data_ptr(), sms, s) == 0
        torch.cuda.synchronize()
        gemm.check_status()
        assert int(done) == 0 and int(flags[16]) == epoch and int(flags.abs().sum()) == epoch
    want = ref * weight[:R, None].double()
    # the accumulation, the product in fp32, one rounding to bf16
    bound = want.abs() * (2.0 ** -8 + 2.0 ** -23) + room * weight[:R, None]
    assert bool(((comb[place[:R]].double() - want).abs() <= bound).all())
    rest = torch.ones(slots, dtype=torch.bool, device="cuda")
    rest[place[:R]] = False
    assert bool((comb[rest] == 7).all())


def test_swiglu_quotient_of_every_float():
    """The grouped GEMM's own division gives the general division's quotient for all 2^32 gates, bit for bit."""
    import ctypes as C
    from memfabric_hybrid_b200.ops import moe as M
    f = M._cu().mf_swiglu_debug_probe
    f.restype, f.argtypes = C.c_int, [C.c_uint32, C.c_uint64, C.c_void_p, C.c_void_p]
    differ = torch.zeros(1, dtype=torch.int64, device="cuda")
    for part in range(16):
        assert f(part << 28, 1 << 28, differ.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert int(differ) == 0


@pytest.mark.parametrize("gate", ["79", "80", "200", "inf", "nan"])
@pytest.mark.parametrize("sign", [1, -1])
def test_swiglu_of_gates_that_leave_the_fast_divisions_range(gate, sign):
    """One column of gates on either side of the range's end (80), and one row's gate infinite or not a number: the bytes are the other kernel's."""
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    R, N, K = 96, 256, 128
    gen = torch.Generator("cuda").manual_seed(9)
    x, w = torch.zeros(R, K, device="cuda"), torch.zeros(N, K, device="cuda")
    x[:, :2] = 1
    w[:, 0] = torch.randint(-8, 9, (N,), generator=gen, device="cuda").float()
    xs, ws = torch.ones(R, 1, device="cuda"), torch.ones(1, N // 128, 1, device="cuda")
    a, b = {"79": (64, 15), "80": (64, 16), "200": (128, 72), "inf": (448, 0), "nan": (1, 0)}[gate]   # values that e4m3 has
    w[37, 0], w[37, 1] = sign * a, sign * b
    if gate == "inf":
        xs[50] = 2.0 ** 127   # 448 * 2^127 and most other sums of that row leave fp32
    if gate == "nan":
        x[50, 0] = float("nan")
    xq, wq = x.to(torch.float8_e4m3fn), w.to(torch.float8_e4m3fn)[None]
    off = torch.tensor([0, R], dtype=torch.int32, device="cuda")
    st, s = gemm.status_word(), torch.cuda.current_stream().cuda_stream
    got, want = (torch.full((R, N // 2), 7.0, device="cuda").to(torch.bfloat16) for _ in range(2))
    assert cu.mf_grouped_gemm_fp8_mx(xq.data_ptr(), xs.data_ptr(), R, M.interleave_gate_up_fp8(wq, tile=128).data_ptr(), ws.data_ptr(), off.data_ptr(), 1, N, K,
                                     got.data_ptr(), N // 2, None, 1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    assert cu.mf_grouped_gemm_fp8(xq.data_ptr(), xs.data_ptr(), R, M.interleave_gate_up_fp8(wq, tile=64).data_ptr(), ws.data_ptr(), off.data_ptr(), 1, N, K,
                                  want.data_ptr(), N // 2, 1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert gate not in ("inf", "nan") or not bool(torch.isfinite(want[50].float()).all())


@pytest.mark.parametrize("K", [128, 384, 512, 2560])
def test_grouped_gemm_fp8_scales_on_and_off_16_bytes(K):
    """Rows of scales that start on 16 bytes are read four at a time, others one by one: the same bytes, with scales that differ from row to row and
    block to block, in front of a last span of 16 blocks that is not full (2560: 20 blocks)."""
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    G, N, counts = 3, 512, [300, 1, 95]
    R, kb = sum(counts), K // 128
    gen = torch.Generator("cuda").manual_seed(K)
    off = torch.tensor([0, 300, 301, R], dtype=torch.int32, device="cuda")
    x = torch.randint(-8, 9, (R, K), generator=gen, device="cuda").float().to(torch.float8_e4m3fn)
    w = torch.randint(-8, 9, (G, N, K), generator=gen, device="cuda").float().to(torch.float8_e4m3fn)
    xs = 2.0 ** torch.randint(-3, 4, (R, kb), generator=gen, device="cuda").float()
    ws = 2.0 ** torch.randint(-3, 4, (G, N // 128, kb), generator=gen, device="cuda").float()
    ref = torch.cat([_deq(x[off[g]:off[g + 1]], xs[off[g]:off[g + 1]]).double() @ _deq_w(w[g], ws[g]).double().t() for g in range(G)])
    st, s = gemm.status_word(), torch.cuda.current_stream().cuda_stream
    for shift in (0, 1):   # floats by which both arrays of scales are moved off 16 bytes
        xo, wo = (torch.full((t.numel() + 8,), float("nan"), device="cuda")[shift:shift + t.numel()].view(t.shape) for t in (xs, ws))
        xo.copy_(xs)
        wo.copy_(ws)
        out = torch.zeros(R, N, dtype=torch.bfloat16, device="cuda")
        assert cu.mf_grouped_gemm_fp8_mx(x.data_ptr(), xo.data_ptr(), R, w.data_ptr(), wo.data_ptr(), off.data_ptr(), G, N, K, out.data_ptr(), N, None, 0, None,
                                         None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
        torch.cuda.synchronize()
        gemm.check_status()
        # whole numbers times powers of two that span 2^12: 13 + 12 bits, up to one unit of fp32 in the sum, and one rounding to bf16
        assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + ref.abs().max() * 2.0 ** -22).all()), shift


def test_swiglu_of_the_expert_kernels_is_the_same():
    """Small whole numbers: both kernels' sums are exact (14 bits), so that every bf16 activation has to be the same one, and with it
    every byte of a layer that changes its kernel with its shape. 2 M activations: a quotient one unit of fp32 off moves a few dozen."""
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    G, R, N, K = 2, 4096, 1024, 256
    gen = torch.Generator("cuda").manual_seed(5)
    x = torch.randint(-8, 9, (R, K), generator=gen, device="cuda").float().to(torch.float8_e4m3fn)
    w = torch.randint(-8, 9, (G, N, K), generator=gen, device="cuda").float().to(torch.float8_e4m3fn)
    xs, ws = torch.full((R, K // 128), 2.0 ** -3, device="cuda"), torch.full((G, N // 128, K // 128), 2.0 ** -3, device="cuda")
    off = torch.tensor([0, 1500, R], dtype=torch.int32, device="cuda")
    st, s = gemm.status_word(), torch.cuda.current_stream().cuda_stream
    got, want = (torch.zeros(R, N // 2, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert cu.mf_grouped_gemm_fp8_mx(x.data_ptr(), xs.data_ptr(), R, M.interleave_gate_up_fp8(w, tile=128).data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K,
                                     got.data_ptr(), N // 2, None, 1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    assert cu.mf_grouped_gemm_fp8(x.data_ptr(), xs.data_ptr(), R, M.interleave_gate_up_fp8(w, tile=64).data_ptr(), ws.data_ptr(), off.data_ptr(), G, N, K,
                                  want.data_ptr(), N // 2, 1, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    assert int((got != want).sum()) == 0 and float(got.abs().max()) > 100


def _moe_ranks(rank, world, url, T, H, I, E, K, sync):
    import torch
    from memfabric_hybrid_b200.ops import gemm
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    from memfabric_hybrid_b200.models.deepseek_moe import ExpertParallelMoE
    from memfabric_hybrid_b200.ops import moe as M
    dev = rank % torch.cuda.device_count()
    max_recv = T * world * min(K, E // world)
    need = (2 << 20) + max_recv * (H + H // 128 * 4 + 16) + T * K * H * 2 + (4 << 20)
    heap = SymmetricHeap(url, world, rank, dev, need)
    layer = ExpertParallelMoE(heap, H, I, E, K, max_tokens=T, seed=5)
    worst = 0.0
    for it in range(2):
        def inputs(r):
            g = torch.Generator("cuda").manual_seed(97 * it + r)
            return (torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16), torch.randn(T, E, device="cuda", generator=g))
        x, logits = inputs(rank)
        y = layer.forward(x, logits)
        torch.cuda.synchronize()
        gemm.check_status()
        # reference: quantise the token like the dispatch does, run every chosen expert in fp32 on dequantised fp8 weights
        idx, w = layer.route(logits, K)
        xq, xs = torch.empty(T, H, dtype=torch.uint8, device="cuda"), torch.empty(T, H // 128, device="cuda")
        n = torch.tensor([T], dtype=torch.int32, device="cuda")
        M._cu().mf_quant_rows_fp8(x.data_ptr(), H, n.data_ptr(), H, xq.data_ptr(), xs.data_ptr(), 64, torch.cuda.current_stream().cuda_stream)
        xd = (xq.view(torch.float8_e4m3fn).float().view(T, H // 128, 128) * xs[:, :, None]).view(T, H)
        ref = torch.zeros(T, H, device="cuda")
        el = E // world
        for r in range(world):
            w1, w2 = layer.make_weights(r, 5, x.device)
            w1q, w1s = M.quantize_weight_fp8(w1)
            w2q, w2s = M.quantize_weight_fp8(w2)
            w1d = (w1q.float().reshape(el, 2 * I // 128, 128, H // 128, 128) * w1s[:, :, None, :, None]).reshape(el, 2 * I, H)
            w2d = (w2q.float().reshape(el, H // 128, 128, I // 128, 128) * w2s[:, :, None, :, None]).reshape(el, H, I)
            for le in range(el):
                e = r * el + le
                tk = (idx == e).nonzero()
                if tk.numel() == 0:
                    continue
                rows = xd[tk[:, 0]]
                gu = rows @ w1d[le].t()
                h = (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]).to(torch.bfloat16)
                hq, hs = torch.empty(h.shape[0], I, dtype=torch.uint8, device="cuda"), torch.empty(h.shape[0], I // 128, device="cuda")
                nn_ = torch.tensor([h.shape[0]], dtype=torch.int32, device="cuda")
                M._cu().mf_quant_rows_fp8(h.data_ptr(), I, nn_.data_ptr(), I, hq.data_ptr(), hs.data_ptr(), 64,
                                          torch.cuda.current_stream().cuda_stream)
                hd = (hq.view(torch.float8_e4m3fn).float().view(-1, I // 128, 128) * hs[:, :, None]).view(-1, I)
                yrows = (hd @ w2d[le].t()) * w[tk[:, 0], tk[:, 1]][:, None]
                ref.index_add_(0, tk[:, 0], yrows.to(torch.bfloat16).float())
        err = (y.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-9)
        worst = max(worst, err)
    st = heap.status()[0]
    heap.close()
    SymmetricHeap.shutdown()
    return worst, st


def test_moe_layer_world1():
    url = f"127.0.0.1:{free_port()}"
    (worst, st), = run_ranks(_moe_ranks, 1, (url, 256, 512, 256, 8, 4), timeout=300, with_barrier=True)
    assert st == 0 and worst < 4e-2, (worst, st)


@pytest.mark.multigpu
def test_moe_layer_multi_gpu():
    n = 2 if torch.cuda.device_count() < 4 else 4
    url = f"127.0.0.1:{free_port()}"
    res = run_ranks(_moe_ranks, n, (url, 256, 512, 256, 16, 4), timeout=300, with_barrier=True)
    for worst, st in res:
        assert st == 0 and worst < 4e-2, res


def _canary_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import gemm
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    from memfabric_hybrid_b200.models.deepseek_moe import ExpertParallelMoE
    T, H, I, E, K = 128, 512, 256, 8, 4
    heap = SymmetricHeap(url, 1, 0, 0, (2 << 20) + T * K * (H + H // 128 * 4 + 16) + T * K * H * 2 + (4 << 20))
    layer = ExpertParallelMoE(heap, H, I, E, K, max_tokens=T, seed=5)
    assert len(layer.comm._guards) == 5
    g = torch.Generator("cuda").manual_seed(1)
    x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    logits = torch.randn(T, E, device="cuda", generator=g)
    layer.forward(x, logits)            # checks the guards at the end of combine
    layer.forward(x, logits)
    gemm.check_status()
    # a store that runs past the token rows lands in the guard behind them
    heap.view(layer.comm._guards[1], (4,), torch.int32)[2] = 7
    try:
        layer.comm.check_canaries()
        caught = False
    except RuntimeError as e:
        caught = "guard 1" in str(e)
    heap.close()
    SymmetricHeap.shutdown()
    return caught


def test_moe_receive_areas_are_guarded_by_canaries():
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_canary_rank, 1, (url,), timeout=300, with_barrier=True, env={"MF_MOE_CANARY": "1"}) == [True]


def _prepare_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import gemm, moe as M
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    H, E, K, Tmax = 512, 48, 4, 1300
    heap = SymmetricHeap(url, 1, 0, 0, (2 << 20) + Tmax * K * (H + H // 128 * 4 + 16) + Tmax * K * H * 2 + (4 << 20))
    comm = M.MoEComm(heap, Tmax, H, E, K, max_recv=Tmax * K)
    bad = []
    for T in (1, 7, 255, 256, 257, 1023, 1024, 1025, 1300):   # 4096 entries is where the one-launch layout ends
        g = torch.Generator("cuda").manual_seed(T)
        x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
        idx = torch.rand(T, E, device="cuda", generator=g).topk(K, dim=-1).indices.to(torch.int32)
        idx[torch.rand(T, K, device="cuda", generator=g) < 0.1] = -1    # unselected slots
        w = torch.rand(T, K, device="cuda", generator=g)
        st = comm.dispatch(x, idx, w)
        torch.cuda.synchronize()
        gemm.check_status()
        flat = idx.view(-1).cpu().long()
        on = flat >= 0
        counts = torch.bincount(flat[on], minlength=E)
        pos = torch.zeros_like(flat)
        seen = [0] * E
        for i, e in enumerate(flat.tolist()):
            if e >= 0:
                pos[i] = seen[e]
                seen[e] += 1
        first = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
        ok = torch.equal(st.tokens_per_expert.cpu().long(), counts) and torch.equal(st.row_off.cpu().long(), first)
        ok = ok and torch.equal(st.recv_per_expert.cpu().long(), counts) and torch.equal(st.put_off.cpu().long(), first[:-1])
        ok = ok and torch.equal(st.src_off.cpu().long(), first[:-1])
        ok = ok and torch.equal(st.send_idx.cpu().long()[on], pos[on]) and bool((st.send_idx.cpu()[~on] == 0).all())
        any_on = (idx >= 0).any(1)
        ok = ok and int(st.tokens_per_rank[0]) == int(any_on.sum()) and torch.equal(st.is_token_in_rank[:, 0].bool(), any_on)
        # every row where the tables say, with its token's values, scales and origin
        rows = (first[flat[on]] + pos[on]).cuda()
        tok = torch.arange(T).repeat_interleave(K)[on].cuda()
        got = (comm.recv_x()[rows].float().view(-1, H // 128, 128) * comm.recv_scale()[rows][:, :, None]).view(-1, H)
        want = x[tok].float()
        block = want.view(-1, H // 128, 128).abs().amax(2, keepdim=True).expand(-1, -1, 128).reshape(-1, H)
        ok = ok and bool(((got - want).abs() <= want.abs() / 16 + block / 448).all())   # e4m3: half a step of 2^-3, 2^-9 at the bottom
        info = comm.recv_info()[rows]
        ok = ok and torch.equal(info[:, 1].long(), tok) and torch.equal(info[:, 3].contiguous().view(torch.float32), w.view(-1)[on.cuda()])
        comm.combine_push(torch.zeros(int(first[-1]), H, dtype=torch.bfloat16, device="cuda"), st)
        comm.combine(st)
        if not ok:
            bad.append(T)
    heap.close()
    SymmetricHeap.shutdown()
    return bad


def test_dispatch_tables_and_rows_around_the_one_launch_layout():
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_prepare_rank, 1, (url,), timeout=300, with_barrier=True) == [[]]


def _absent_peer_team(spin_limit):
    """Rank 0 of a group of two whose other rank never arrives: both slots are on this GPU, nothing else runs in them."""
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    heap = EmulatedHeap(2, 8 << 20)
    team = heap.team()
    team.emu, team.spin_limit = 0, spin_limit
    hp = M.MoeHeapC()
    hp.counts, hp.flags = heap.alloc(2 * 8 * 4), heap.alloc(4 * 16 * 4)
    hp.recv_x, hp.recv_scale, hp.recv_info, hp.comb = heap.alloc(1 << 20), heap.alloc(1 << 18), heap.alloc(1 << 18), heap.alloc(1 << 20)
    return heap, team, hp


@pytest.mark.parametrize("waiter", ["wait_all", "prepare"])
def test_a_wait_for_peers_leaves_the_sms_to_other_streams(waiter):
    """One rank polls for a peer that never comes, with a GEMM that fills every SM queued behind the poll. A collective on
    another stream (all ranks of its group in one cooperative launch over nearly every SM) must run meanwhile: on several GPUs it
    may be what the peer is waiting in. The poll ends by its own limit and says so."""
    import ctypes as C
    from memfabric_hybrid_b200.ops import gemm, moe as M
    from memfabric_hybrid_b200.ops.collectives import Communicator
    from memfabric_hybrid_b200.ops.heap import EmulatedHeap
    cu = M._cu()
    heap, team, hp = _absent_peer_team(1 << 20)   # a few tenths of a second
    i32 = dict(dtype=torch.int32, device="cuda")
    st = torch.zeros(1, **i32)
    T, K, E, G, N, H = 4, 2, 8, 2, 256, 256
    idx = torch.zeros(T, K, **i32)
    out = {n: torch.zeros(64, **i32) for n in ("tpe", "tpr", "sidx", "rpe", "row_off", "put_off", "src_off")}
    inr = torch.zeros(T, 2, dtype=torch.uint8, device="cuda")
    a, b = torch.zeros(128, H, dtype=torch.uint8, device="cuda"), torch.zeros(G, N, H, dtype=torch.uint8, device="cuda")
    sa, sb = torch.ones(128, H // 128, device="cuda"), torch.ones(G, N // 128, H // 128, device="cuda")
    rows, c = torch.tensor([0, 64, 128], **i32), torch.empty(128, N, dtype=torch.bfloat16, device="cuda")

    def poll(epoch, t, s):
        if waiter == "wait_all":
            assert cu.mf_moe_wait_all(C.byref(t), C.byref(hp), 0, epoch, st.data_ptr(), s) == 0
        else:
            assert cu.mf_moe_prepare(C.byref(t), C.byref(hp), idx.data_ptr(), T, K, E, out["tpe"].data_ptr(), out["tpr"].data_ptr(),
                                     out["sidx"].data_ptr(), inr.data_ptr(), out["rpe"].data_ptr(), out["row_off"].data_ptr(),
                                     out["put_off"].data_ptr(), out["src_off"].data_ptr(), epoch, s) == 0
        assert cu.mf_grouped_gemm_fp8_mx(a.data_ptr(), sa.data_ptr(), 128, b.data_ptr(), sb.data_ptr(), rows.data_ptr(), G, N, H, c.data_ptr(), N,
                                         None, 0, None, None, 0, 1, st.data_ptr(), gemm.sm_count(), s) == 0

    x = torch.ones(8, 4 << 20, device="cuda")
    comm = Communicator(EmulatedHeap(8, (4 * 16 << 20) + (2 << 20)), stage_bytes=16 << 20)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    # everything once before: modules loaded, buffers made, the flags' epoch 0 there from the start
    alone = M.TeamC.from_buffer_copy(team)
    alone.world = 1
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        poll(0, alone, s1.cuda_stream)
    with torch.cuda.stream(s2):
        comm.all_reduce(x, out=y)
    torch.cuda.synchronize()
    y.zero_()
    torch.cuda.synchronize()
    polled, reduced = torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(s1):
        poll(5, team, s1.cuda_stream)
        polled.record()
    with torch.cuda.stream(s2):
        comm.all_reduce(x, out=y)
        reduced.record()
    reduced.synchronize()
    still_polling = not polled.query()
    torch.cuda.synchronize()
    assert still_polling, "the collective waited for the poll"
    code, where, epoch, _ = heap.status()
    assert (code, where, epoch) == (1, 0x410 if waiter == "wait_all" else 0x1008, 5)
    assert int(st.item()) == (0x410 if waiter == "wait_all" else 0)
    assert bool((y == 8.0).all()) and comm.heap.status()[0] == 0


@pytest.mark.parametrize("raw_bf16", [0, 1], ids=["warp_per_token", "cta_per_token"])
@pytest.mark.parametrize("how", ["prepare", "notify", "low_latency"])
def test_a_count_exchange_that_times_out_sends_and_receives_nothing(how, raw_bf16):
    """The peer never comes: the exchange gives up, says so, and leaves tables by which the push stores no row anywhere and
    the receiver sees none. (The tables' memory is garbage before the call.)"""
    import ctypes as C
    from memfabric_hybrid_b200.ops import gemm, moe as M
    cu = M._cu()
    heap, team, hp = _absent_peer_team(20_000)   # a few milliseconds
    T, K, E, H = 5, 2, 8, 512
    s = torch.cuda.current_stream().cuda_stream
    bad = lambda n: torch.full((n,), 0x3FFFFFFF, dtype=torch.int32, device="cuda")   # noqa: E731
    tpe, tpr, sidx, rpe, row_off, put_off, src_off = bad(E), bad(2), bad(T * K), bad(E // 2), bad(E // 2 + 1), bad(E), bad(E)
    inr = torch.zeros(T, 2, dtype=torch.uint8, device="cuda")
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    idx = torch.arange(T * K, dtype=torch.int32, device="cuda").view(T, K) % E
    w = torch.ones(T, K, device="cuda")
    st, done, epoch_dev = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(3))
    data = heap._buf.view(2, -1)[:, hp.recv_x:]   # everything behind the flags, in both slots
    data.fill_(0x5A)
    a = M.DispatchArgsC(team, hp, M.MoeShapeC(T, K, E, H, 1 << 30), x.data_ptr(), idx.data_ptr(), w.data_ptr(), sidx.data_ptr(), put_off.data_ptr(),
                        done.data_ptr(), 1, 0 if how == "low_latency" else 1, st.data_ptr(), raw_bf16, None)
    if how == "low_latency":
        assert cu.mf_moe_ll_dispatch(C.byref(a), tpe.data_ptr(), rpe.data_ptr(), row_off.data_ptr(), src_off.data_ptr(), epoch_dev.data_ptr(), 4, s) == 0
    else:
        if how == "prepare":
            assert cu.mf_moe_prepare(C.byref(team), C.byref(hp), idx.data_ptr(), T, K, E, tpe.data_ptr(), tpr.data_ptr(), sidx.data_ptr(),
                                     inr.data_ptr(), rpe.data_ptr(), row_off.data_ptr(), put_off.data_ptr(), src_off.data_ptr(), 1, s) == 0
        else:
            assert cu.mf_moe_layout(idx.data_ptr(), T, K, E, 2, tpe.data_ptr(), tpr.data_ptr(), sidx.data_ptr(), inr.data_ptr(), s) == 0
            assert cu.mf_moe_notify(C.byref(team), C.byref(hp), E, tpe.data_ptr(), rpe.data_ptr(), row_off.data_ptr(), put_off.data_ptr(),
                                    src_off.data_ptr(), 1, s) == 0
        assert cu.mf_moe_dispatch(C.byref(a), gemm.sm_count(), s) == 0
    torch.cuda.synchronize()
    assert heap.status()[0] == 1 and heap.status()[1] == (0x1009 if how == "low_latency" else 0x1008)
    assert int(st.item()) == (0x420 if how == "low_latency" else 0)
    assert not row_off.any() and not rpe.any() and not src_off.any() and bool((put_off == -1).all())
    assert bool((data == 0x5A).all()), "a row was stored"


def _ll_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.gemm import check_status
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    bad = []
    heap = SymmetricHeap(url, 1, 0, 0, 256 << 20)
    # (hidden, experts, copies, tokens): a token per CTA, up to four, and more (the kernel with a grid-wide barrier); entries that nobody selected
    for H, E, K, sizes in ((512, 8, 2, (1, 3)), (7168, 32, 8, (1, 147, 149, 256)), (1152, 40, 5, (1, 7, 593, 600)), (640, 1024, 16, (2, 256, 257))):
        mark = heap.mark()
        comm = M.MoEComm(heap, max(sizes), H, E, K, max_recv=max(sizes) * K)
        for T in sizes:
            g = torch.Generator("cuda").manual_seed(T + H)
            x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
            idx = torch.stack([torch.randperm(E, device="cuda", generator=g)[:K] for _ in range(T)]).to(torch.int32)
            if T > 2:
                idx[1] = -1
                idx[2, 0] = -1
            w = torch.rand(T, K, device="cuda", generator=g)
            for _ in range(2):   # the counter of calls moves on
                d = comm.ll_dispatch(x, idx, w)
                rows = int(d.row_off[-1])
                q, s = comm.recv_x()[:rows].float(), comm.recv_scale()[:rows]
                y = (q.view(rows, -1, 128) * s[:, :, None]).view(rows, H).to(torch.bfloat16)
                info = comm.recv_info()[:rows].cpu()
                out = comm.ll_combine(y, d)
                torch.cuda.synchronize()
                check_status()
                flat = idx.cpu().view(-1)
                counts = torch.bincount(flat[flat >= 0].long(), minlength=E)
                off = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
                ok = torch.equal(d.row_off.cpu().long(), off) and torch.equal(d.recv_per_expert.cpu().long(), counts) and torch.equal(d.tokens_per_expert.cpu().long(), counts)
                ok = ok and torch.equal(d.put_off.cpu().long(), off[:-1]) and torch.equal(d.src_off.cpu().long(), off[:-1])
                # every selected entry once, in its expert's group, where send_idx says
                entry = info[:, 1].long() * K + info[:, 2].long()
                ok = ok and torch.equal(entry.sort().values, (flat >= 0).nonzero().view(-1))
                ok = ok and torch.equal(off[flat[entry].long()] + d.send_idx.cpu().long()[entry], torch.arange(rows))
                ok = ok and torch.equal(info[:, 3].view(torch.float32), w.cpu().view(-1)[entry])
                # a row is its token quantised; the sum of the weighted answers in bf16 steps
                xq = y.cpu()
                for a in {0, rows // 2, rows - 1} if rows else ():
                    t = x[int(info[a, 1])].cpu().float()
                    ok = ok and bool(((xq[a].float() - t).abs() <= t.abs() * 2.0 ** -4 + t.view(-1, 128).abs().amax(1).repeat_interleave(128) * 2.0 ** -9).all())
                ref = torch.zeros(T, H)
                ref.index_add_(0, info[:, 1].long(), (xq.float() * w.cpu().view(-1)[entry][:, None]).to(torch.bfloat16).float())
                got = out.cpu().float()
                ok = ok and bool(((got - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all())
                if not ok:
                    bad.append((H, E, K, T))
        heap.release_to(mark)
    st = heap.status()[0]
    heap.close()
    SymmetricHeap.shutdown()
    return bad, st


def test_low_latency_pair_around_its_tokens_per_cta():
    url = f"127.0.0.1:{free_port()}"
    (bad, st), = run_ranks(_ll_rank, 1, (url,), timeout=300, with_barrier=True)
    assert not bad and st == 0, (bad, st)


@pytest.mark.parametrize("T,K", [(1, 1), (127, 16), (341, 3), (1025, 1), (4099, 8)])
@pytest.mark.parametrize("world,E", [(1, 32), (3, 96), (8, 1024), (16, 64)])
def test_layout_of_tokens_cut_over_ctas(T, K, world, E):
    """Positions in token order, counts per expert and per rank, and each token's ranks, whatever the outputs held before; ids outside of [0, E) count nowhere."""
    from memfabric_hybrid_b200.ops import moe as M
    g = torch.Generator().manual_seed(T + K)
    idx = torch.randint(-3, E + 3, (T, K), generator=g, dtype=torch.int32)
    tpe, tpr, sidx = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (E, world, T * K))
    inr = torch.full((T, world), 9, dtype=torch.uint8, device="cuda")
    d = idx.cuda()
    for _ in range(2):
        assert M._cu().mf_moe_layout(d.data_ptr(), T, K, E, world, tpe.data_ptr(), tpr.data_ptr(), sidx.data_ptr(), inr.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream) == 0
    flat = idx.view(-1).long()
    on = (flat >= 0) & (flat < E)
    hot = torch.nn.functional.one_hot(torch.where(on, flat, E), E + 1)[:, :E]
    before = (hot.cumsum(0) - hot)
    assert torch.equal(tpe.cpu().long(), hot.sum(0))
    assert torch.equal(sidx.cpu().long(), torch.where(on, before.gather(1, flat.clamp(0, E - 1)[:, None])[:, 0], 0))
    ranks = hot.view(T, K, world, E // world).sum((1, 3)) > 0
    assert torch.equal(inr.cpu().bool(), ranks) and int(inr.max()) <= 1
    assert torch.equal(tpr.cpu().long(), ranks.sum(0))


def _mixed_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.gemm import status_word
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    H, E, K = 512, 8, 8
    heap = SymmetricHeap(url, 1, 0, 0, 64 << 20)
    comm = M.MoEComm(heap, 700, H, E, K, max_recv=700 * K)
    g = torch.Generator("cuda").manual_seed(3)
    fine = []
    for step, T in enumerate((4, 4, 700, 64, 700, 1, 1)):
        x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
        w = torch.rand(T, K, device="cuda", generator=g)
        if step in (1, 6):
            st = comm.dispatch_cached(x, st, w)
        else:
            st = comm.dispatch(x, torch.rand(T, E, device="cuda", generator=g).argsort(1).to(torch.int32), w)
        comm.combine_push(torch.ones(T * K, H, dtype=torch.bfloat16, device="cuda"), st)
        want = w.to(torch.bfloat16).float().sum(1, keepdim=True).expand(T, H)   # of rows that were rounded to bf16 when they were pushed
        fine.append(bool(((comm.combine(st).float() - want).abs() <= want * 2.0 ** -8).all()) and int(st.row_off[-1]) == T * K)
    fine.append(int(status_word("cuda").item()) == 0 and heap.status()[0] == 0)
    heap.close()
    SymmetricHeap.shutdown()
    return fine


def test_dispatch_kernels_that_count_and_do_not_count_their_ctas_take_turns():
    """One rank's few tokens leave the counter of finished CTAs and the flag alone; calls of the kernels that use both follow in any order."""
    url = f"127.0.0.1:{free_port()}"
    (fine,) = run_ranks(_mixed_rank, 1, (url,), timeout=300, with_barrier=True)
    assert all(fine), fine


def _raw_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.gemm import check_status
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    heap, E, K, bad = SymmetricHeap(url, 1, 0, 0, 256 << 20), 16, 4, []
    for H in (128, 1152, 7168):
        mark = heap.mark()
        comm = M.MoEComm(heap, 1100, H, E, K, max_recv=1100 * K, raw_bf16=True)
        for T in (1, 3, 149, 593, 1100):    # one launch of few tokens, the small exchange, launches of their own
            x = torch.randn(T, H, device="cuda", generator=torch.Generator("cuda").manual_seed(T)).to(torch.bfloat16)
            idx = torch.rand(T, E, device="cuda").topk(K, 1).indices.to(torch.int32)
            idx[T // 2, 1] = -1
            for how in ("dispatch", "cached", "low latency"):
                comm.recv_x().fill_(7.0)
                if how == "cached":
                    st = comm.dispatch_cached(x, st, torch.rand(T, K, device="cuda"))
                else:
                    st = (comm.dispatch if how == "dispatch" else comm.ll_dispatch)(x, idx, torch.rand(T, K, device="cuda"))
                rows = int(st.row_off[-1])
                got, tok = comm.recv_x(), comm.recv_info()[:rows, 1].long()
                if rows != T * K - 1 or not torch.equal(got[:rows], x[tok]) or not bool((got[rows:] == 7.0).all()):
                    bad.append((H, T, how))
                if how == "low latency":
                    comm.ll_combine(got[:rows].clone(), st)   # the pair: the next call counts on it
        heap.release_to(mark)
    torch.cuda.synchronize()
    check_status()
    ok = heap.status()[0] == 0
    heap.close()
    SymmetricHeap.shutdown()
    return bad, ok


def test_rows_that_travel_as_bf16():
    """Every row whole, where the tables say, and nothing behind the last one."""
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_raw_rank, 1, (url,), timeout=300, with_barrier=True) == [([], True)]


def _overfull_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.gemm import status_word
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    H, E, K, T, room = 512, 8, 2, 32, 40
    heap = SymmetricHeap(url, 1, 0, 0, 16 << 20)
    comm = M.MoEComm(heap, T, H, E, K, max_recv=room)
    idx = torch.stack([torch.randperm(E - 1, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).to(torch.int32)
    idx[0, 0] = E - 1   # the last row of all: dropped
    order = idx.view(-1).argsort(stable=True)
    kept = torch.zeros(T * K)
    kept[order[:room]] = 1
    want = kept.view(T, K).sum(1, keepdim=True).expand(T, H)
    x, w, d = torch.ones(T, H, dtype=torch.bfloat16, device="cuda"), torch.ones(T, K, device="cuda"), idx.cuda()
    y = torch.full((T * K, H), float("nan"), dtype=torch.bfloat16, device="cuda")   # what lies behind the caller's `room` rows
    y[:room] = 1
    right = []
    for pair in ("normal", "low latency"):
        heap.view(comm.hp.recv_info, (comm.hp.comb - comm.hp.recv_info + T * K * H * 2,), torch.uint8).zero_()
        if pair == "normal":
            st = comm.dispatch(x, d, w)
            comm.combine_push(y[:room], st)
            out = comm.combine(st)
        else:
            st = comm.ll_dispatch(x, d, w)
            out = comm.ll_combine(y[:room], st)
        right.append(torch.equal(out.float().cpu(), want) and int(st.row_off[-1]) == T * K and int(status_word(comm.dev).item()) == 0x401)
        status_word(comm.dev).zero_()
    torch.cuda.synchronize()
    right.append(heap.status()[0] == 0)
    heap.close()
    SymmetricHeap.shutdown()
    return right


def test_combine_of_a_receive_buffer_that_was_too_small():
    """Rows without room are dropped and reported; the rows of the answers end where the receive buffer ends, and nothing behind them is read or sent."""
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_overfull_rank, 1, (url,), timeout=300, with_barrier=True) == [[True, True, True]]


def _overfull_ffn_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.gemm import status_word
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    H, I, E, K, T, room = 640, 256, 8, 2, 32, 40   # 640 columns: the kernels with a re-quantisation pass of its own
    heap = SymmetricHeap(url, 1, 0, 0, 16 << 20)
    comm = M.MoEComm(heap, T, H, E, K, max_recv=room)
    q, s = torch.full((T * K, I), 0x5A, dtype=torch.uint8, device="cuda"), torch.full((T * K, I // 128), 7.0, device="cuda")
    comm._hq, comm._hs = q[:room], s[:room]
    w1, w2 = torch.zeros(E, 2 * I, H, dtype=torch.uint8, device="cuda"), torch.zeros(E, H, I, dtype=torch.uint8, device="cuda")
    idx = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).to(torch.int32).cuda()
    heap.view(comm.hp.comb, (T * K * H * 2,), torch.uint8).zero_()
    st = comm.dispatch(torch.ones(T, H, dtype=torch.bfloat16, device="cuda"), idx, torch.ones(T, K, device="cuda"))
    comm.expert_ffn(st, w1, torch.ones(E, 2 * I // 128, H // 128, device="cuda"), w2, torch.ones(E, H // 128, I // 128, device="cuda"))
    y = comm.combine(st)
    torch.cuda.synchronize()
    ok = int(status_word(comm.dev).item()) == 0x401 and int(st.row_off[-1]) == T * K
    ok = ok and bool((q[room:] == 0x5A).all()) and bool((s[room:] == 7.0).all()) and not bool(q[:room].any()) and not bool(y.any())
    status_word(comm.dev).zero_()
    ok = ok and heap.status()[0] == 0
    heap.close()
    SymmetricHeap.shutdown()
    return ok


def test_expert_ffn_of_a_receive_buffer_that_was_too_small():
    """The activations are quantised up to the last row of the buffers, whatever the dispatch has counted."""
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_overfull_ffn_rank, 1, (url,), timeout=300, with_barrier=True) == [True]


def _refused_rank(rank, world, url, sync):
    import torch
    from memfabric_hybrid_b200.ops import moe as M
    from memfabric_hybrid_b200.ops.heap import SymmetricHeap
    H, E, K, many = 512, 8, 2, 2100   # more than 4096 entries: layout and count exchange have launches of their own
    heap = SymmetricHeap(url, 1, 0, 0, 32 << 20)
    comm = M.MoEComm(heap, 4096, H, E, K, max_recv=many * K)
    x, idx, w = torch.randn(many, H, device="cuda").to(torch.bfloat16), torch.zeros(many, K, dtype=torch.int32, device="cuda"), torch.ones(many, K, device="cuda")
    idx[:, 1] = 5
    lib = M._cu()

    class Refusing:
        """The library, with some calls answered on the host."""
        answers = {}

        def __getattr__(self, name):
            return (lambda *a: self.answers[name]) if name in self.answers else getattr(lib, name)

    fake = Refusing()
    M._cu = lambda: fake
    numbers = []
    for t, answers in ((4, {}), (0, {}), (4, {}), (many, {}), (many, {"mf_moe_layout": -1}), (many, {"mf_moe_notify": -1}), (many, {}),
                       (4, {"mf_moe_dispatch_alone": -3, "mf_moe_prepare": -1}), (4, {"mf_moe_dispatch_alone": -3}), (many, {"mf_moe_dispatch": -1}), (many, {}),
                       (4, {"mf_moe_dispatch_alone": -1}), (4, {})):
        fake.answers = answers
        try:
            st = comm.dispatch(x[:t], idx[:t], w[:t])
            comm.combine_push(torch.ones(t * K, H, dtype=torch.bfloat16, device="cuda"), st)
            y = comm.combine(st)
            numbers.append((comm._epoch, comm._counted, bool((y == 2).all())))
        except RuntimeError:
            numbers.append((comm._epoch, comm._counted, None))
    torch.cuda.synchronize()
    st = heap.status()[0]
    heap.close()
    SymmetricHeap.shutdown()
    return numbers, st


def test_a_refused_dispatch_leaves_the_ranks_in_step():
    """Refused by the library (no tokens), or any of the calls of a dispatch by a stand-in for it. The call numbers that the ranks' flags carry must not advance on
    the rank that was refused, or its next call waits for a number that no peer sends; nor may the number that the counter of finished CTAs is
    compared with. An exchange that was launched counts, even if the push behind it was refused."""
    url = f"127.0.0.1:{free_port()}"
    assert run_ranks(_refused_rank, 1, (url,), timeout=300, with_barrier=True) == [
        ([(1, 0, True), (1, 0, None), (2, 0, True), (3, 1, True), (3, 1, None), (3, 1, None), (4, 2, True), (4, 2, None), (5, 3, True), (6, 3, None), (7, 4, True),
          (7, 4, None), (8, 4, True)], 0)]
