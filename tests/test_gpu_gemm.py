"""tcgen05/TMEM GEMM kernels against fp32 PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 256), (256, 512, 512), (200, 320, 1024), (1024, 1024, 4096),
                                   (8, 264, 72), (4096, 7168, 2048)])
@pytest.mark.parametrize("pair", [False, True], ids=["one_cta", "cta_pair"])
def test_gemm_bf16(M, N, K, pair):
    from memfabric_hybrid_b200.ops import gemm
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    c = gemm.gemm_bf16(a, b, pair=pair)
    torch.cuda.synchronize()
    gemm.check_status()
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, f"max abs err {err} vs scale {scale}"


@pytest.mark.parametrize("pair", [False, True], ids=["one_cta", "cta_pair"])
@pytest.mark.parametrize("M,F,K", [(256, 256, 512), (1000, 1024, 2048)])
def test_gemm_bf16_swiglu_epilogue(M, F, K, pair):
    """gate / up weights interleaved per 128 rows; the epilogue writes silu(gate) * up."""
    from memfabric_hybrid_b200.ops import gemm
    torch.manual_seed(M + F + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    wg = (torch.randn(F, K, device="cuda") * 0.05).to(torch.bfloat16)
    wu = (torch.randn(F, K, device="cuda") * 0.05).to(torch.bfloat16)
    c = gemm.gemm_bf16(a, gemm.interleave_gate_up(wg, wu), swiglu=True, pair=pair)
    torch.cuda.synchronize()
    gemm.check_status()
    assert c.shape == (M, F)
    ref = torch.nn.functional.silu(a.float() @ wg.float().t()) * (a.float() @ wu.float().t())
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, f"max abs err {err} vs scale {scale}"


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (8, 136, 72), (33, 520, 200), (64, 7168, 2048), (127, 1000, 512), (129, 256, 1024), (260, 384, 4096)])
@pytest.mark.parametrize("split", [0, 1, 2, 5, 8])
def test_gemm_bf16_split_over_a_cluster(M, N, K, split):
    """Few rows: K split over the CTAs of a cluster, the partial tiles added through distributed shared memory. The result
    is one bf16 rounding away from the exact product (2^-9 of the value) plus fp32 accumulation (K 2^-24 of the terms)."""
    from memfabric_hybrid_b200.ops import gemm
    if split > (K + 63) // 64:
        pytest.skip("more CTAs than steps of K")
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    ld = N + (8 if split % 2 else 3)   # rows of C that 16-byte stores reach, and rows that they do not
    c = torch.full((M, ld), 7.0, device="cuda", dtype=torch.bfloat16)
    assert gemm._cu().mf_gemm_bf16_splitk(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, K, K, ld, gemm.status_word().data_ptr(), gemm.sm_count(), 0, split,
                                          torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    gemm.check_status()
    ref = a.double() @ b.double().t()
    bound = ref.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * K * 2.0 ** -24
    assert ((c[:, :N].double() - ref).abs() <= bound).all()
    assert bool((c[:, N:] == 7.0).all()), "columns past N were written"


@pytest.mark.parametrize("M,F,K", [(1, 128, 128), (32, 3584, 8192), (130, 256, 512)])
def test_gemm_bf16_swiglu_few_rows(M, F, K):
    """The library's own choice for few rows, next to the one-CTA kernel on the same operands."""
    from memfabric_hybrid_b200.ops import gemm
    torch.manual_seed(M + F + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * 0.05).to(torch.bfloat16)
    c = gemm.gemm_bf16(a, w, swiglu=True)
    one = gemm.gemm_bf16(a, w, swiglu=True, pair=False)
    torch.cuda.synchronize()
    gemm.check_status()
    # both round the same fp32 value once; the sums differ by K 2^-24 of their terms, which SwiGLU scales by about |up|
    assert ((c.float() - one.float()).norm() / one.float().norm()).item() <= 2.0 ** -8


@pytest.mark.parametrize("M,N,K", [(1, 256, 512), (31, 512, 576), (129, 256, 2048)])
@pytest.mark.parametrize("split", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("swiglu", [0, 1])
def test_partial_tiles_added_by_any_number_of_ctas(M, N, K, split, swiglu):
    """Items of four columns, several of them at once for 1, 2 and 4 CTAs, rows of C at 2, 4, 8 and 16 bytes. One bf16 rounding (2^-8 of the value) plus fp32 accumulation
    (K 2^-24 of the terms), which SwiGLU scales by |up| times the slope of silu (at most 1.1) and by |silu|; its exponential and quotient stay below 2^-16."""
    from memfabric_hybrid_b200.ops import gemm
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    n_out = N // 2 if swiglu else N
    ref, err = a.double() @ b.double().t(), (a.double().abs() @ b.double().abs().t()) * K * 2.0 ** -24
    if swiglu:
        (g, u), (eg, eu) = (t.view(M, N // 256, 2, 128).permute(2, 0, 1, 3).reshape(2, M, n_out) for t in (ref, err))
        ref = torch.nn.functional.silu(g) * u
        err = 1.1 * eg * u.abs() + torch.nn.functional.silu(g).abs() * eu + ref.abs() * 2.0 ** -16
    for ld, off in ((n_out + 8, 0), (n_out + 4, 4), (n_out + 2, 2), (n_out + 1, 1)):
        buf = torch.full((off + M * ld,), 7.0, device="cuda", dtype=torch.bfloat16)
        c = buf[off:].view(M, ld)
        assert gemm._cu().mf_gemm_bf16_splitk(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, K, K, ld, gemm.status_word().data_ptr(), gemm.sm_count(), swiglu,
                                              split, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        gemm.check_status()
        assert ((c[:, :n_out].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + err).all(), ld
        assert bool((c[:, n_out:] == 7.0).all()) and bool((buf[:off] == 7.0).all()), "columns past N were written"


@pytest.mark.parametrize("M", [32, 4096])
def test_gemm_bf16_in_a_cuda_graph(M):
    """Two products in a row, captured: the second may start under the end of the first (few rows) and must still see all of it."""
    from memfabric_hybrid_b200.ops import gemm
    torch.manual_seed(M)
    a = torch.randn(M, 2048, device="cuda").to(torch.bfloat16)
    w1 = (torch.randn(4096, 2048, device="cuda") * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(2048, 4096, device="cuda") * 0.05).to(torch.bfloat16)
    h, y = torch.empty(M, 4096, device="cuda", dtype=torch.bfloat16), torch.empty(M, 2048, device="cuda", dtype=torch.bfloat16)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        gemm.gemm_bf16(gemm.gemm_bf16(a, w1, out=h), w2, out=y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        gemm.gemm_bf16(gemm.gemm_bf16(a, w1, out=h), w2, out=y)
    for i in range(3):
        a.copy_(torch.randn(M, 2048, device="cuda").to(torch.bfloat16))
        g.replay()
        torch.cuda.synchronize()
        gemm.check_status()
        ref = h.float() @ w2.float().t()
        assert ((h.float() - a.float() @ w1.float().t()).norm() / h.float().norm()).item() <= 2.0 ** -8
        assert ((y.float() - ref).norm() / ref.norm()).item() <= 2.0 ** -8


def test_status_word_of_a_device_without_an_index_is_the_current_one():
    from memfabric_hybrid_b200.ops import gemm
    here = torch.device("cuda", torch.cuda.current_device())
    assert gemm.status_word("cuda") is gemm.status_word(here) and gemm.status_word() is gemm.status_word(here)
    gemm.status_word().fill_(0x401)
    with pytest.raises(RuntimeError, match="0x401"):
        gemm.check_status("cuda")
    gemm.check_status()
