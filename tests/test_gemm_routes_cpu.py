"""Which kernel and which split of K a bf16 product gets: rules on sizes, checked without a GPU."""
import ctypes as C

import pytest

from memfabric_hybrid_b200 import _native as N


@pytest.fixture(scope="module")
def split():
    f = N.cuda().mf_gemm_bf16_split
    f.restype, f.argtypes = C.c_int, [C.c_int] * 4
    return f


@pytest.mark.parametrize("M,N,K,best", [(32, 7168, 8192, 4), (1, 1024, 4096, 8), (128, 1024, 8192, 8), (256, 4096, 8192, 4), (1024, 1280, 1024, 1),
                                        # nearly two CTAs per SM in clusters of two: larger clusters would need a second round
                                        (256, 9216, 8192, 2), (1024, 2304, 16384, 2), (16, 18944, 4096, 2), (128, 18944, 16384, 2), (64, 17408, 4096, 2)])
def test_split_is_the_measured_best(split, M, N, K, best):
    """148 SMs; the times are in the comment of the rule (mf_gemm_splitk.cu)."""
    assert split(M, N, K, 148) == best


@pytest.mark.parametrize("M,N,K,best", [(1, 2048, 2432, 8), (6, 2624, 1856, 4), (31, 4096, 704, 4), (31, 4680, 704, 2)])
def test_split_leaves_clusters_their_sms(split, M, N, K, best):
    """16 and 17 tiles in clusters of eight, 32 and 37 in clusters of four: behind the edge clusters would share SMs."""
    assert split(M, N, K, 148) == best


@pytest.mark.parametrize("M,N,K,best", [(947, 304, 7040, 4), (700, 304, 7040, 4), (962, 224, 4928, 4), (128, 1920, 4096, 8), (800, 200, 8192, 8)])
def test_split_of_whole_tiles_around_the_last_clusters_of_eight_with_sms_of_their_own(split, M, N, K, best):
    """24, 18 and 16 tiles of 128 rows: what clusters of eight share costs them 14 to 27 %; with 15 and 14 tiles they are the fastest by as much."""
    assert split(M, N, K, 148) == best


@pytest.mark.parametrize("sms", [0, 1, 16, 132, 148, 160])
def test_split_never_exceeds_the_steps_of_k(split, sms):
    for M in (1, 8, 100, 128, 129, 2000):
        for N in (8, 128, 1000, 20000):
            for K in (8, 64, 72, 128, 200, 512, 4096):
                s = split(M, N, K, sms)
                assert s in (1, 2, 4, 8) and s <= (K + 63) // 64, (M, N, K, s)


def test_a_product_that_the_split_kernel_cannot_take_goes_to_the_persistent_ones():
    """Without a device nothing launches and the number of SMs is unknown: the library's choice ends as the persistent kernels
    do, not with the split kernel's refusal."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("needs a machine without a device")
    l = N.cuda()

    def rc(name, *extra):
        f = getattr(l, name)
        f.restype = C.c_int
        f.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_int64] * 3 + [C.c_void_p] + [C.c_int] * (2 + len(extra)) + [C.c_void_p]
        return f(4096, 4096, 4096, 32, 1024, 1024, 1024, 1024, 1024, 4096, 148, 0, *extra, None)

    assert rc("mf_gemm_bf16_one") == rc("mf_gemm_bf16_pair") != rc("mf_gemm_bf16_splitk", 0)
    assert rc("mf_gemm_bf16") == rc("mf_gemm_bf16_one")


@pytest.mark.parametrize("steps", [1, 6, 7, 8, 48, 1000, 65_536, 122_606, 122_607, 122_608, 1 << 20, (1 << 26) - 1, 1 << 26])
@pytest.mark.parametrize("widest", [1, 3, 7])
def test_rows_of_a_group_are_cut_into_tiles_without_gaps(steps, widest):
    """Runs of 32 rows, up to the 2^31 rows that the entry takes: every run belongs to one tile and no tile is wider than the others need.
    A 32-bit product of the tile's number and the runs left its range at 122 607 runs (3.9 M rows) in tiles of seven."""
    cut = N.cuda().mf_grouped_gemm_fp8_mx_cut
    cut.restype, cut.argtypes = None, [C.c_int] * 3 + [C.POINTER(C.c_int)] * 2
    cnt = -(-steps // widest)
    first, gran = C.c_int(), C.c_int()
    many = cnt > 2000
    for lo, hi in ([(0, 500), (cnt // 2, cnt // 2 + 500), (cnt - 500, cnt)] if many else [(0, cnt)]):
        end = None
        for mi in range(lo, hi):
            cut(steps, cnt, mi, C.byref(first), C.byref(gran))
            assert 1 <= gran.value <= -(-steps // cnt) and (end is None or first.value == end), mi
            assert mi > 0 or first.value == 0
            end = first.value + gran.value
        assert hi < cnt or end == steps


def test_sm_count_of_a_device_without_an_index_follows_the_current_device(monkeypatch):
    import types

    import torch
    from memfabric_hybrid_b200.ops import gemm

    def props(device):
        d = torch.device(device) if not isinstance(device, int) else torch.device("cuda", device)
        if d.type != "cuda":
            raise ValueError(f"Expected a cuda device, but got: {d}")
        return types.SimpleNamespace(multi_processor_count=100 + (d.index if d.index is not None else torch.cuda.current_device()))

    current = [0]
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    monkeypatch.setattr(torch.cuda, "get_device_properties", props)
    gemm._sms.cache_clear()
    try:
        for current[0] in (0, 1, 0):
            want = 100 + current[0]
            assert [gemm.sm_count(d) for d in (None, "cuda", torch.device("cuda"))] == [want] * 3
            assert [gemm.sm_count(d) for d in (1, "cuda:1", torch.device("cuda", 1))] == [101] * 3
            with pytest.raises(ValueError):
                gemm.sm_count("cpu")
    finally:
        gemm._sms.cache_clear()
