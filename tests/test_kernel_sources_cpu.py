"""Rules of the kernel sources that no run can show reliably."""
import re

import pytest

from conftest import ROOT

KERNELS = ROOT / "memfabric_hybrid_b200" / "csrc" / "kernels"


def _functions(text):
    """name -> (signature, body) of every function definition (comments removed; a later overload adds to an earlier one)."""
    text = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
    out = {}
    for m in re.finditer(r"(__global__|__device__)[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*(const\s*)?\{", text):
        sig = re.sub(r"__launch_bounds__\s*\([^()]*(\([^()]*\)[^()]*)*\)", "", m.group(0))
        name = re.search(r"(\w+)\s*\(", sig[len(m.group(1)):])
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        old = out.get(name.group(1), ("", ""))
        out[name.group(1)] = (old[0] + sig, old[1] + text[m.end():i])
    return out


def _overlapped():
    """Kernels that may start under the end of their predecessor, each with every device function it can reach."""
    headers = "".join(p.read_text() for p in sorted(KERNELS.glob("*.cuh")))
    for src in sorted(KERNELS.glob("*.cu")):
        text = src.read_text()
        if "after_predecessor()" not in text:
            continue
        fns = _functions(headers + text)
        for name, (sig, body) in sorted(fns.items()):
            if "__global__" in sig and "after_predecessor()" in body:
                reach, todo = set(), [name]
                while todo:
                    f = todo.pop()
                    if f not in reach:
                        reach.add(f)
                        todo += [c for c in re.findall(r"\b(\w+)\s*(?:<[^<>;()]*>)?\s*\(", fns[f][1]) if c in fns]
                yield src.name, name, {f: fns[f] for f in reach}


def test_overlapped_kernels_are_found():
    names = {k for _, k, _ in _overlapped()}
    assert {"k_moe_prepare", "k_moe_dispatch", "k_moe_dispatch_warp", "k_moe_wait_all", "k_moe_combine_reduce", "k_grouped_fp8_mx",
            "k_gemm_bf16_splitk"} <= names


@pytest.mark.parametrize("src,kernel,reach", list(_overlapped()), ids=lambda v: v if isinstance(v, str) else "")
def test_overlapped_kernels_read_nothing_through_the_read_only_path(src, kernel, reach):
    """A kernel that is placed under the end of its predecessor is there while that one still writes. __ldg and const
    __restrict__ parameters say that nothing changes during the kernel, and allow loads in front of the wait."""
    for name, (sig, body) in reach.items():
        assert "__ldg(" not in body, f"{src}: {name} (reached from {kernel}) reads through the read-only path"
        assert not re.search(r"const\b[^,()]*__restrict__", sig), f"{src}: {name} (reached from {kernel}) takes a read-only pointer"


def test_what_crosses_a_cluster_is_ordered_for_the_cluster():
    """An arrival or a wait without a scope orders the memory of one CTA. An arrival on another CTA's barrier names the cluster, with a release of its own
    or right behind a fence; a barrier that another CTA's threads arrive on is waited for with an acquire of the same scope."""
    text = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(KERNELS.glob("*.cu*"))}
    arrivals = [(n, m.group(0)) for n, t in text.items() for m in re.finditer(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.]*", t)]
    assert len(arrivals) >= 2
    for name, a in arrivals:
        assert ".release.cluster" in a or ".relaxed.cluster" in a, (name, a)
        if ".relaxed.cluster" in a:
            assert re.search(r"fence\.release\.sync_restrict::shared::cta\.cluster;[\s\\nt\"]*" + re.escape(a), text[name]), (name, a)
    pair = text["mf_gemm_fp8_pair.cu"]
    shared = set(re.findall(r"mbar_arrive_cluster(?:_smem)?\(mapa_u32\(smem_u32\(sm\.(\w+)\(", pair))
    assert shared == {"sf_full", "tempty", "amax_full"}
    for bar in shared:
        waits = re.findall(r"mbar_wait(<true>)?\(sm\." + bar + r"\(", pair)
        assert waits and all(waits), bar
