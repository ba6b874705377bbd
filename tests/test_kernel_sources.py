"""Ordering rules of the GEMM kernels that no run can show to be kept, read off their sources."""
import re
from pathlib import Path

import pytest

GEMM = Path(__file__).resolve().parent.parent / "csrc" / "gemm"
KERNELS = ["fo_gemm_plain_sm100.cuh", "fo_gemm_sm100.cuh", "fo_gemm_splitk_sm100.cuh"]


def _code(name):
    return re.sub(r"//[^\n]*", "", (GEMM / name).read_text())


@pytest.mark.parametrize("name", KERNELS)
def test_tmem_base_is_read_behind_an_ordering_barrier(name):
    """tcgen05.alloc writes the TMEM address to shared memory, and one thread clears the abort flag: the
    barrier between them and their readers must order memory (a CTA barrier or a cluster barrier's
    release form), in every branch."""
    code = _code(name)
    begin, end = code.index("tmem_alloc"), code.index("tmem_base = *s_tmem_base")
    setup = code[code.rindex("tmem_relinquish", begin, end):end]
    pair, _, single = setup.partition("} else {") if "if constexpr (CTA2)" in setup else (setup, "", setup)
    for branch in (pair, single):
        barriers = re.findall(r"cluster_arrive_\w+|__syncthreads", branch)
        assert barriers and barriers[0] in ("__syncthreads", "cluster_arrive_release"), barriers


def test_fused_pairs_hand_accumulators_back_at_cluster_scope():
    """CTA pairs of the kernels that run over several GPUs keep the arrive that releases at cluster scope; the
    CTA-scope form is the plain kernel's and, on its own barrier, that of a CTA by itself."""
    ptx = re.sub(r"//[^\n]*", "", (GEMM.parent / "common" / "fo_ptx.cuh").read_text())
    body = ptx[ptx.index("void mbar_arrive_cluster("):]
    assert "mbarrier.arrive.release.cluster.shared::cluster" in body[:body.index("}")]
    fused = re.sub(r"\s+", " ", _code("fo_gemm_sm100.cuh"))
    assert re.search(r"if constexpr \(CTA2\) \{ ptx::mbar_arrive_cluster\([^;]*\); \} else \{ ptx::mbar_arrive_cluster_tmem\(", fused)
    assert fused.count("mbar_arrive_cluster") == 2


def test_objects_and_launches_query_no_device_properties():
    """cudaGetDeviceProperties takes milliseconds: not once per object, nor per kernel of a choice."""
    for path in ("runtime/overlap_impl.cpp", "runtime/loopback.cpp", "gemm/fo_gemm_launch.cuh", "gemm/fo_gemm_splitk_launch.cu"):
        assert "cudaGetDeviceProperties(" not in re.sub(r"//[^\n]*", "", (GEMM.parent / path).read_text()), path


@pytest.mark.parametrize("name,barrier", [("fo_gemm_plain_sm100.cuh", "cluster_arrive_relaxed"), ("fo_gemm_splitk_sm100.cuh", "cluster_arrive_release")])
def test_roles_join_their_warps_before_the_cluster_barrier(name, barrier):
    """barrier.cluster's aligned form is undefined for a warp whose lanes arrive apart; the roles end in
    code that one lane runs."""
    code = _code(name)
    tail = code[:code.rindex(barrier)].rstrip()
    assert "__syncwarp();" in tail[-250:], tail[-250:]


def test_a_tile_is_stamped_as_signalled_before_its_owners_can_see_it():
    code = _code("fo_gemm_sm100.cuh")
    loop = code[code.index("const int g = s_sig_g[slot]"):code.index("mbar_arrive(&sig_empty_bar[slot])")]
    assert loop.index("kTraceSignalled") < loop.index("red_relaxed_sys_add")
