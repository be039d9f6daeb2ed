"""What the kernels' correctness rests on and no run shows, read from their sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfx1151_engine_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_hand_overs_between_ctas_have_the_clusters_scope():
    """A thread's arrival on another CTA's barrier publishes something that CTA goes on with: the default scope, one CTA, does
    not. Copies of a pair of CTAs complete on the barrier that is waited on, and every wait of that kernel acquires at the cluster's scope."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert not re.search(r"mbarrier\.arrive(\.expect_tx)?\.shared::cluster", source(os.path.basename(path))), path
    dense = source("expert_dense.cu")
    assert ".cta_group::2 [%0]" in dense and "tma_load_2d(" not in dense
    assert "mbar_wait(" not in dense and dense.count("mbar_wait<true>(") == 4


def test_aborted_kernels_wait_for_their_copies():
    """A kernel whose bounded wait gave up (abort_flag) lets copies in flight land before it frees its tensor memory and leaves."""
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for kernel in source(os.path.basename(path)).split("__global__")[1:]:
            if "abort_flag" not in kernel or "dealloc" not in kernel:
                continue
            end = kernel[:kernel.index("dealloc")][-900:]
            assert re.search(r"rg_settle\(abort_flag\)|if \(\*abort_flag\) \{[^}]*now_ns\(\) - t0 < 200000ull", end), path
            found += 1
    assert found == 5


def test_an_arrival_is_made_once():
    """The few-row GEMM's dequantising warps tell of a quad's stores later; once told, it is not told again when a wait behind it gives up."""
    few = source("expert_few.cu")
    signal = few[few.index("auto signal = [&]() {"):]
    assert re.search(r"mbar_arrive\(pending\);\s*pending = 0;", signal[:signal.index("};")])


def test_popular_experts_gemm_keeps_out_of_plans_with_a_margin():
    """Launches that fill the GPU and let the next one start early are refused where SMs are to stay free for exchange kernels."""
    dense = source("expert_dense.cu")
    for name in ("launch_expand", "launch_down_dense"):
        body = dense[dense.index("cudaError_t %s(" % name):]
        assert re.match(r"[^{]*\{[^;]*plan->margin > 0\) return cudaErrorNotSupported;", body), name
