"""The first segments of a segmented prefill run beside the transitions, whose launch stands between them and the chunk-parallel kernel: they
do not wait for a grid before they read that kernel's blocks and norms, so the order is handed on by fences (sm100_ptx.cuh,
grid_dep_handover).  A missing one shows in no result that could be provoked, hence this look at the source."""
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h100_gdn_cuda_b200", "csrc", "kernels")


def text(name):
    with open(os.path.join(KERNELS, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_transitions_release_what_they_have_waited_for():
    calls = re.findall(r"grid_dep_(wait|handover|launch)\(\)", text("prefill_transition.cuh"))
    # the CTA without work, whose end releases the next launch; the producer of the others, and the warp that lets the next launch start
    assert calls == ["wait", "handover", "wait", "wait", "handover", "launch"]


def test_first_segments_acquire_before_they_read():
    t = text("prefill_fused.cuh")
    kernel = t[t.index("gdn_fused_seq_kernel("):]
    producer, prefetcher = kernel[kernel.index("warp == 12"):kernel.index("warp == 14")], kernel[kernel.index("warp == 14"):kernel.index("warp == 13")]
    for role in (producer, prefetcher):
        assert "grid_dep_takeover()" in role
        assert role.index("grid_dep_takeover()") < min(role.index(x) for x in ("p.blocks", "p.norms") if x in role)
    assert "__ldg(nr" not in kernel
