"""The autotuner's two sides do the same work, checked in its source (which side is
faster is a measurement): what the fused kernel forms that the batched GEMMs do not,
the lift and Rh, is timed on the pair's side."""
import os
import re

CAPI = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfem_b200", "csrc", "hfem_capi.cu")


def test_passes_around_the_pair_are_timed():
    src = re.sub(r"//[^\n]*", "", open(CAPI).read())
    body = src[src.index("int hfem_autotune("):src.index("struct hfem_graph {")]
    for name in ("lift_F", "gemv_Rh"):
        assert re.search(r"\b%s\b" % name, body), name
    # the assembly runs the same two around the pair
    pair = src[src.index("int enqueue_assembly("):src.index("int finish_assembly(")]
    assert "lift_F(c)" in pair and "gemv_Rh(c)" in pair
