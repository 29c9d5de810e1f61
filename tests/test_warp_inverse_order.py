"""Order of the warp inverse's shared-memory accesses, checked in its source.  Step k
writes the pivot row to buffer k & 1 and all lanes read it; the step after writes the
other, so a buffer's next write is a warp barrier behind its reads.  Between two matrices
that does not hold by itself: with an odd order, or after a singular matrix, the next
first step writes the buffer just read, and votes and shuffles order no memory.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfem_b200", "csrc")


def test_warp_barrier_between_matrices():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "inverse_blocked.cuh")).read())
    body = src[src.index("inverse_warp_kernel("):]
    loop = body.index("for (int e = ")
    write = body.index("b[c] = make_double2", loop)
    read = body.index("const double2 r = b[c];", write)
    assert "__syncwarp();" in body[write:read]                              # write, barrier, read
    assert "__syncwarp();" in body[loop:body.index("for (int k = 0", loop)]  # read, barrier, the next matrix's write
