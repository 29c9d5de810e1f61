"""Ordering of ordinary stores and bulk copies in the element kernel, checked in its
source: the face slices are stored to global memory by all threads and read back by
cp.async.bulk, so every thread needs the proxy fence between its stores and the CTA
barrier ahead of the copies.  (A missing fence shows as a stale read at most, by
chance, so no run can test for it.)
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfem_b200", "csrc")


def _code(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", src)


def test_global_proxy_fence_is_the_global_one():
    body = re.search(r"bulk_proxy_fence_global\(\)\s*\{(.*?)\}", _code("bulk_copy.cuh"), re.S)
    assert body and "fence.proxy.async.global" in body.group(1)


def test_face_slices_fenced_before_they_are_bulk_loaded():
    src = _code("elem_kernel.cuh")
    stores = [m.end() for m in re.finditer(r"\bslu?\[[^;]*?\] \+?= [^;]*;", src)]
    calls = [m.end() for m in re.finditer(r"\bboundary_fluxes\([^)]*\);", src)]
    assert stores and calls
    last = max(stores + calls)                       # the flux phase's last store of a slice
    load = src.index("bulk_load(sfu, slices")
    assert last < load
    barrier = src.index("__syncthreads();", last)
    assert "bulk_proxy_fence_global();" in src[last:barrier]
