"""Calls that a thread may make with another device current select the context's device
ahead of their first launch, allocation or event, checked in the source (a run would
need a second GPU).
"""
import os
import re

import pytest

CAPI = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfem_b200", "csrc", "hfem_capi.cu")


@pytest.mark.parametrize("name", ["hfem_problem_rnorms", "hfem_update_problems", "set_aside", "form_blocks"])
def test_device_selected_first(name):
    src = re.sub(r"//[^\n]*", "", open(CAPI).read())
    body = src[src.index("int %s(" % name):]
    body = body[:body.index("\n}\n")]
    used = [m.start() for m in re.finditer(r"<<<|dalloc\(|cudaEvent\w+\(|element_v\[", body)]
    assert used and 0 <= body.find("cudaSetDevice(c->device)") < min(used)
