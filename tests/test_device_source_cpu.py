"""Rules of the kernels' source that no result shows.

The lanes of a sweep's warp part and meet again (a ray may end without a walk), so every
vote, shuffle and reduction of the tracing kernels names the whole warp and stands where
the whole warp is: a mask gathered before the lanes part would wait for lanes that left.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "sagittasbr_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["trace.cu", "trace.cuh", "ray.cuh", "adjoint.cu", "errbound.cu", "horizon.cu"])
def test_warp_operations_name_the_whole_warp(name):
    masks = re.findall(r"__(?:any|all|ballot|shfl\w*|reduce\w*|match\w*)_sync\(\s*([^,]+),", _code(name))
    assert set(masks) <= {"FULL", "0xffffffffu"}
