"""Rules of the kernels' source that no result shows.

* The lanes of a sweep's warp part and meet again (a ray may end without a walk), so every
  vote, shuffle and reduction of the tracing kernels names the whole warp and stands where
  the whole warp is: a mask gathered before the lanes part would wait for lanes that left.
* Horizon bytes change in place while sweeps of other streams read them: they are not read
  through the read-only path, which assumes memory that nothing writes during the kernel.
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


def test_horizon_bytes_are_not_read_as_read_only():
    reads = re.findall(r"[^\n;]*\bS\.horizon\b[^\n;]*", _code("ray.cuh"))
    assert reads and all("load_horizon(" in r for r in reads)
    assert "ld.relaxed.gpu" in _code("ray.cuh")
    field = re.search(r"[^\n;]*\bhorizon;", _code("common.hpp")).group()
    assert "__restrict__" not in field
