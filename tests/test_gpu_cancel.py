"""A sweep that is running stops when its scene is cancelled: the flag reaches the device
while the persistent kernel holds every multiprocessor, and the sweep ends at its warps'
next work items.  The plan and its scene stay usable."""
import time

import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


@pytest.mark.parametrize("nf", [1, 40])
def test_cancel_ends_a_running_sweep(nf):
    v, t = M.trihedral(1.0, 100)
    G = 2.0 * M.bounding_radius(v)

    def plan(angles):
        ph = np.linspace(0.0, 90.0, angles)
        return sbr.Plan(s, [sbr.JobSpec(np.full(angles, 54.0), ph, np.linspace(9e9, 1e10, nf), 1500, 1500, G, 3)],
                        first_hit=sbr.FIRST_HIT_TRAVERSE)

    with sbr.Scene(v, t) as s:
        p = plan(64)
        p.execute()
        p.results()
        p.execute()
        want = p.results()
        p.close()
        # one launch of about a second
        p = plan(64 * max(1, round(1000.0 / want.device_ms)))
        p.execute()
        whole = p.results().device_ms
        assert whole > 300.0
        p.execute()
        time.sleep(0.1)
        began = time.monotonic()
        s.cancel()
        with pytest.raises(sbr.SbrError) as e:
            p.results()
        assert e.value.status == 11
        assert 1e3 * (time.monotonic() - began) < 0.5 * (whole - 100.0)
        s.reset_cancel()
        p.close()
        p = plan(64)
        p.execute()
        again = p.results()
        np.testing.assert_array_equal(again.field, want.field)
        np.testing.assert_array_equal(again.stats, want.stats)
        p.close()
