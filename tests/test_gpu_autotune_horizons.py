"""The autotuner times every candidate on the same scene: a scene that its candidates' rays
would give horizons gets them before the first of them, not in the middle."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


def _kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    found = sorted((e.time_range.start, e.name) for e in prof.events() if "k_trace<" in e.name or "k_horizon" in e.name)
    return ["horizon" if "k_horizon" in n else "trace" for _, n in found]


@pytest.mark.parametrize("nx, built", [(40, False), (300, True)])
def test_candidates_run_on_one_state_of_the_scene(nx, built):
    v, t = M.icosphere(3, 1.0)
    job = sbr.JobSpec(np.full(8, 80.0), np.linspace(0.0, 300.0, 8), [1e9], nx, nx, 2.1, 3)
    with sbr.Scene(v, t) as s:
        # 24 sweeps of the sample against 1,500 rays per triangle
        assert (24 * 8 * nx * nx >= 2 * 1500 * t.shape[0]) == built
        plans = []
        ran = _kernels(lambda: plans.append(sbr.Plan(s, [job], autotune=True, first_hit=sbr.FIRST_HIT_TRAVERSE)))
        assert ran.count("trace") == 24
        assert ran.count("horizon") == int(built)
        if built:
            assert ran[0] == "horizon"
        plans[0].execute()
        got = plans[0].results()
        plans[0].close()
        want = sbr.run(s, job)
        np.testing.assert_array_equal(got.stats, want.stats)
