"""A per-angle sweep's launches run on side streams: the fields are those of a sweep of each
angle alone, on the scene's stream and on a caller's, and consecutive sweeps on different
streams do not mix."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


@pytest.mark.parametrize("prec", [sbr.PREC_FP32, sbr.PREC_MIXED])
@pytest.mark.parametrize("n", [1, 3, 15, 16, 17, 40])
def test_per_angle_sweep_equals_its_angles(n, prec):
    import torch
    v, t = M.plate_cluster(6, 4, seed=9)
    ph = np.linspace(0.0, 330.0, n)
    th = np.full(n, 70.0)
    fr = [1e9, 2e9]
    with sbr.Scene(v, t) as s:
        alone = [sbr.run(s, sbr.JobSpec(th[k:k + 1], ph[k:k + 1], fr, 64, 57, 2.2, 4), mode=sbr.MODE_PER_ANGLE,
                         precision=prec) for k in range(n)]
        field = np.concatenate([a.field for a in alone])
        stats = np.concatenate([a.stats for a in alone])
        job = sbr.JobSpec(th, ph, fr, 64, 57, 2.2, 4)
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        plans = [sbr.Plan(s, [job], mode=sbr.MODE_PER_ANGLE, precision=prec, stream=q.cuda_stream) for q in streams]
        plans.append(sbr.Plan(s, [job], mode=sbr.MODE_PER_ANGLE, precision=prec))
        for _ in range(2):
            for p in plans:
                p.execute()
        for p in plans:
            r = p.results()
            np.testing.assert_array_equal(r.field, field)
            np.testing.assert_array_equal(r.stats, stats)
            p.close()
