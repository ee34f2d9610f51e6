"""The stated error: its fixed-point term."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


@pytest.mark.parametrize("nx, n", [(2, 1), (4, 3), (12, 1), (30, 2), (230, 3), (300, 90), (1500, 2)])
def test_the_fixed_point_term_covers_every_rays_rounding(nx, n):
    """Four specks that no ray meets: only the fixed-point term is left.  It has to cover the
    rounding of every ray's term, real and imaginary, to half a unit, independent of one
    another (6 sqrt(N / 2) units), and for a single ray as it stands."""
    corner = np.array([[-1, -1, -1], [1, 1, 1], [1, -1, 1], [-1, 1, -1]], dtype=np.float64)
    v = (0.9 * corner[:, None, :] + 1e-6 * np.eye(3)[None]).reshape(-1, 3).astype(np.float32)
    t = np.arange(12, dtype=np.uint32).reshape(-1, 3)
    job = sbr.JobSpec(np.linspace(77.0, 78.0, n), np.linspace(33.0, 34.0, n), [1e9], nx, nx, 4.0, 3)
    with sbr.Scene(v, t) as s:
        r = sbr.run(s, job)
        rays = r.stats[:, 0].astype(np.float64)
        assert rays.min() > 0 and r.stats[:, 1].max() == 0
        err, _ = sbr.error_bound(s, job, r)
    k = 2.0 * np.pi * 1e9 / 299792458.0
    # the unit: 2^-62 of the bound of the rays' sum, the rays' share of the grid taken as a power of two
    share = 2.0 ** np.floor(np.log2(nx * nx / rays))
    unit = 2.0 * k * 4.0 ** 2 / (4.0 * np.pi) / 2.0 ** 62 / share
    assert np.all(err >= (6.0 * np.sqrt(0.5 * rays) + 1.0) * unit * (1.0 - 1e-12))
    assert np.all(err <= 1e-12)
