"""The stated error: on little memory, and its fixed-point term."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


def test_the_list_of_flagged_rays_shrinks_to_the_memory_there_is():
    """17 M rays list up to 400 MB at once; with less free, they go in several launches."""
    import torch
    v, t = M.ellipsoid_sh(n_theta=40, n_phi=80)
    G = 2.0 * M.bounding_radius(v)
    small = sbr.JobSpec([80.0], [10.0], [5e9], 100, 100, G, 4)
    job = sbr.JobSpec(np.full(24, 80.0), np.linspace(0.0, 90.0, 24), [5e9], 2000, 2000, G, 4)
    with sbr.Scene(v, t, want_fp64=True) as s:
        sbr.error_bound(s, small, sbr.run(s, small))  # code and stacks of the kernels are on the device
        r = sbr.run(s, job, first_hit=sbr.FIRST_HIT_TRAVERSE)
        assert int(r.stats[:, 0].sum()) > 17_000_000
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        rest = torch.empty(max(0, free - (200 << 20)), dtype=torch.uint8, device="cuda")
        try:
            little = sbr.error_bound(s, job, r)
        finally:
            del rest
            torch.cuda.empty_cache()
        plenty = sbr.error_bound(s, job, r)
    # sums of the same terms in another order
    for a, b in zip(little, plenty):
        np.testing.assert_allclose(a, b, rtol=1e-9)


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


@pytest.mark.parametrize("refl, bounces", [(1.0, 3), (-1.0, 3), (30.0, 8), (-30.0, 8), (100.0, 6)])
def test_equal_terms_round_equally(refl, bounces):
    """A plate seen face on: all rays have one path and one amplitude, so all terms are rounded
    alike.  With a large max(1, R)^max_bounces the unit is coarse against them, and the sum of
    the roundings is a share of the field."""
    v = np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]], dtype=np.float32)
    t = np.array([[0, 1, 2], [0, 2, 3]], dtype=np.uint32)
    G, n = 4.0, 201
    f = np.linspace(1e9, 2e9, 4)
    job = sbr.JobSpec([0.0], [0.0], f, n, n, G, bounces, refl)
    with sbr.Scene(v, t) as s:
        r = sbr.run(s, job)
        err, _ = sbr.error_bound(s, job, r)
    hits = int(r.stats[0, 1])
    assert hits > 5000 and r.stats[0, 2] == hits
    # path 10 G to the plate at z = 0, term k A / (4 pi) * 2 R (-sin, cos)(2 k L)
    k = 2.0 * np.pi * f / 299792458.0
    term = k * (G * G / (n * n)) / (4.0 * np.pi) * 2.0 * refl
    phase = 2.0 * k * 10.0 * G
    exact = hits * term * (-np.sin(phase) + 1j * np.cos(phase))
    assert np.all(np.abs(r.field - exact) <= err)
