"""The raster's per-triangle coverage keeps every hit: first hits of the raster equal the
walk's, ray by ray, where triangles are much smaller than a pixel, much larger than a tile,
seen edge-on, or listed in tiles of every length around the batch of 32 (the last few of a
list are tested without coverage)."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


def _mesh(name):
    rng = np.random.default_rng(11)
    if name == "subpixel":
        return M.icosphere(6, 1.0)
    if name == "large":
        return M.plate_cluster(9, 1, 1.2, 1.0, seed=2)
    if name == "slivers":  # long thin skins seen along and across
        v, t = M.superellipsoid_fuselage(20.0, 1.5, 400, 7)
        return (v + rng.normal(0.0, 1e-3, v.shape)).astype(np.float32), t.astype(np.uint32)
    v, t = M.ellipsoid_sh(n_theta=48, n_phi=96)
    return (v + np.array([3.0, -2.0, 1.0])).astype(np.float32), t


@pytest.mark.parametrize("cap", [1, 4, 5, 6, 31, 32, 33, 37, 38, 64, 1024])
@pytest.mark.parametrize("name", ["subpixel", "large", "slivers", "offset"])
def test_raster_first_hits_equal_the_walk(name, cap):
    v, t = _mesh(name)
    th, ph = np.array([90.0, 90.0, 90.0, 37.0, 0.0, 121.0]), np.array([0.0, 0.7, 90.0, 211.0, 0.0, 300.0])
    G = 2.0 * float(np.abs(v).max()) * 1.5
    job = sbr.JobSpec(th, ph, [2e9], 131, 113, G, 1)
    with sbr.Scene(v, t) as s:
        a = sbr.trace_records(s, job, first_hit=sbr.FIRST_HIT_RASTER, tile_cap=cap)
        b = sbr.trace_records(s, job, first_hit=sbr.FIRST_HIT_TRAVERSE)
    assert (b["count"] > 0).any()
    for key in ("count", "tri", "dist", "normal", "lastdir"):
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
