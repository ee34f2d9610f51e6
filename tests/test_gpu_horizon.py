"""Horizons only skip walks that return a miss: a scene with horizons traces bit for bit
like the same scene without them.  A scene gets them once its sweeps have launched 1,500
rays per triangle; a refit to the vertices it already has recomputes the same boxes and triangles
and drops them again.  Plans made before the horizons change read them as well."""
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
    rng = np.random.default_rng(7)
    if name == "trihedral":        # walls at right angles, coplanar neighbours
        return M.trihedral(1.0, 20)
    if name == "dihedral":
        return M.dihedral(1.0, 16)
    if name == "plates":           # crossing plates, lit and unlit sides
        return M.plate_cluster(24, 6, seed=5)
    if name == "aircraft":         # jittered skins, thin edges, wing and body
        return M.aircraft(3, 1e-3, (60, 36), (12, 40), (6, 14))
    v, t = M.ellipsoid_sh(n_theta=24, n_phi=48)
    if name == "jittered":
        v = (v + rng.normal(0.0, 0.02, v.shape)).astype(np.float32)
    elif name == "tiny":           # triangles below tMin and the nudge
        v = (2e-3 * v + rng.normal(0.0, 2e-5, v.shape)).astype(np.float32)
    elif name == "far":            # coordinates rounded to a good part of the nudge
        v = (8.0 * v + np.array([20.0, -10.0, 5.0])).astype(np.float32)
    elif name == "huge":           # beyond the tolerances: no horizons
        v = (60.0 * v).astype(np.float32)
    return v, t


@pytest.mark.parametrize("prec", [sbr.PREC_MIXED, sbr.PREC_FP64])
@pytest.mark.parametrize("name", ["trihedral", "dihedral", "plates", "aircraft", "ellipsoid", "jittered", "tiny", "far",
                                  "huge"])
def test_horizons_change_nothing(name, prec):
    v, t = _mesh(name)
    rng = np.random.default_rng(1)
    th, ph = rng.uniform(0.0, 180.0, 7), rng.uniform(0.0, 360.0, 7)
    G = 2.0 * float(np.abs(v).max()) * 1.8
    job = sbr.JobSpec(th, ph, [1e9, 1.7e9, 3e9, 4e9, 6e9, 9e9], 90, 83, G, 6)
    # scene b: below 1,500 rays per triangle over all its sweeps (the records do not count)
    assert 3 * 7 * 90 * 83 < 1500 * t.shape[0]
    with sbr.Scene(v, t, want_fp64=True) as a, sbr.Scene(v, t, want_fp64=True) as b:
        n, rays = 1500, 0
        while rays <= 1500 * t.shape[0]:
            many = sbr.JobSpec(np.linspace(20.0, 160.0, 5), np.linspace(0.0, 300.0, 5), [1e9], n, n, G, 1)
            rays += int(sbr.run(a, many).stats[:, 0].sum())
        if prec == sbr.PREC_FP64:
            plan = sbr.Plan(a, [job], precision=prec)
            plan.execute()
            with_them = plan.results()
            a.update_vertices(v)
            plan.execute()  # the same plan, walking
            np.testing.assert_array_equal(plan.results().field, with_them.field)
            plan.close()
            rays = 0
            while rays <= 1500 * t.shape[0]:
                rays += int(sbr.run(a, many).stats[:, 0].sum())
        ra, rb = sbr.trace_records(a, job, precision=prec), sbr.trace_records(b, job, precision=prec)
        for key in ("count", "tri", "dist", "normal", "lastdir", "flags"):
            np.testing.assert_array_equal(ra[key], rb[key], err_msg=key)
        for pol in (sbr.POL_SCALAR, sbr.POL_HHVV):
            fa, fb = (sbr.run(s, job, precision=prec, polarization=pol) for s in (a, b))
            np.testing.assert_array_equal(fa.field, fb.field)
            np.testing.assert_array_equal(fa.stats, fb.stats)
        if name != "tiny" and name != "huge":
            assert fa.bounces > 0
        cot = np.ones(fa.stats.shape[0] * 6, complex)
        ga, gb = (sbr.adjoint(s, job, cot, precision=prec)[0] for s in (a, b))
        np.testing.assert_allclose(ga, gb, rtol=1e-9, atol=1e-9 * np.abs(gb).max() + 1e-300)
