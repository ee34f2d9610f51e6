"""An angle's field does not depend on the other angles of its plan, on how a sweep is split
between plans, or on the entry point: each sample is an integer sum of its rays' (or, for
many channels, its groups of rays') rounded terms, whatever items and launches they come
from.  Sizes: work items of 1, 2, 4 and 8 blocks, ragged and whole; launches that share a
block between warps and launches that do not."""
import ctypes as C

import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import _lib
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


@pytest.mark.parametrize("nf", [1, 4, 5, 40])
@pytest.mark.parametrize("prec", [sbr.PREC_MIXED, sbr.PREC_FP32, sbr.PREC_FP64])
@pytest.mark.parametrize("nx, ny, n", [(9, 5, 90), (64, 57, 90), (255, 251, 60), (300, 290, 60), (390, 383, 40),
                                       (1100, 1031, 12), (1601, 1500, 6)])
def test_an_angle_alone_and_among_others(nx, ny, n, prec, nf):
    v, t = M.plate_cluster(12, 5, seed=4)
    fr = np.linspace(1e9, 3e9, nf)
    th, ph = np.linspace(50.0, 120.0, n), np.linspace(0.0, 350.0, n)
    G = 2.0 * M.bounding_radius(v)

    def job(a, b):
        return sbr.JobSpec(th[a:b], ph[a:b], fr, nx, ny, G, 4)

    with sbr.Scene(v, t, want_fp64=True) as s:
        whole = sbr.run(s, job(0, n), precision=prec)
        halves = [sbr.run(s, job(0, n // 3), precision=prec), sbr.run(s, job(n // 3, n), precision=prec)]
        np.testing.assert_array_equal(np.concatenate([h.field for h in halves]), whole.field)
        # the same angle twelve times over: another number of blocks for each warp
        more = sbr.run(s, sbr.JobSpec(np.tile(th, 12), np.tile(ph, 12), fr, nx, ny, G, 4), precision=prec) \
            if nx < 1000 else whole
        np.testing.assert_array_equal(more.field[:whole.field.size], whole.field)
        for k in (0, n // 2, n - 1):
            one = sbr.run(s, job(k, k + 1), precision=prec)
            np.testing.assert_array_equal(one.field, whole.field[k * nf:(k + 1) * nf])
            np.testing.assert_array_equal(one.stats[0], whole.stats[k])


@pytest.mark.parametrize("nf", [1, 40])
@pytest.mark.parametrize("first_hit", [sbr.FIRST_HIT_TRAVERSE, sbr.FIRST_HIT_RASTER])
def test_every_cut_of_large_angles(nf, first_hit):
    """Angles of 276,000 blocks, 58 for each resident warp: 1, 10 and 36 of them are cut into
    items of 2, 4 and 8 blocks, ragged at both edges.  With many channels the items share runs
    of 8 blocks."""
    v, t = M.icosphere(4, 1.0)
    th, ph = np.linspace(60.0, 100.0, 36), np.linspace(0.0, 200.0, 36)
    fr = np.linspace(1e9, 3e9, nf)
    with sbr.Scene(v, t) as s:
        runs = [sbr.run(s, sbr.JobSpec(th[:n], ph[:n], fr, 3001, 2941, 2.01, 3), first_hit=first_hit)
                for n in (1, 10, 36)]
    for few, many in zip(runs, runs[1:]):
        np.testing.assert_array_equal(many.field[:few.field.size], few.field)
        np.testing.assert_array_equal(many.stats[:few.stats.shape[0]], few.stats)


@pytest.mark.parametrize("nf", [1, 3])
def test_polarised(nf):
    v, t = M.icosphere(4, 1.0)
    th, ph = np.linspace(60.0, 100.0, 4), np.linspace(0.0, 200.0, 4)
    fr = np.linspace(1e9, 3e9, nf)
    with sbr.Scene(v, t, want_fp64=True) as s:
        for nx, prec in ((700, sbr.PREC_MIXED), (130, sbr.PREC_MIXED), (130, sbr.PREC_FP64)):
            whole = sbr.run(s, sbr.JobSpec(th, ph, fr, nx, nx - 3, 2.1, 3), precision=prec, polarization=sbr.POL_HHVV)
            one = sbr.run(s, sbr.JobSpec(th[2:3], ph[2:3], fr, nx, nx - 3, 2.1, 3), precision=prec,
                          polarization=sbr.POL_HHVV)
            np.testing.assert_array_equal(one.field, whole.field[2 * nf:3 * nf])


@pytest.mark.parametrize("nx, n", [(64, 3), (300, 40), (700, 9)])
def test_the_allocation_free_sweep_adds_the_same_items(nx, n):
    import torch
    v, t = M.icosphere(4, 1.0)
    job = sbr.JobSpec(np.full(n, 80.0), np.linspace(0.0, 300.0, n), [1e9, 2e9], nx, nx, 2.1, 3)
    with sbr.Scene(v, t, device=0) as s:
        want = sbr.run(s, job)
        field = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        jc, opts = job.to_c(), _lib.RunOpts()
        _lib.check(_lib.lib().sbr_run_noalloc(s.handle, C.byref(jc), C.c_void_p(field.data_ptr()), None,
                                              C.byref(opts)), "sbr_run_noalloc")
        f = field.cpu().numpy()
        np.testing.assert_array_equal(f[0::2] + 1j * f[1::2], want.field)
