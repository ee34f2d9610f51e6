"""How a sweep's blocks are cut into work items only regroups FP64 sums: automatic items
(cut down by the sweep's size) against explicit ones, on grids with and without ragged
blocks, in every precision and with few and many channels.  The groups of 32 rays whose
terms the many-channel mixed sweep adds in FP32 stay those of the uncut runs, so that sweep
agrees with runs of the same length to FP64 rounding as well."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"


@pytest.mark.parametrize("nf", [1, 4, 5, 40])
@pytest.mark.parametrize("prec", [sbr.PREC_MIXED, sbr.PREC_FP32, sbr.PREC_FP64])
@pytest.mark.parametrize("nx, ny, run", [(256, 256, 1), (411, 373, 4), (701, 699, 8)])
def test_automatic_items_equal_whole_runs(nx, ny, run, prec, nf):
    v, t = M.icosphere(4, 1.0)
    # a box around the sphere that the projection fills: clipped grids of every raggedness
    th, ph = np.full(6, 70.0), np.linspace(0.0, 100.0, 6)
    job = sbr.JobSpec(th, ph, np.linspace(1e9, 3e9, nf), nx, ny, 2.1, 3)
    with sbr.Scene(v, t, want_fp64=True) as s:
        a = sbr.run(s, job, precision=prec)
        b = sbr.run(s, job, precision=prec, blocks_per_item=run)
    np.testing.assert_array_equal(a.stats, b.stats)
    # FP64 sums of the same terms: a few roundings of each partial sum
    assert np.abs(a.field - b.field).max() <= 1e-12 * np.abs(b.field).max()


@pytest.mark.parametrize("nf", [1, 3, 4, 5, 40])
@pytest.mark.parametrize("prec", [sbr.PREC_MIXED, sbr.PREC_FP32, sbr.PREC_FP64])
@pytest.mark.parametrize("nx, ny", [(9, 5), (33, 31), (64, 64), (130, 127), (200, 190)])
def test_small_launch_equals_its_part_of_a_large_one(nx, ny, prec, nf):
    """One angle alone (its blocks shared by several warps) and among 80 (whole blocks)."""
    v, t = M.plate_cluster(12, 5, seed=4)
    fr = np.linspace(1e9, 3e9, nf)
    ph = np.linspace(0.0, 350.0, 80)
    with sbr.Scene(v, t, want_fp64=True) as s:
        many = sbr.run(s, sbr.JobSpec(np.full(80, 65.0), ph, fr, nx, ny, 2.2, 4), precision=prec)
        for k in (0, 37, 79):
            one = sbr.run(s, sbr.JobSpec([65.0], ph[k:k + 1], fr, nx, ny, 2.2, 4), precision=prec)
            np.testing.assert_array_equal(one.stats[0], many.stats[k])
            m = many.field[k * nf:(k + 1) * nf]
            # FP64 sums of the same terms, and roundings to units of 2^-60 of the field's bound
            assert np.abs(one.field - m).max() <= 1e-12 * np.abs(many.field).max()
