"""The accumulator layout a sweep's channel count picks (per lane, or lanes owning 32, 64 or
128 channels) changes no field: jobs at the edges of the layouts against the same
frequencies of the widest job."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M

pytestmark = pytest.mark.gpu

# Scalar mixed terms are explicitly rounded FP32 operations added in one order, so only the
# FP64 sums may differ; elsewhere the compiler may fuse a term's products differently: FP64
# phases of up to 1e3 rad by 1e-13, the FP32 polarised amplitudes by an ulp a term.
CASES = [(sbr.PREC_MIXED, sbr.POL_SCALAR, 1e-12), (sbr.PREC_FP64, sbr.POL_SCALAR, 1e-9),
         (sbr.PREC_MIXED, sbr.POL_HHVV, 1e-5), (sbr.PREC_FP64, sbr.POL_HHVV, 1e-9)]


@pytest.mark.parametrize("prec, pol, tol", CASES)
@pytest.mark.parametrize("channels", [6, 30, 32, 34, 62, 64, 66, 126])
def test_channel_layouts_agree(prec, pol, tol, channels):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    per = 2 if pol == sbr.POL_HHVV else 1
    v, t = M.icosphere(3, 1.0)
    th, ph = np.full(3, 70.0), np.linspace(0.0, 100.0, 3)
    f = np.linspace(1e9, 3e9, 128 // per)
    with sbr.Scene(v, t, want_fp64=True) as s:
        wide = sbr.run(s, sbr.JobSpec(th, ph, f, 131, 127, 2.1, 3), precision=prec, polarization=pol)
        part = sbr.run(s, sbr.JobSpec(th, ph, f[:channels // per], 131, 127, 2.1, 3), precision=prec, polarization=pol)
    np.testing.assert_array_equal(part.stats, wide.stats)
    got = part.field.reshape(3, channels // per, per)
    ref = wide.field.reshape(3, 128 // per, per)[:, :channels // per]
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
