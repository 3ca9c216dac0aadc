"""The work arrays a plan holds on the device, in bytes: the spectrum build leaves the array of the
realization's first pass at the size that pass uses."""
import ctypes as C

import numpy as np
import pytest
import torch

import pfb200

pytestmark = pytest.mark.gpu

F64, F32 = pfb200.PREC_F64, pfb200.PREC_F32


def held(plan):
    info = pfb200.PlanInfo()
    assert pfb200.lib().pf_plan_get_info(plan.h, C.byref(info)) == pfb200.PF_OK
    return int(info.device_bytes)


def make(cells, precision, **kw):
    plan = pfb200.Plan(pfb200.make_desc(dim=len(cells), cells=cells, covariance="exponential", corr_length=0.1,
                                        approximate=True, precision=precision, **kw))
    plan.spectrum_build()
    return plan


def device(n, precision):
    return torch.empty(n, dtype=torch.float64 if precision == F64 else torch.float32, device="cuda")


def complex_rows(cells):
    """complex elements of one row of the half spectrum: T0/2 + 1 padded to a multiple of 8"""
    return (cells[0] + 1 + 7) // 8 * 8


# DCT matrices whose spectrum array is a few percent smaller than the realization's (FP64 2D, FP32
# 3D) or half of it (FP64 3D); sides up to 192 so that the arrays stay small
KEPT = {
    "2d-f64-512": ((512, 512), F64),
    "2d-f64-odd": ((75, 33), F64),
    "3d-f64-100": ((100, 100, 100), F64),
    "3d-f32-128": ((128, 128, 128), F32),
    "3d-f32-192": ((192, 192, 192), F32),
    "3d-f64-ragged": ((30, 21, 17), F64),
}


@pytest.mark.parametrize("name", list(KEPT))
def test_first_realization_keeps_the_spectrums_array(name):
    """the first realization adds only the buffers that the build cannot have made: the second work
    array of 3D fields and the tile counters of the paired FP32 passes"""
    cells, precision = KEPT[name]
    plan = make(cells, precision)
    before = held(plan)
    out = device(int(np.prod(cells)), precision)
    plan.generate(seed=1, out=out)
    es = 16 if precision == F64 else 8
    second = es * complex_rows(cells) * cells[1] * cells[2] if len(cells) == 3 else 0
    counters = 32 if precision == F32 else 0
    assert held(plan) - before == second + counters
    after = held(plan)
    plan.spectrum_build()
    plan.generate(seed=2, out=out)
    assert held(plan) == after
    plan.close()
