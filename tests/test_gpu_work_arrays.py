"""The work arrays a plan holds on the device, in bytes: the spectrum build leaves the array of the
realization's first pass at the size that pass uses, and the products use the same array, so that
no plan holds one that its calls do not touch."""
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


def make(cells, precision, corr_length=0.1, **kw):
    plan = pfb200.Plan(pfb200.make_desc(dim=len(cells), cells=cells, covariance="exponential",
                                        corr_length=corr_length, approximate=True, precision=precision, **kw))
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


GEO2 = (0.2, 0.05, -0.05, 0.15)
PRODUCTS = {
    "2d-f64": ((512, 512), F64, {}),
    "2d-f32-odd": ((75, 33), F32, {}),
    "2d-r2c": ((60, 50), F64, dict(corr_length=GEO2)),
    "2d-dft": ((48, 36), F64, dict(field_backend=pfb200.FIELD_DFT, matrix_backend=pfb200.MATRIX_DFT)),
    "3d-f64": ((100, 60, 40), F64, {}),
    "3d-f32": ((128, 64, 32), F32, {}),
    "3d-dft": ((24, 20, 18), F64, dict(field_backend=pfb200.FIELD_DFT, matrix_backend=pfb200.MATRIX_DFT)),
}


@pytest.mark.parametrize("name", list(PRODUCTS))
def test_plan_that_only_multiplies_holds_two_arrays(name):
    """the eigenvalues and their square roots in both precisions (24 bytes a value) and the scan's
    result, one factor array, the padded spectrum (X2) and, in 3D, the rows' spectrum (X1)"""
    cells, precision, kw = PRODUCTS[name]
    plan = make(cells, precision, **kw)
    n = int(np.prod(cells))
    x = torch.ones(n, dtype=torch.float64 if precision == F64 else torch.float32, device="cuda")
    plan.matvec(x, precision=precision, out=torch.empty_like(x))
    es = 16 if precision == F64 else 8
    row = 2 * cells[0] if "dft" in name else complex_rows(cells)
    size = int(plan.info.spectrum_size)
    factors = size * es // 2
    if len(cells) == 2:
        work = es * row * cells[1]
    else:
        work = es * row * cells[2] * (cells[1] + 2 * cells[1])
    small = 24 + 32  # scan result; tile counters of the paired FP32 passes
    rest = held(plan) - (24 * size + factors + work)
    assert 0 <= rest <= small
    plan.close()


@pytest.mark.parametrize("cells", [(40, 24), (64, 64, 48)])
def test_fp64_products_of_an_fp32_plan_replace_no_array(cells):
    """they add an array for the padded spectrum; the rows' spectrum of 3D products takes the
    realization's first array, which has its size"""
    plan = make(cells, F32)
    n = int(np.prod(cells))
    plan.generate(seed=1, out=device(n, F32))
    before = held(plan)
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    plan.matvec(x, precision=F64, out=torch.empty_like(x))
    padded = 16 * complex_rows(cells) * (cells[1] if len(cells) == 2 else 2 * cells[1] * cells[2])
    assert held(plan) - before == 8 * int(plan.info.spectrum_size) + padded
    plan.close()


@pytest.mark.parametrize("precision", [F64, F32])
@pytest.mark.parametrize("cells", [(40, 24), (40, 24, 18), (128, 128, 16)])
def test_calls_sharing_the_array_do_not_disturb_each_other(cells, precision):
    """realizations, products of both precisions, and rebuilt spectra on one plan in turn:
    every repeat is bit for bit the first result"""
    plan = make(cells, precision)
    n = int(np.prod(cells))
    es = torch.float64 if precision == F64 else torch.float32
    x64 = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda")

    def results():
        out = [plan.generate(seed=3, out=torch.empty(n, dtype=es, device="cuda")),
               plan.generate_batch(5, 3, out=torch.empty(3 * n, dtype=es, device="cuda"))]
        for p in (F32, F64):
            x = x64.to(torch.float64 if p == F64 else torch.float32)
            out.append(plan.matvec(x, precision=p, out=torch.empty_like(x)))
        out.append(plan.generate(seed=3, out=torch.empty(n, dtype=es, device="cuda")))
        return out

    first = results()
    assert torch.equal(first[0], first[-1])
    for _ in range(2):
        plan.spectrum_build()
        for a, b in zip(first, results()):
            assert torch.equal(a, b)
    plan.close()
