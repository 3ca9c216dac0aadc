"""Measured planning times the kernels a pass really has: passes with one kernel are not timed, their
wisdom holds the default choice, and caps that change nothing are not recorded."""
import numpy as np
import pytest

import pfb200

pytestmark = pytest.mark.gpu

F64, F32 = pfb200.PREC_F64, pfb200.PREC_F32


def tuned(cells, precision):
    """launches of one planning with one repetition, and its wisdom: pass -> (variant, cap)"""
    plan = pfb200.Plan(pfb200.make_desc(dim=len(cells), cells=cells, covariance="exponential", corr_length=0.1,
                                        approximate=True, precision=precision))
    plan.spectrum_build()
    pfb200.wisdom_forget()
    before = plan.launch_count()
    assert plan.autotune(repetitions=1) is True
    launches = plan.launch_count() - before
    rows = [[int(v) for v in line.split()] for line in pfb200.wisdom_export().strip().splitlines()]
    pfb200.wisdom_forget()
    plan.close()
    return launches, {r[0]: (r[5], r[6]) for r in rows}


@pytest.mark.parametrize("cells", [(64, 64), (100, 60), (75, 33)])
def test_fp64_fields_time_the_batch_modes_only(cells):
    """one kernel for each of two passes; each batch mode runs a warm-up and a timed batch of 4"""
    launches, wisdom = tuned(cells, F64)
    assert launches == 2 * 2 * 4 * 2
    assert wisdom[0] == wisdom[2] == (0, 0)


@pytest.mark.parametrize("cells,precision,single", [
    # FP32 axis 1 of 192 and 1024 points: the any-length kernel or, at a power of two, staged tiles;
    # rows of 192 points: any-length
    ((96, 96, 8), F32, (0, 1, 2)),       # noise pass of 16 points
    ((192, 96, 64), F32, (1, 2)),        # noise pass of 128 points: paired or any-length
    ((20, 512, 6), F32, (0, 2)),
    ((64, 50, 40), F64, (0, 1, 2)),
    ((128, 128, 64), F64, (0, 1, 2)),
])
def test_passes_with_one_kernel_keep_the_default(cells, precision, single):
    for _ in range(2):
        _, wisdom = tuned(cells, precision)
        for p in single:
            assert wisdom[p] == (0, 0)
        for p in set(range(3)) - set(single):
            variant, cap = wisdom[p]
            assert variant != 1 or cap == 0  # the any-length kernel has no cap


def test_rows_have_no_paired_kernel():
    """2D FP32 rows of 256 points: the any-length kernel without a cap, or staged by bulk copies"""
    for _ in range(3):
        _, wisdom = tuned((256, 256), F32)
        assert wisdom[2] == (0, 0) or wisdom[2][0] == 2


def test_repeated_plannings_agree():
    """256^3 FP32: 256-point rows staged by bulk copies take 72 us, the any-length ones 70, in events
    that resolve 2 us; forty plannings of one repetition all keep the latter"""
    plan = pfb200.Plan(pfb200.make_desc(dim=3, cells=(256, 256, 256), covariance="matern32", corr_length=0.1,
                                        approximate=True, precision=F32))
    plan.spectrum_build()
    seen = set()
    for _ in range(40):
        pfb200.wisdom_forget()
        plan.autotune(repetitions=1)
        seen |= {line.split()[5] for line in pfb200.wisdom_export().strip().splitlines() if line.split()[0] == "2"}
    pfb200.wisdom_forget()
    plan.close()
    assert seen == {"0"}


@pytest.mark.parametrize("cells,precision", [((128, 128, 64), F32), ((192, 96, 192), F32), ((64, 48), F64)])
def test_planned_fields_equal_unplanned_ones(cells, precision):
    """to the rounding of the kernels that planning may exchange: FP32 1e-5 (eps 6e-8 times a few
    roundings per stage), FP64 bit for bit (one kernel)"""
    d = pfb200.make_desc(dim=len(cells), cells=cells, covariance="exponential", corr_length=0.1, approximate=True,
                         precision=precision)
    plan = pfb200.Plan(d)
    plan.spectrum_build()
    ref = plan.generate(seed=4).astype(np.float64)
    pfb200.wisdom_forget()
    plan.autotune(repetitions=1)
    got = plan.generate(seed=4).astype(np.float64)
    pfb200.wisdom_forget()
    err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    assert err <= (0.0 if precision == F64 else 1e-5)
    plan.close()
