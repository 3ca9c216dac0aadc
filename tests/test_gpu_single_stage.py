"""Any-length passes of one stage, where the first stage is also the last: every radix that is
built (1, 2, 3, 4, 5, 6, 7, 8, 11, 13) as the whole row, the whole strided pencil and the whole
fused pencil of a product.  Odd pencils are periodic fields with the R2C matrix, whose torus is the
domain.  Against the oracle with the suite's bounds: FP64 1e-12 for eigenvalues and products, 1e-11
for fields; FP32 1e-5.  And the launches of one plan in turn: results repeat bit for bit."""
import numpy as np
import pytest
import torch

import pfb200
from helpers import desc_of, rel

pytestmark = pytest.mark.gpu

F64, F32 = pfb200.PREC_F64, pfb200.PREC_F32
ODD = dict(periodic=True, matrix_backend=pfb200.MATRIX_R2C, field_backend=pfb200.FIELD_R2C)
# rows have half the extended cells of dimension 0
SINGLE = {
    "rows-1": dict(cells=(1, 3)),
    "rows-2-pencils-6": dict(cells=(2, 3)),
    "rows-3-pencils-8": dict(cells=(3, 4)),
    "rows-4-pencils-4": dict(cells=(4, 2)),
    "rows-5-pencils-2": dict(cells=(5, 1)),
    "rows-6": dict(cells=(6, 4)),
    "rows-7": dict(cells=(7, 2)),
    "rows-8": dict(cells=(8, 3)),
    "rows-11": dict(cells=(11, 4)),
    "rows-13": dict(cells=(13, 2)),
    "pencils-1": dict(cells=(8, 1), **ODD),
    "pencils-3": dict(cells=(26, 3), **ODD),
    "pencils-5": dict(cells=(10, 5), **ODD),
    "pencils-7": dict(cells=(14, 7), **ODD),
    "pencils-11": dict(cells=(22, 11), **ODD),
    "pencils-13": dict(cells=(16, 13), **ODD),
    "3d-3-8-6": dict(cells=(3, 4, 3)),
    "3d-5-4-8": dict(cells=(5, 2, 4)),
    "3d-13-7-5": dict(cells=(26, 7, 5), **ODD),
    "3d-7-13-11": dict(cells=(14, 13, 11), **ODD),
}


@pytest.mark.parametrize("prec", [F64, F32])
@pytest.mark.parametrize("name", list(SINGLE))
def test_single_stage(oracle, name, prec):
    cfg = dict(dim=len(SINGLE[name]["cells"]), covariance="exponential", corr_length=0.15, approximate=True)
    cfg.update(SINGLE[name])
    d = desc_of(cfg, precision=prec)
    lam, _, _ = oracle.spectrum(d)
    g = oracle.resolve(d)
    P = pfb200.Plan(d)
    P.spectrum_build()
    f64 = prec == F64
    assert rel(P.spectrum(), lam) < 1e-12
    noise = oracle.noise(7, g.noise)
    ref, _ = oracle.generate(d, lam, noise)
    assert rel(P.generate(noise=noise), ref) < (1e-11 if f64 else 1e-5)
    ref, _ = oracle.generate(d, lam, P.export_noise(41))
    assert rel(P.generate(seed=41), ref) < (1e-11 if f64 else 1e-5)
    x = np.random.default_rng(5).standard_normal(g.domain).astype(np.float64 if f64 else np.float32)
    y = P.matvec(x, op=pfb200.OP_MUL, precision=prec)
    assert rel(y, oracle.matvec(d, lam, pfb200.OP_MUL, x.astype(np.float64))) < (1e-12 if f64 else 1e-5)
    P.close()


@pytest.mark.parametrize("cells", [(128, 128), (192, 64, 96), (128, 128, 128)])
def test_repeated_and_batched_launches_agree(cells):
    """FP32 lengths of the paired kernels, whose tile counters reset themselves: realizations alone and
    in two-stream batches, products and rebuilt spectra in turn, each repeat bit for bit the first"""
    P = pfb200.Plan(pfb200.make_desc(dim=len(cells), cells=cells, covariance="exponential", corr_length=0.1,
                                     approximate=True, precision=F32))
    n = P.info.domain_size
    x = torch.linspace(-1.0, 1.0, n, device="cuda")
    first = None
    for _ in range(3):
        P.spectrum_build()
        singles = [P.generate(seed=60 + r, out=torch.empty(n, device="cuda")) for r in range(5)]
        batch = P.generate_batch(60, 5, out=torch.empty(5 * n, device="cuda"))
        y = P.matvec(x, precision=F32, out=torch.empty(n, device="cuda"))
        torch.cuda.synchronize()
        for r in range(5):
            assert torch.equal(batch[r * n:(r + 1) * n], singles[r]), r
        if first is None:
            first = singles + [y]
        assert all(torch.equal(a, b) for a, b in zip(first, singles + [y]))
    P.close()
