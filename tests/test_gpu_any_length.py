"""The any-length passes at the edges of their rules: every radix alone and in chains, lengths with
the factors 11 and 13, Bluestein lengths beside the smooth ones, odd cells (field rows that cannot
be read in pairs), odd and even numbers of pencils, all eigenvalue layouts and draw orders, and
sizes that give the smallest and the largest tiles.  Against the oracle, with the suite's bounds:
FP64 1e-12 for eigenvalues and products, 1e-11 for fields; FP32 1e-5 (eps 6e-8 times a few
roundings per stage, at most 8 stages and two transforms)."""
import numpy as np
import pytest

import pfb200
from helpers import counter_noise, desc_of, rel

pytestmark = pytest.mark.gpu

LENGTHS = {
    # torus lengths 2 n: one radix (2..16), two and more stages, 7-, 11- and 13-smooth, odd cells
    "2d-r2-r6": dict(cells=(2, 3)),
    "2d-r10-r14": dict(cells=(10, 7)),
    "2d-r22-r26": dict(cells=(11, 13)),
    "2d-7smooth": dict(cells=(49, 63)),
    "2d-121-169": dict(cells=(121, 169)),
    "2d-odd-75-125": dict(cells=(75, 125)),
    "2d-long-1000": dict(cells=(1000, 6)),
    "2d-long-last": dict(cells=(6, 1500)),
    "2d-prime-rows": dict(cells=(17, 64)),
    "2d-prime-last": dict(cells=(64, 17)),
    "2d-prime-1021": dict(cells=(1021, 5)),
    "2d-geo": dict(cells=(30, 50), corr_length=(0.2, 0.05, -0.05, 0.15)),
    "3d-ragged": dict(cells=(9, 10, 15)),
    "3d-r2c-untransposed": dict(cells=(14, 9, 11), matrix_backend=pfb200.MATRIX_R2C, transposed=0),
    "3d-dft-matrix": dict(cells=(6, 10, 7), matrix_backend=pfb200.MATRIX_DFT, field_backend=pfb200.FIELD_R2C),
    "3d-many-pencils": dict(cells=(100, 40, 12)),
}


@pytest.mark.parametrize("prec", [pfb200.PREC_F64, pfb200.PREC_F32])
@pytest.mark.parametrize("name", list(LENGTHS))
def test_any_length(oracle, name, prec):
    cfg = dict(dim=len(LENGTHS[name]["cells"]), covariance="exponential", corr_length=0.15, approximate=True)
    cfg.update(LENGTHS[name])
    d = desc_of(cfg, precision=prec)
    lam, st, _ = oracle.spectrum(d)
    g = oracle.resolve(d)
    P = pfb200.Plan(d)
    P.spectrum_build()
    assert rel(P.spectrum(), lam) < 1e-12
    f64 = prec == pfb200.PREC_F64
    noise = oracle.noise(7, g.noise)
    ref, _ = oracle.generate(d, lam, noise)
    assert rel(P.generate(noise=noise), ref) < (1e-11 if f64 else 1e-5)
    ref, _ = oracle.generate(d, lam, counter_noise(g, 41, f64))
    assert rel(P.generate(seed=41), ref) < (1e-9 if f64 else 1e-5)
    x = np.random.default_rng(5).standard_normal(g.domain).astype(np.float64 if f64 else np.float32)
    y = P.matvec(x, op=pfb200.OP_MUL, precision=prec)
    assert rel(y, oracle.matvec(d, lam, pfb200.OP_MUL, x.astype(np.float64))) < (1e-12 if f64 else 1e-5)
    P.close()


def test_rejected_lengths_stay_rejected():
    """lengths the passes refuse: above 4096 with a prime factor above 13, and FP64 pencils whose
    two copies do not fit in shared memory"""
    for cells, msg in (((64, 2053), "above 4096 has a prime factor above 13"),
                       ((64, 4096), "does not fit in shared memory")):
        P = pfb200.Plan(desc_of(dict(dim=2, cells=cells, covariance="exponential", corr_length=0.1)))
        with pytest.raises(pfb200.PfError, match=msg):
            P.spectrum_build()
        P.close()
