"""The box derivatives' two forms (csrc/adjoint.cu): one filter an axis divided by
the factor, and the whole operator where a factor leaves 2^-60 .. 2^60, against
the oracle's spectral formula, in every precision, on register, generic and
tensor-core lines, with chunks of steps that do not divide the blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [((32, 32, 32), "df"), ((64, 64, 1), "df"), ((12, 8, 6), "fp64"), ((66, 4, 130), "fp64"),
         ((16, 12, 1), "fp64"), ((20, 1, 1), "fp64"), ((64, 64, 16), "fp32"), ((18, 20, 14), "fp32")]
# FP64 and pairs: their unit (1e-16, 4e-15) times some hundred roundings of each
# of the steps' sums; FP32 the same with 6e-8
TOL = {"fp64": 1e-10, "df": 1e-9, "fp32": 2e-4}


@pytest.mark.parametrize("grid,prec", GRIDS)
@pytest.mark.parametrize("spike", [False, True])
def test_stress_and_lnq_gradient(pkg, orc, grid, prec, spike):
    nx, ny, nz = grid
    batch = 2 if nx < 32 else 1
    kw = dict(nx=nx, ny=ny, nz=nz, lx=3.1, ly=2.7, lz=2.4, hAB=15.0, fA=0.35, ds0=0.05, batch=batch)
    rng = np.random.default_rng(nx + ny)
    wa, wb = rng.normal(0, 1.5, (2, batch, nz, ny, nx))
    if spike:                 # 1/W = e^45 (2^65) at a point, where the field shuts the chain out
        wa[0, 0, 0, 1] = wb[0, 0, 0, 3] = 1800.0
    p = orc.Params(**kw)
    with pkg.Context(**kw, precision={"fp64": 0, "fp32": 1, "df": 2}[prec]) as c:
        c.set_w(wa, wb)
        c.get_conc()
        sig, Q = c.stress(), c.Q()
        gL = None if prec == "df" else c.adjoint(Q_bar=1.0 / Q)[2]
    ref = orc.stress_spectral(wa, wb, p)
    assert np.abs(sig - ref).max() < TOL[prec] * np.abs(ref).max()
    if gL is not None:
        assert np.abs(np.reshape(gL, np.shape(sig)) + sig).max() < TOL[prec] * np.abs(ref).max()
