"""Contexts whose passes run on different kernels: tensor-core axes beside register and
FFT axes in every place of the fused schedules, against the oracle and against one
launch per pass; and repeated runs of the tensor-core marches bit by bit."""
import numpy as np
import pytest

from test_tc_gpu import run, worst

pytestmark = pytest.mark.gpu

# FP32: the tensor cores along x, y, z and pairs of them, register kernels on the rest;
# FP64: an axis above 128 points (FFT) beside tensor-core ones
MIXED = [((100, 64, 64), 1), ((64, 100, 64), 1), ((64, 64, 20), 1), ((64, 20, 64), 1), ((100, 80, 64), 1),
         ((96, 60, 32), 1), ((100, 64, 1), 1), ((130, 64, 32), 0), ((64, 20, 132), 0), ((32, 140, 1), 0)]


@pytest.mark.parametrize("grid,prec", MIXED)
@pytest.mark.parametrize("ds", [0.05, 0.025])      # odd and even step counts
def test_mixed_axes(pkg, grid, prec, ds):
    tol = (1e-12, 5e-6)[prec]
    fused, ref = run(pkg, grid, prec, ds=ds)
    assert worst(fused, ref) < tol
    plain, _ = run(pkg, grid, prec, flags=pkg.FLAG_NO_FUSED_STEPS, ds=ds)
    assert worst(plain, ref) < tol


@pytest.mark.parametrize("grid,prec", [((60, 60, 60), 1), ((100, 80, 60), 1), ((100, 64, 64), 1),
                                       ((130, 20, 12), 1), ((96, 80, 40), 0), ((60, 48, 40), 0),
                                       ((32, 24, 1), 0), ((64, 64, 1), 0)])
def test_get_conc_is_bit_reproducible(pkg, grid, prec):
    from scft_gb300 import fields
    nx, ny, nz = grid
    wa, wb = fields.gyroid(nx, ny, nz, 3.8, 3.8, 3.8, 18.0, seed=4, batch=2)
    with pkg.Context(nx=nx, ny=ny, nz=nz, lx=3.8, ly=3.8, lz=3.8, hAB=18.0, fA=0.36, ds0=0.01,
                     batch=2, precision=prec) as ctx:
        ctx.set_w(wa, wb)
        ctx.get_conc()
        ref = (ctx.pha.copy(), ctx.phb.copy(), ctx.Q().copy())
        for _ in range(8):
            ctx.set_w(wa, wb)
            ctx.iterate(1)            # other fields in between
            ctx.set_w(wa, wb)
            ctx.get_conc()
            for a, b in zip((ctx.pha, ctx.phb, ctx.Q()), ref):
                assert np.array_equal(a, b)
