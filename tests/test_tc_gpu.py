"""Tensor-core passes (csrc/k_tc.cu) against the oracle at the sizes where they
can go wrong: line lengths around multiples of 32 (the points per thread group),
line counts around 128 (the tile), batches, films, every precision, and the
fused march against one launch per pass."""
import numpy as np
import pytest

from oracle import scft_oracle as orc

pytestmark = pytest.mark.gpu

GRIDS = [(2, 4, 6), (30, 2, 34), (32, 34, 4), (34, 62, 1), (64, 2, 66), (66, 6, 10), (16, 8, 1),
         (96, 10, 14), (98, 4, 30), (126, 6, 2), (128, 18, 1), (14, 128, 8)]


def run(pkg, grid, prec, flags=0, batch=1, L=3.0, ds=0.05):
    from scft_gb300 import fields
    nx, ny, nz = grid
    wa, wb = fields.gyroid(nx, ny, nz, L, L, L, 18.0, seed=3, batch=batch)
    with pkg.Context(nx=nx, ny=ny, nz=nz, lx=L, ly=L, lz=L, hAB=18.0, fA=0.36, ds0=ds,
                     batch=batch, precision=prec, flags=flags) as c:
        c.set_w(wa, wb)
        c.get_conc()
        got = [c.pha, c.phb, c.Q(), c.get_q(pkg.Q_B, c.dNsB), c.get_q(pkg.Q_CA, 0)]
    op = orc.Params(nx=nx, ny=ny, nz=nz, lx=L, ly=L, lz=L, hAB=18.0, fA=0.36, ds0=ds, batch=batch)
    ref = orc.get_conc(wa, wb, op)
    return got, ref


def worst(got, ref):
    return max(np.abs(got[0] / ref.pha - 1).max(), np.abs(got[1] / ref.phb - 1).max(),
               np.abs(got[2] / ref.Q - 1).max())


@pytest.mark.parametrize("grid", GRIDS)
def test_fp64_lines(pkg, grid):
    batch = 3 if grid[0] < 40 else 1
    fused, ref = run(pkg, grid, pkg.PREC_FP64, batch=batch)
    assert worst(fused, ref) < 1e-12
    plain, _ = run(pkg, grid, pkg.PREC_FP64, flags=pkg.FLAG_NO_FUSED_STEPS, batch=batch)
    assert worst(plain, ref) < 1e-12
    for a, b in zip(fused[3:], plain[3:]):
        assert np.abs(a - b).max() < 1e-13 * np.abs(b).max()


@pytest.mark.parametrize("grid", GRIDS + [(130, 6, 4), (192, 2, 2), (10, 224, 4), (2, 6, 228)])
def test_fp32_lines(pkg, grid):
    got, ref = run(pkg, grid, pkg.PREC_FP32, batch=2)
    assert worst(got, ref) < 5e-6


def test_strong_fields_and_a_wide_box(pkg):
    """Factors far from one (their exponents differ within a line) and kernels
    with ripples of both signs: the integer units follow the values."""
    rng = np.random.default_rng(5)
    nx, ny, nz, ds = 32, 24, 16, 0.1
    kw = dict(nx=nx, ny=ny, nz=nz, lx=6.0, ly=9.0, lz=5.0, hAB=40.0, fA=0.4, ds0=ds)
    wa = rng.uniform(-60.0, 60.0, (1, nz, ny, nx))
    wb = -wa
    op = orc.Params(**kw)
    ref = orc.get_conc(wa, wb, op)
    with pkg.Context(**kw, precision=pkg.PREC_FP64) as c:
        c.set_w(wa, wb)
        c.get_conc()
        scale = np.abs(ref.pha).max()
        assert np.abs(c.pha - ref.pha).max() < 1e-11 * scale
        assert np.abs(c.phb - ref.phb).max() < 1e-11 * scale
        assert abs(c.Q()[0] / ref.Q[0] - 1) < 1e-11


def test_non_finite_values_spread(pkg):
    """A NaN in a field gives NaN densities, as the FFT passes give."""
    wa = np.zeros((2, 8, 8, 16))
    wa[1, 3, 2, 5] = np.nan
    with pkg.Context(nx=16, ny=8, nz=8, lx=3.0, ly=3.0, lz=3.0, fA=0.5, ds0=0.05, batch=2,
                     precision=pkg.PREC_FP64) as c:
        c.set_field(pkg.FIELD_WA, wa)
        c.set_field(pkg.FIELD_WB, np.zeros_like(wa))
        c.get_conc()
        pha = c.pha
        assert np.isfinite(pha[0]).all()
        assert np.isnan(pha[1]).all()
