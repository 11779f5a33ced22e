"""Factors that are no ordinary numbers in the FP64 marches: points where the field is
so high that a factor is zero or denormal, so low that it is infinite, or not a number.
Zero and denormal factors empty their own point and leave the rest as accurate as
before; one that is not finite spoils its instance and no other."""
import numpy as np
import pytest

import test_small_values_gpu as sv

pytestmark = pytest.mark.gpu

GRIDS = [(24, 16, 12), (64, 12, 10), (96, 10, 6), (10, 66, 8), (12, 8, 98), (34, 62, 1), (30, 16, 1), (36, 1, 14)]
DS = 0.1


def point(a, b, grid, value):
    a[b, grid[2] // 2, grid[1] // 2, grid[0] // 3] = value


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("value", [1e6, 2.0 * 720.0 / DS])    # W = 0, W = 1e-313
@pytest.mark.parametrize("grid", GRIDS)
def test_vanishing_factor(pkg, grid, value, fused):
    wa, wb = sv.fields("rough", grid, 2, 0)
    wa, wb = 0.1 * wa, 0.1 * wb
    point(wb, 1, grid, value)
    with pkg.Context(nx=grid[0], ny=grid[1], nz=grid[2], lx=sv.L[0], ly=sv.L[1], lz=sv.L[2], hAB=20.0,
                     fA=0.4, ds0=DS, batch=2, flags=0 if fused else pkg.FLAG_NO_FUSED_STEPS) as c:
        c.set_w(wa, wb)
        c.get_conc()
        ns = (c.NsA, c.dNsB)
        got = [c.get_q(pkg.Q_B, s) for s in range(1, ns[1] + 1)]
    ref = sv.exact(grid, (wa, wb), DS, ns)[ns[0]:]
    fft = sv.by_fft(grid, (wa, wb), DS, ns, np.float64)[ns[0]:]
    here = np.zeros(wb.shape, bool)
    point(here, 1, grid, True)
    for x in got:
        assert np.isfinite(x).all() and (np.abs(x[here]) < 1e-300).all()
    keep = ~here
    err, lim = [max(np.abs(x[keep] / r[keep] - 1).max() for x, r in zip(v, ref)) for v in (got, fft)]
    assert err <= 3 * lim + 4 * 2.0 ** -53 * np.sqrt(sum(ns))


@pytest.mark.parametrize("value", [-1e6, np.nan, np.inf])
@pytest.mark.parametrize("grid", GRIDS)
def test_factor_that_is_not_finite(pkg, grid, value):
    wa, wb = sv.fields("rough", grid, 3, 0)
    clean = wb.copy()
    with pkg.Context(nx=grid[0], ny=grid[1], nz=grid[2], lx=sv.L[0], ly=sv.L[1], lz=sv.L[2], hAB=20.0,
                     fA=0.4, ds0=DS, batch=3) as c:
        c.set_w(wa, wb)
        c.get_conc()
        want = c.phb
        point(wb, 1, grid, value)
        if np.isposinf(value):          # exp(-inf) = 0: an empty point
            c.set_w(wa, wb)
            c.get_conc()
            assert np.isfinite(c.phb).all()
            return
        c.set_w(wa, wb)
        c.get_conc()
        got = c.phb
        assert np.isnan(got[1]).all()
        assert np.array_equal(got[[0, 2]], want[[0, 2]])
        c.set_w(wa, clean)
        c.get_conc()
        assert np.array_equal(c.phb, want)
