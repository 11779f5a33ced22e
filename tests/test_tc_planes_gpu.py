"""Steps on whole planes (csrc/k_tc.cu, k_planes) against the oracle and against
one launch per axis: planes that fill a CTA's lines and that do not, several
planes per CTA, one to four copies of a line, films, odd and even step counts."""
import numpy as np
import pytest

from test_tc_gpu import run, worst
from oracle import scft_oracle as orc

pytestmark = pytest.mark.gpu

CASES = [((64, 64, 6), 1), ((62, 64, 10), 1), ((60, 34, 4), 2), ((20, 20, 20), 1), ((12, 10, 14), 40),
         ((32, 2, 6), 1), ((2, 4, 2), 3), ((36, 36, 6), 12), ((64, 64, 2), 80),
         ((32, 32, 1), 1), ((30, 16, 1), 3), ((2, 2, 1), 1), ((4, 32, 1), 200)]


@pytest.mark.parametrize("grid,batch", CASES)
@pytest.mark.parametrize("ds", [0.05, 0.02])       # 7 + 13 steps, 18 + 32 steps
def test_fp64_planes(pkg, grid, batch, ds):
    planes, ref = run(pkg, grid, pkg.PREC_FP64, batch=batch, ds=ds)
    assert worst(planes, ref) < 1e-12
    passes, _ = run(pkg, grid, pkg.PREC_FP64, flags=pkg.FLAG_NO_XY, batch=batch, ds=ds)
    for a, b in zip(planes[3:], passes[3:]):
        assert np.abs(a - b).max() < 1e-13 * np.abs(b).max()


@pytest.mark.parametrize("grid,batch", [c for c in CASES if c[0][2] > 1] + [((60, 60, 60), 1)])
def test_fp32_planes(pkg, grid, batch):
    got, ref = run(pkg, grid, pkg.PREC_FP32, batch=batch)
    assert worst(got, ref) < 5e-6


def test_film_strong_fields_and_non_finite(pkg):
    """A film's segment keeps its own units from step to step; an instance with a
    NaN in a field gives NaN densities and leaves the others alone."""
    rng = np.random.default_rng(7)
    kw = dict(nx=32, ny=24, nz=1, lx=6.0, ly=9.0, lz=1.0, hAB=40.0, fA=0.4, ds0=0.1)
    wa = rng.uniform(-60.0, 60.0, (3, 1, 24, 32))
    ref = orc.get_conc(wa, -wa, orc.Params(**kw, batch=3))
    bad = wa.copy()
    bad[1, 0, 5, 7] = np.nan
    with pkg.Context(**kw, batch=3, precision=pkg.PREC_FP64) as c:
        for field, spoilt in ((wa, ()), (bad, (1,))):
            c.set_field(pkg.FIELD_WA, field)
            c.set_field(pkg.FIELD_WB, -wa)
            c.get_conc()
            for b in range(3):
                pha = c.pha.reshape(3, -1)[b]
                if b in spoilt:
                    assert np.isnan(pha).all()
                else:
                    want = ref.pha.reshape(3, -1)[b]
                    assert np.abs(pha - want).max() < 1e-11 * np.abs(want).max()
