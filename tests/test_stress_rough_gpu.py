"""Box derivatives in rough fields, whose Boltzmann factors carry every wave number:
FP32 and double-float against the same call in FP64.  The rounding of N contour steps
adds up like a walk; the bound is four times that, 4 sqrt(N) units in the last place of
the working precision, relative to the largest component.  Smooth fields with some
noise, which may take the cheaper form, are held to the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = (3.8, 3.5, 3.2)
EPS = {"fp32": 2.0 ** -24, "df": 2.0 ** -48}


def fields(kind, grid, batch=1):
    rng = np.random.default_rng(3)
    shape = (batch, grid[2], grid[1], grid[0])
    if kind == "rough":
        wa = rng.uniform(-15.0, 15.0, shape)
        return wa, -wa
    x = [2 * np.pi * np.arange(n) / n for n in grid]
    g = (np.sin(x[0])[None, None, :] * np.cos(x[1])[None, :, None] +
         np.sin(x[1])[None, :, None] * np.cos(x[2])[:, None, None])
    r = rng.normal(0, 0.02, (2,) + shape)
    if kind == "edge":                  # about as rough as the cheaper form is taken for
        r *= 3.0
    if kind == "mixed":                 # the first instance smooth, the last one rough
        r[:, -1] *= 500.0
    return 6.0 * g + r[0], -6.0 * g + r[1]


def results(pkg, grid, prec, w, batch, adjoint):
    with pkg.Context(nx=grid[0], ny=grid[1], nz=grid[2], lx=L[0], ly=L[1], lz=L[2], hAB=18.0, fA=0.36,
                     ds0=0.02, batch=batch, precision=prec) as c:
        c.set_w(*w)
        c.get_conc()
        out = [c.stress()]
        if adjoint:
            a, b = c.pha, c.phb         # of one sign: sums without cancellation
            out.append(np.asarray(c.adjoint(a, b, np.full(batch, 0.5), want_L=True)[2]).reshape(batch, 3))
        return out


@pytest.mark.parametrize("grid,batch", [((64, 64, 64), 1), ((128, 64, 32), 1), ((64, 64, 32), 2),
                                        ((64, 64, 1), 2)])
@pytest.mark.parametrize("kind", ["rough", "smooth", "edge", "mixed"])
def test_box_derivatives(pkg, grid, batch, kind):
    if kind == "mixed" and batch == 1:
        pytest.skip("one instance")
    w = fields(kind, grid, batch)
    adjoint = kind == "rough" and grid[2] > 1     # (a film's gradient cancels)
    ref = results(pkg, grid, pkg.PREC_FP64, w, batch, adjoint)
    for name, prec in (("fp32", pkg.PREC_FP32), ("df", pkg.PREC_DF)):
        got = results(pkg, grid, prec, w, batch, adjoint)
        for what, a, b in zip(("stress", "gradient"), got, ref):
            err = (np.abs(a - b).max(axis=1) / np.abs(b).max(axis=1)).max()
            print("%s %s %s %s %.2e" % (grid, kind, name, what, err))
            assert err < 4 * np.sqrt(50) * EPS[name], (name, what)
