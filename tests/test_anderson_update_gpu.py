"""One Anderson field update (csrc/k_anderson.cu) against its formulas in NumPy:
list lengths around the Gram row's and the update's chunks, point counts from
below a block's up, several instances, and values that leave the integer
conversions' range.  Fields and densities are random, so that U's condition
number is about the history's length; the bound is that times the pairs' 2^-48
times the number of terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HAB, LAM, WCMP = 18.0, 0.5, 0.1


def direction(a, c, pa, pb):
    eta, psum = (a + c - HAB) / 2, 1.0 - pa - pb
    d = np.stack([HAB * pb + eta - a - WCMP * psum, HAB * pa + eta - c - WCMP * psum])
    return d - d.reshape(2, -1).mean(axis=1).reshape(2, 1, 1, 1)


def update(ring):
    """w of one instance from its (w, d) pairs, the newest last."""
    u = [w + LAM * d for w, d in ring]
    d = [x[1].ravel() for x in ring][::-1]               # current, c-1, c-2, ...
    n = len(ring) - 1
    g = np.array([[x @ y for y in d] for x in d])
    U = g[0, 0] - g[0, 1:, None] - g[0, None, 1:] + g[1:, 1:]
    U = U + np.eye(n) * (1e-12 * np.abs(np.diag(U)).max() + 1e-300)
    x = np.linalg.solve(U, g[0, 0] - g[0, 1:])
    w = (1 - x.sum()) * u[-1]
    for k in range(n):
        w = w + x[k] * u[-2 - k]
    return w


@pytest.mark.parametrize("grid,hist,batch,scale", [
    ((2, 2, 2), 1, 1, 1.0), ((2, 2, 2), 4, 3, 1.0), ((6, 10, 2), 5, 2, 1.0), ((34, 18, 6), 7, 1, 1.0),
    ((32, 32, 16), 9, 1, 1.0), ((62, 34, 18), 19, 2, 1.0), ((64, 64, 64), 20, 1, 1.0),
    ((40, 36, 30), 30, 1, 1.0), ((32, 16, 16), 6, 1, 1e-25)])
def test_update(pkg, grid, hist, batch, scale):
    nx, ny, nz = grid
    rng = np.random.default_rng(hist)
    with pkg.Context(nx=nx, ny=ny, nz=nz, hAB=HAB, ds0=0.5, batch=batch, precision=pkg.PREC_FP32,
                     mixing=pkg.MIX_ANDERSON, anderson_history=hist, anderson_lambda=LAM,
                     anderson_start=1e9, wopt=0.05, wcmp=WCMP) as c:
        view = {f: c.field_view(f) for f in (pkg.FIELD_WA, pkg.FIELD_WB, pkg.FIELD_PHA, pkg.FIELD_PHB)}
        shape = tuple(view[pkg.FIELD_WA].shape)
        rings = [[] for _ in range(batch)]
        for step in range(hist + 2):                     # the last ones drop the oldest entry
            vals = {}
            for f, v in view.items():
                if f in (pkg.FIELD_PHA, pkg.FIELD_PHB) or step == 0:
                    x = rng.normal(0, 1, shape)
                    if f in (pkg.FIELD_PHA, pkg.FIELD_PHB):
                        x = 0.5 + x * scale              # tiny: d is left of a cancellation
                    else:
                        x *= scale
                    x[..., 0] = x[..., -1]
                    v.copy_(torch.from_numpy(x))
                vals[f] = v.cpu().numpy().reshape((batch, nz, ny, nx)).copy()
            torch.cuda.synchronize()
            for b in range(batch):
                a, w = vals[pkg.FIELD_WA][b], vals[pkg.FIELD_WB][b]
                rings[b].append((np.stack([a, w]),
                                 direction(a, w, vals[pkg.FIELD_PHA][b], vals[pkg.FIELD_PHB][b])))
            c.phi_w()
            c.synchronize()
            if step == 0 or scale != 1.0:
                continue
            got = np.stack([view[f].cpu().numpy().reshape((batch, nz, ny, nx))
                            for f in (pkg.FIELD_WA, pkg.FIELD_WB)], axis=1)
            for b in range(batch):
                if step > hist:
                    rings[b].pop(0)
                want = update(rings[b])
                bound = 4e-15 * 16 * (hist + 1) ** 2
                assert np.abs(got[b] - want).max() < bound * max(1.0, np.abs(want).max()), step
        assert np.isfinite(view[pkg.FIELD_WA].cpu().numpy()).all()
