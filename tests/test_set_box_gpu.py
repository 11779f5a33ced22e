"""A new box rewrites a context's tables in place, under its captured graphs and
those of a group: the next call must see them.  A box so short that an axis's box
derivatives are near underflow has no tensor-core table: that axis goes back to its
FFT pass, the graphs are captured anew, and the old box brings the first kernels
back."""
import numpy as np
import pytest

from oracle import scft_oracle as orc

pytestmark = pytest.mark.gpu

DS = 0.05
SHORT = 0.0546      # ds k^2 = 662: a derivative's largest gain is below 2^-900


def start(grid, batch=1, seed=3):
    from scft_gb300 import fields
    return fields.gyroid(*grid, 3.0, 2.7, 2.4, 18.0, seed=seed, batch=batch)


def params(grid, box, batch=1):
    return dict(nx=grid[0], ny=grid[1], nz=grid[2], lx=box[0], ly=box[1], lz=box[2], hAB=18.0,
                fA=0.36, ds0=DS, batch=batch)


def conc(c, w):
    c.set_w(*w)
    c.get_conc()
    return c.pha, c.phb, c.Q()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("grid,prec", [((24, 20, 18), 0), ((96, 10, 14), 0), ((40, 34, 1), 0),
                                       ((30, 16, 1), 0), ((64, 32, 32), 0), ((130, 16, 12), 0),
                                       ((30, 20, 14), 1), ((80, 10, 20), 1), ((100, 64, 64), 1),
                                       ((30, 16, 1), 1)])
def test_axis_without_a_table(pkg, grid, prec, axis):
    if grid[axis] == 1:
        pytest.skip("no pass along this axis")
    box = [3.0, 2.7, 2.4]
    short = list(box)
    short[axis] = SHORT
    w, tol = start(grid), (1e-12, 5e-6)[prec]
    with pkg.Context(**params(grid, box), precision=prec) as c:
        first = conc(c, w)
        for _ in range(2):
            c.set_box(*short)
            got = conc(c, w)
            ref = orc.get_conc(*w, orc.Params(**params(grid, short)))
            for a, b in zip(got, (ref.pha, ref.phb, ref.Q)):
                assert np.abs(a / b - 1).max() < tol
            assert np.isfinite(c.stress()).all()
            c.set_box(*box)
            for a, b in zip(conc(c, w), first):
                assert np.array_equal(a, b)


@pytest.mark.parametrize("grid,prec", [((60, 60, 60), 0), ((128, 64, 32), 0), ((128, 64, 32), 1),
                                       ((100, 80, 60), 1), ((64, 64, 64), 2), ((200, 6, 4), 0)])
def test_next_call_sees_the_new_box(pkg, grid, prec):
    w = start(grid)
    boxes = [[3.0, 2.7, 2.4], [4.4, 3.1, 5.2]]
    want = []
    for box in boxes:
        with pkg.Context(**params(grid, box), precision=prec) as c:
            want.append(conc(c, w))
    with pkg.Context(**params(grid, boxes[0]), precision=prec) as c:
        for k in range(6):
            c.set_w(*w)
            c.set_box(*boxes[k % 2])
            c.get_conc()
            for a, b in zip((c.pha, c.phb, c.Q()), want[k % 2]):
                assert np.array_equal(a, b)


@pytest.mark.parametrize("grid,n", [((40, 40, 40), 4), ((80, 10, 20), 5), ((20, 20, 20), 2)])
def test_group_member_without_a_table(pkg, grid, n):
    """One member of a batched march loses an axis's table and gets it back."""
    ctxs, ws = [], []
    for i in range(n):
        ctxs.append(pkg.Context(**params(grid, [3.0, 2.7, 2.4]), precision=pkg.PREC_FP32))
        ws.append(start(grid, seed=i))
    solo = pkg.Context(**params(grid, [3.0, 2.7, 2.4]), precision=pkg.PREC_FP32)
    with pkg.Group(ctxs) as g:
        for lx in (3.0, SHORT, 3.0):
            ctxs[1].set_box(lx, 2.7, 2.4)
            for c, w in zip(ctxs, ws):
                c.set_w(*w)
            g.iterate(2)
            for i, (c, w) in enumerate(zip(ctxs, ws)):
                solo.set_box(lx if i == 1 else 3.0, 2.7, 2.4)
                solo.set_w(*w)
                solo.iterate(2)
                # FP32 round-off (6e-8) of two schedules over 40 dependent steps
                assert np.abs(c.wa - solo.wa).max() < 2e-5 * np.abs(solo.wa).max()
                assert np.abs(c.pha - solo.pha).max() < 2e-5 * np.abs(solo.pha).max()
    for c in ctxs + [solo]:
        c.close()
