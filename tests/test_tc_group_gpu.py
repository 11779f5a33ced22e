"""Groups of members on the tensor cores: a bucket's batched march on whole planes
(four of 40^3) and pass by pass (planes that would not pay, and lines above 64
points), and members that keep their own marches, against their solo runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,n", [((40, 40, 40), 4), ((12, 20, 28), 12), ((80, 10, 20), 5),
                                    ((20, 20, 20), 2)])
def test_members_match_their_solo_runs(pkg, grid, n):
    from scft_gb300 import fields
    nx, ny, nz = grid
    members = [dict(nx=nx, ny=ny, nz=nz, lx=3.0 + 0.1 * i, ly=3.2, lz=2.8, hAB=14.0 + i, fA=0.3 + 0.01 * i,
                    ds0=1.0 / (40 + 3 * i), precision=pkg.PREC_FP32) for i in range(n)]
    start = [fields.gyroid(nx, ny, nz, m["lx"], m["ly"], m["lz"], m["hAB"], seed=i)
             for i, m in enumerate(members)]
    solo = []
    for m, w in zip(members, start):
        with pkg.Context(**m) as c:
            c.set_w(*w)
            c.iterate(4)
            solo.append((c.wa, c.pha))
    ctxs = [pkg.Context(**m) for m in members]
    for c, w in zip(ctxs, start):
        c.set_w(*w)
    with pkg.Group(ctxs) as g:
        g.iterate(4)
    for c, (wa, pha) in zip(ctxs, solo):
        # FP32 round-off (6e-8) of two schedules over up to 150 dependent steps
        assert np.abs(c.wa - wa).max() < 2e-5 * np.abs(wa).max()
        assert np.abs(c.pha - pha).max() < 2e-5 * np.abs(pha).max()
        c.close()
