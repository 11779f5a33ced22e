"""Batched marches of FP32 films: a film has no pass after its x and y ones, so
nothing but those can apply the factor that closes a step.  Members without fused
steps share a march from two on, fused ones once their launches fill the device
(153 films of 16 x 16); every member against its solo run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,n,fused", [((16, 16, 1), 2, False), ((32, 32, 1), 2, False),
                                          ((30, 24, 1), 3, False), ((16, 16, 1), 153, True)])
def test_film_members_match_their_solo_runs(pkg, grid, n, fused):
    from scft_gb300 import fields
    nx, ny, nz = grid
    flags = 0 if fused else pkg.FLAG_NO_FUSED_STEPS
    members = [dict(nx=nx, ny=ny, nz=nz, lx=3.0 + 0.01 * i, ly=3.2, lz=1.0, hAB=14.0 + i % 7,
                    fA=0.3 + 0.02 * (i % 5), ds0=1.0 / (40 + 3 * (i % 4)), flags=flags,
                    precision=pkg.PREC_FP32) for i in range(n)]
    start = [fields.gyroid(nx, ny, nz, m["lx"], m["ly"], m["lz"], m["hAB"], seed=i)
             for i, m in enumerate(members)]
    ctxs = [pkg.Context(**m) for m in members]
    for c, w in zip(ctxs, start):
        c.set_w(*w)
    with pkg.Group(ctxs) as g:
        g.iterate(2)
    for c, m, w in zip(ctxs, members, start):
        with pkg.Context(**m) as solo:
            solo.set_w(*w)
            solo.iterate(2)
            wa, pha = solo.wa, solo.pha
        # FP32 round-off (6e-8) of two schedules over up to 98 dependent steps
        assert np.abs(c.wa - wa).max() < 2e-5 * np.abs(wa).max()
        assert np.abs(c.pha - pha).max() < 2e-5 * np.abs(pha).max()
        c.close()
