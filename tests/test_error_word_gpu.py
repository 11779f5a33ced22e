"""Every call that waits for the device reports a kernel that gave up a bounded
wait, and clears the word, so that no later call is blamed for it.  The word is
set from the host (scft_selftest_set_error): nothing hangs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(nx=16, ny=8, nz=4, lx=3.0, ly=2.0, lz=1.5, hAB=18.0, fA=0.5, ds0=0.1)


@pytest.fixture
def ctx(pkg):
    from scft_gb300 import fields
    with pkg.Context(**KW) as c:
        c.set_w(*fields.gyroid(16, 8, 4, 3.0, 2.0, 1.5, 18.0, seed=1))
        c.get_conc()
        c.synchronize()
        yield c


CALLS = {
    "adjoint": lambda c, tmp: c.adjoint(np.ones(c.shape), np.ones(c.shape), np.ones(1)),
    "stress": lambda c, tmp: c.stress(),
    "get_q": lambda c, tmp: c.get_q(0, 1),
    "get_Q": lambda c, tmp: c.Q(),
    "time_iterations": lambda c, tmp: c.time_iterations(1),
    "synchronize": lambda c, tmp: c.synchronize(),
    "write_pha_dat": lambda c, tmp: c.write_pha_dat(str(tmp / "pha.dat")),
    "write_vtk": lambda c, tmp: c.write_vtk(str(tmp / "pha.vtk")),
    "save_checkpoint": lambda c, tmp: c.save_checkpoint(str(tmp / "ckpt")),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_call_reports_the_word(pkg, ctx, name, tmp_path):
    assert ctx.lib.scft_selftest_set_error(ctx.h, 2) == pkg.OK
    with pytest.raises(pkg.ScftError) as e:
        CALLS[name](ctx, tmp_path)
    assert e.value.status == pkg.ERR_CUDA and "error word 2" in str(e.value)
    # propagators that cannot be trusted are not used, and the word is gone
    with pytest.raises(pkg.ScftError) as e:
        ctx.stress()
    assert e.value.status == pkg.ERR_INVALID_ARG
    ctx.get_conc()
    CALLS[name](ctx, tmp_path)


@pytest.mark.parametrize("member", [0, 1, 2])
@pytest.mark.parametrize("timed", [False, True])
def test_group_reports_any_member(pkg, member, timed):
    from scft_gb300 import fields
    ctxs = [pkg.Context(**KW, precision=pkg.PREC_FP32, flags=pkg.FLAG_NO_FUSED_STEPS) for _ in range(2)]
    ctxs.append(pkg.Context(**KW))
    for i, c in enumerate(ctxs):
        c.set_w(*fields.gyroid(16, 8, 4, 3.0, 2.0, 1.5, 18.0, seed=i))
    with pkg.Group(ctxs) as g:
        call = (lambda: g.time_iterations(1)) if timed else (lambda: g.iterate(1))
        call()
        assert ctxs[member].lib.scft_selftest_set_error(ctxs[member].h, 2) == pkg.OK
        with pytest.raises(pkg.ScftError) as e:
            call()
        assert e.value.status == pkg.ERR_CUDA and "error word 2" in str(e.value)
        with pytest.raises(pkg.ScftError):
            ctxs[1].stress()
        call()
        for c in ctxs:
            c.synchronize()
    for c in ctxs:
        c.close()
