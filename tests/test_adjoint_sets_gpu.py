"""The adjoint's independent chains run as sets of launches and its segments
share one buffer, filled from either end in turn (csrc/adjoint.cu): checkpoint
intervals that leave short, single-step and odd last segments change no bit, in
every precision, with trapezoid and Simpson sums, and on every kind of pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(64, 64, 32), (40, 36, 12), (128, 64, 2), (18, 10, 1), (80, 6, 4), (32, 64, 64)]


def gradients(pkg, grid, prec, flags, every, fA=0.4):
    nx, ny, nz = grid
    rng = np.random.default_rng(5)
    with pkg.Context(nx=nx, ny=ny, nz=nz, lx=3.0, ly=2.7, lz=2.5, hAB=15.0, fA=fA, ds0=0.05,
                     precision=prec, flags=flags, batch=2 if nx < 64 else 1) as c:
        wa, wb = rng.normal(0, 1.5, c.shape), rng.normal(0, 1.5, c.shape)
        c.set_w(wa, wb)
        pa, pb = rng.normal(0, 1, c.shape), rng.normal(0, 1, c.shape)
        pa[..., ::3] = 0.0
        return [c.adjoint(pa, pb, 0.3, want_L=k != 7, checkpoint_every=k)[:2] for k in every]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("simpson", [False, True])
def test_intervals_and_precisions(pkg, grid, simpson):
    flags = pkg.FLAG_SIMPSON if simpson else 0
    every = (1, 2, 3, 7, 0, 19, 20)              # 20 steps
    ref = gradients(pkg, grid, pkg.PREC_FP64, flags, every)
    f32 = gradients(pkg, grid, pkg.PREC_FP32, flags, every)
    for runs in (ref, f32):
        for r in runs[1:]:
            assert np.array_equal(r[0], runs[0][0]) and np.array_equal(r[1], runs[0][1])
    # FP32 round-off (6e-8) over 40 dependent steps of up to 20 roundings each
    for a, b in zip(f32[0], ref[0]):
        assert np.abs(a - b).max() < 5e-5 * np.abs(b).max()


@pytest.mark.parametrize("fA", [0.0, 1.0, 0.05])
def test_empty_and_one_step_blocks(pkg, fA):
    a = gradients(pkg, (16, 12, 10), pkg.PREC_FP64, 0, (1, 4), fA=fA)
    assert np.array_equal(a[0][0], a[1][0]) and np.array_equal(a[0][1], a[1][1])
    if fA == 0.0:
        assert not a[0][0].any()
    if fA == 1.0:
        assert not a[0][1].any()
