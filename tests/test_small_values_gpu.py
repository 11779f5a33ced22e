"""Propagator values far below the largest one: strong fields and deep wells spread a
slice over tens of decades, and every value has to be as good, relative to itself, as
the same passes by FFTs in the working precision leave it.  The reference is the
march with the same gains as dense convolutions in extended precision.

Both sides round each pass at the scale of the line that it filters, the FFT over
log2(n) stages, the integer convolution once on load; the bound is the FFT's own worst
error, three times over (two maxima of the same kind of noise), and the few roundings
that every step takes at a value's own scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PI_REF = 3.1415926535
L = (3.0, 2.7, 2.4)


def gains(n, box, ds):
    i = np.arange(n)
    i = np.where(i <= n // 2 - 1, i, i - n)
    return np.exp(-ds * (2 * PI_REF * i / box) ** 2)


def dense(n, box, ds):
    """K[d] of the filter with these gains, in extended precision, as a matrix."""
    g = gains(n, box, ds).astype(np.longdouble) / n
    m = np.arange(n)
    pi = 4 * np.arctan(np.longdouble(1))
    K = np.cos(2 * pi * (np.outer(m, m) % n).astype(np.longdouble) / n) @ g
    return K[(m[:, None] - m[None, :]) % n]


def march(grid, w, ds, ns, step):
    """q of the chain's end, and every slice before it, per instance."""
    W = [np.exp(-f * ds / 2) for f in w]
    q, out = np.ones_like(w[0]), []
    for f, n in zip((0, 1), ns):
        for _ in range(n):
            q = step(q, W[f])
            out.append(q)
    return out


def exact(grid, w, ds, ns):
    axes = [a for a in range(3) if grid[a] > 1]
    unit = np.prod([np.exp(-ds * (2 * PI_REF / L[a]) ** 2) for a in range(3) if grid[a] == 1])
    K = {a: dense(grid[a], L[a], ds) for a in axes}

    def step(q, W):
        x = q.astype(np.longdouble) * W
        for a in axes:
            x = np.moveaxis(np.tensordot(K[a], x, axes=(1, 3 - a)), 0, 3 - a)
        return x * W * unit
    return march(grid, w, ds, ns, step)


def by_fft(grid, w, ds, ns, real):
    axes = [a for a in range(3) if grid[a] > 1]
    unit = np.prod([np.exp(-ds * (2 * PI_REF / L[a]) ** 2) for a in range(3) if grid[a] == 1])

    def step(q, W):
        x = (q * W.astype(real)).astype(real)
        for a in axes:
            shape = [1, 1, 1, 1]
            shape[3 - a] = grid[a]
            g = (gains(grid[a], L[a], ds) * (unit if a == axes[0] else 1.0)).astype(real)
            f = np.fft.fft(x, axis=3 - a)
            assert f.dtype == (np.complex128 if real == np.float64 else np.complex64)
            x = np.fft.ifft(f * g.reshape(shape), axis=3 - a).real.astype(real)
        return (x * W.astype(real)).astype(real)
    return march(grid, [f.astype(np.float64) for f in w], ds, ns, step)


def fields(kind, grid, batch, prec):
    rng = np.random.default_rng(11)
    shape = (batch, grid[2], grid[1], grid[0])
    if kind == "rough":
        wa = rng.uniform(-60.0, 60.0, shape)
    elif kind == "low":                  # towards the smallest normal numbers and below
        wa, wb = rng.uniform(0.0, 4.0, (2,) + shape)
        wa -= wa.mean(axis=(1, 2, 3), keepdims=True)
        return wa, wb + (1040.0 if prec == 0 else 126.0)
    else:                                # a well, and rough hills around it
        wa = rng.uniform(0.0, 4.0, shape)
        z, y, x = grid[2] // 3, grid[1] // 2, grid[0] // 4
        wa[:, z, y, x] = -200.0 if prec == 0 else -60.0
    wa -= wa.mean(axis=(1, 2, 3), keepdims=True)
    return wa, -0.5 * wa


def worst(a, ref):
    return float(max(np.abs(x / r - 1).max() for x, r in zip(a, ref)))


CASES = [((24, 16, 12), 0, 2), ((64, 12, 10), 0, 1), ((96, 10, 6), 0, 1), ((10, 66, 8), 0, 1),
         ((12, 8, 98), 0, 1), ((34, 62, 1), 0, 2), ((30, 16, 1), 0, 2), ((36, 1, 14), 0, 1), ((130, 8, 6), 0, 1),
         ((30, 20, 14), 1, 2), ((80, 10, 12), 1, 1), ((130, 6, 4), 1, 1), ((30, 16, 1), 1, 1)]


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("kind", ["rough", "well", "low"])
@pytest.mark.parametrize("grid,prec,batch", CASES)
def test_every_value_is_as_good_as_by_ffts(pkg, grid, prec, batch, kind, fused):
    ds, f = (0.1, 0.4) if kind == "rough" else (0.02, 0.3)
    w = fields(kind, grid, batch, prec)
    flags = 0 if fused else pkg.FLAG_NO_FUSED_STEPS
    with pkg.Context(nx=grid[0], ny=grid[1], nz=grid[2], lx=L[0], ly=L[1], lz=L[2], hAB=20.0, fA=f,
                     ds0=ds, batch=batch, precision=prec, flags=flags) as c:
        c.set_w(*w)
        c.get_conc()
        ns = (c.NsA, c.dNsB)
        got = ([c.get_q(pkg.Q_A, s) for s in range(1, ns[0] + 1)] +
               [c.get_q(pkg.Q_B, s) for s in range(1, ns[1] + 1)])
    ref = exact(grid, w, ds, ns)
    fft = by_fft(grid, w, ds, ns, (np.float64, np.float32)[prec])
    eps = (2.0 ** -53, 2.0 ** -24)[prec]
    err, lim = worst(got, ref), worst(fft, ref)
    print("%s %s %s: %.2e, by FFTs %.2e" % (grid, kind, "fused" if fused else "passes", err, lim))
    assert err <= 3 * lim + 4 * eps * np.sqrt(sum(ns))
