"""FP64 plane transforms on the integer pipe (fft_int_rows.cu, fft_int_cols.cu)
at every length they are instantiated for, against the same transforms in
extended precision.

Tolerances, relative L2 over the planes, set before the first run: a pass
rounds its result to FP64 once (2^-53 of each value at most) and carries an
error of at most a few units of 2^-55 of the row's largest value, so one plane
transform (two passes) stays below 4 x 2^-53 = 4.4e-16 and a round trip with
its derivative below 8 x 2^-53.
"""
import numpy as np
import pytest

import les_gb300 as lg

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53

# (nx, ny): x half lengths 16..192 of the small and 3/2 grids, y lengths 16..384
GRIDS = [(32, 16), (48, 24), (72, 36), (64, 32), (96, 48), (144, 72), (128, 64), (192, 96), (256, 128), (216, 108),
         (32, 144), (36, 192), (144, 216), (64, 256), (256, 288), (128, 384)]


def rel(a, b):
    a, b = a.astype(np.clongdouble), b.astype(np.clongdouble)
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.fixture(scope="module")
def ctx_of(gpu_lib):
    made = {}

    def get(nx, ny):
        if (nx, ny) not in made:
            cfg = lg.make_config(nx, ny, 4, rmsdiv_every=0)
            made[nx, ny] = lg.Context(cfg, lg.uniform_surface(cfg))
        return made[nx, ny]
    yield get
    for c in made.values():
        c.close()


def planes(kind, n, ny, nx, seed):
    """Values the path meets: a mean with small fluctuations, white noise, a single point, a steep field."""
    g = np.random.default_rng(seed)
    if kind == "wind":
        return 13.0 + 0.1 * g.standard_normal((n, ny, nx))
    if kind == "point":
        f = np.zeros((n, ny, nx))
        f[:, ny // 3, nx // 5] = 1.7
        return f
    if kind == "steep":
        f = g.standard_normal((n, ny, nx))
        return f * np.exp(-np.arange(nx) / 3.0)[None, None, :]
    if kind == "ridge":  # each column of the y pass is one row and little else
        f = g.standard_normal((n, ny, nx))
        return f * np.exp(-np.arange(ny) / 3.0)[None, :, None]
    return g.standard_normal((n, ny, nx))


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("kind", ["wind", "noise", "point", "steep", "ridge"])
def test_plane_transforms(ctx_of, nx, ny, kind):
    c = ctx_of(nx, ny)
    for big in (0, 1):
        mx, my = (3 * nx // 2, 3 * ny // 2) if big else (nx, ny)
        f = planes(kind, 3, my, mx, nx + ny)
        want = np.fft.rfft2(f.astype(np.longdouble))
        a = np.zeros((3, my, mx + 2))
        a[:, :, :mx] = f
        c.call("fft_r2c", a, ints=(3, big))
        assert rel(a.view(np.complex128), want) < 4 * EPS
        # back from the rounded spectrum: the exact inverse of what the routine is given
        h = a.view(np.complex128).astype(np.clongdouble)
        back = np.fft.irfft2(h, s=(my, mx)) * (mx * my)
        c.call("fft_c2r", a, ints=(3, big))
        assert rel(a[:, :, :mx], back) < 4 * EPS


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_roundings_do_not_meet(ctx_of, nx, ny):
    """No point of a plane collects the others' roundings.  White noise: every error is a sum of many roundings, close
    to normal, so that none of the up to 300,000 values lies beyond 6 of their deviations, 8 with the spread of the
    scales from row to row; the values at zero, which all coherent errors reach, are among them."""
    c = ctx_of(nx, ny)
    for big in (0, 1):
        mx, my = (3 * nx // 2, 3 * ny // 2) if big else (nx, ny)
        f = planes("noise", 2, my, mx, 3 * nx + ny)
        want = np.fft.rfft2(f.astype(np.longdouble))
        a = np.zeros((2, my, mx + 2))
        a[:, :, :mx] = f
        c.call("fft_r2c", a, ints=(2, big))
        h = a.view(np.complex128).astype(np.clongdouble)
        err = np.abs(h - want).astype(np.float64)
        assert err.max() < 8 * max(np.sqrt((err ** 2).mean()), EPS * np.sqrt((np.abs(want) ** 2).mean()))
        back = np.fft.irfft2(h, s=(my, mx)) * (mx * my)
        c.call("fft_c2r", a, ints=(2, big))
        err = np.abs(a[:, :, :mx] - back).astype(np.float64)
        assert err.max() < 8 * max(np.sqrt((err ** 2).mean()), EPS * float(np.sqrt((back ** 2).mean())))


@pytest.mark.parametrize("nx,ny,big", [(256, 256, 1), (256, 128, 1), (384, 256, 0), (192, 256, 1)])
def test_inverse_of_flat_spectrum(ctx_of, nx, ny, big):
    """A single point's spectrum, where the sum of moduli that sets the scale of a row is farthest above its values: no
    further from the exact inverse than FP64 butterflies, 1.7 to 2.3 x 2^-53 in these planes."""
    c = ctx_of(nx, ny)
    mx, my = (3 * nx // 2, 3 * ny // 2) if big else (nx, ny)
    h = np.fft.rfft2(planes("point", 2, my, mx, 0))
    a = np.zeros((2, my, mx + 2))
    a.view(np.complex128)[...] = h
    want = np.fft.irfft2(h.astype(np.clongdouble), s=(my, mx)) * (mx * my)
    c.call("fft_c2r", a, ints=(2, big))
    assert rel(a[:, :, :mx], want) < 1.7 * EPS


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_derivatives_and_filter(ctx_of, nx, ny):
    c = ctx_of(nx, ny)
    f = planes("wind", 2, ny, nx, 5 * nx + ny)
    h = np.fft.rfft2(f.astype(np.longdouble))
    h[:, ny // 2, :] = 0
    h[:, :, -1] = 0
    kx = np.arange(nx // 2 + 1).astype(np.longdouble)[None, None, :]
    ky = (((np.arange(ny) + ny // 2) % ny) - ny // 2).astype(np.longdouble)[None, :, None]
    a = np.zeros((2, ny, nx + 2))
    a[:, :, :nx] = f
    dx, dy = np.zeros_like(a), np.zeros_like(a)
    c.call("filt_da", a, dx, dy, ints=(2,))
    want = np.fft.irfft2(h, s=(ny, nx))
    assert rel(a[:, :, :nx], want) < 8 * EPS
    # derivatives of wind + noise: the error is that of the largest value transformed times the wavenumber
    scale = np.linalg.norm(want) * float(max(nx, ny)) / 2
    for got, k in ((dx, kx), (dy, ky)):
        w = np.fft.irfft2(1j * k * h, s=(ny, nx))
        assert np.linalg.norm((got[:, :, :nx].astype(np.longdouble) - w).ravel()) < 8 * EPS * scale
        assert np.all(got[:, :, nx:] == 0.0)


@pytest.mark.parametrize("nx,ny", [(32, 16), (48, 24), (64, 32), (96, 48), (144, 72), (128, 64), (192, 96), (256, 128),
                                   (32, 144), (36, 192), (64, 256)])
def test_padding_and_truncation(ctx_of, nx, ny):
    c = ctx_of(nx, ny)
    mx, my = 3 * nx // 2, 3 * ny // 2
    f = planes("noise", 2, ny, nx, 7 * nx + ny)
    h = np.fft.rfft2(f.astype(np.longdouble)) / (nx * ny)
    h[:, ny // 2, :] = 0
    h[:, :, -1] = 0
    hb = np.zeros((2, my, mx // 2 + 1), dtype=np.clongdouble)
    hb[:, :ny // 2, :nx // 2] = h[:, :ny // 2, :nx // 2]
    hb[:, my - ny // 2 + 1:, :nx // 2] = h[:, ny // 2 + 1:, :nx // 2]
    want = np.fft.irfft2(hb, s=(my, mx)) * (mx * my)
    a, big, back = np.zeros((2, ny, nx + 2)), np.zeros((2, my, mx + 2)), np.zeros((2, ny, nx + 2))
    a[:, :, :nx] = f
    c.call("dealias1", a, big, ints=(2,))
    assert rel(big[:, :, :mx], want) < 8 * EPS
    c.call("dealias2", back, big, ints=(2,))
    assert rel(back[:, :, :nx], np.fft.irfft2(h, s=(ny, nx)) * (nx * ny)) < 16 * EPS


@pytest.mark.parametrize("nx,ny", [(64, 32), (96, 48), (256, 256)])
def test_range_ends(ctx_of, nx, ny):
    """Zero planes, values near both ends of the FP64 range, and not-a-number or infinity in one plane of several."""
    c = ctx_of(nx, ny)
    g = np.random.default_rng(3)
    f = g.standard_normal((2, ny, nx))
    want = np.fft.rfft2(f.astype(np.longdouble))
    for scale in (2.0 ** -1010, 2.0 ** -900, 2.0 ** 900, 2.0 ** 1000):
        a = np.zeros((2, ny, nx + 2))
        a[:, :, :nx] = f * scale
        c.call("fft_r2c", a, ints=(2, 0))
        got = a.view(np.complex128).astype(np.clongdouble) / np.longdouble(scale)
        # 2^-1010: sums of a few hundred such values; their last bits are subnormal units of 2^-1074
        tol = 4 * EPS if scale > 2.0 ** -1000 else 2.0 ** -50
        assert rel(got, want) < tol
    a = np.zeros((3, ny, nx + 2))
    c.call("fft_r2c", a, ints=(3, 0))
    assert np.all(a == 0.0)
    for bad in (np.nan, np.inf, -np.inf):
        a = np.zeros((3, ny, nx + 2))
        a[0, :, :nx], a[2, :, :nx] = f[0], f[1]
        a[1, 3, 5] = bad
        c.call("fft_r2c", a, ints=(3, 0))
        s = a.view(np.complex128)
        assert not np.any(np.isfinite(s[1].real)) and np.all(np.isfinite(s[[0, 2]]))
        assert rel(s[[0, 2]], want) < 4 * EPS


@pytest.mark.parametrize("nx,ny", GRIDS + [(32, 288), (64, 384)])
@pytest.mark.parametrize("amp", [1.01, 1.45, 1.99])
def test_alternating_rows(ctx_of, nx, ny, amp):
    """Fields that change sign from row to row: all the filter removes, at mantissas of both ends of a binade.

    The filter leaves f less its alternating sums, in units of the field: a few roundings of f, 8 x 2^-53 of its norm;
    its derivatives the same times the largest wavenumber."""
    c = ctx_of(nx, ny)
    alt = (-1.0) ** np.arange(ny)
    low = 0.25 * np.cos(2 * np.pi * np.arange(nx) / nx)
    f = np.empty((3, ny, nx))
    f[0] = amp * alt[:, None]
    f[1] = -amp * alt[:, None] * (1.0 + low / 1024)[None, :]
    f[2] = f[0] + 0.125 * (low[None, :] + np.sin(2 * np.pi * np.arange(ny) / ny)[:, None])
    h = np.fft.rfft2(f.astype(np.longdouble))
    h[:, ny // 2, :] = 0
    h[:, :, -1] = 0
    kx = np.arange(nx // 2 + 1).astype(np.longdouble)[None, None, :]
    ky = (((np.arange(ny) + ny // 2) % ny) - ny // 2).astype(np.longdouble)[None, :, None]
    norm = np.linalg.norm(f.ravel())
    kmax = max(nx, ny) / 2
    a, a2 = np.zeros((3, ny, nx + 2)), np.zeros((3, ny, nx + 2))
    a[:, :, :nx] = f
    a2[:, :, :nx] = f
    dx, dy, dx2, dy2 = (np.zeros_like(a) for _ in range(4))
    c.call("filt_da", a, dx, dy, ints=(3,))
    c.call("ddxy", dx2, dy2, a2, ints=(3,))
    for got, k, s in ((a, 1, 1), (dx, 1j * kx, kmax), (dy, 1j * ky, kmax), (dx2, 1j * kx, kmax), (dy2, 1j * ky, kmax)):
        want = np.fft.irfft2(k * h, s=(ny, nx))
        assert np.linalg.norm((got[:, :, :nx] - want).astype(np.float64).ravel()) < 8 * EPS * s * norm


@pytest.mark.parametrize("nx,ny", [(48, 64), (64, 48), (96, 72), (144, 128), (256, 36), (384, 16)])
def test_pressure_gradient_of_a_large_mean(ctx_of, nx, ny):
    """A uniform divtz at the lower wall moves the plane mean of p and nothing else: every other mode, and so the
    gradient, keeps its bits, whatever the mean's size."""
    c = ctx_of(nx, ny)
    shape = lg.config.field_shape(c.cfg, "u")
    g = np.random.default_rng(nx * ny)
    for nm in ("u", "v", "w"):
        f = np.zeros(shape)
        f[:, :, :nx] = 0.1 * g.standard_normal((shape[0], ny, nx))
        c.set(nm, f)
    got = {}
    for mean in (0.0, 2.0 ** 40):
        d = np.zeros(shape)
        d[0, :, :nx] = mean
        c.set("divtz", d)
        p, x, y = np.zeros(lg.config.field_shape(c.cfg, "p")), np.zeros(shape), np.zeros(shape)
        c.call("press_stag_array", p, x, y)
        got[mean] = (p[1:c.cfg.nz, :, :nx], x[:-1, :, :nx], y[:-1, :, :nx])
    assert np.min(np.abs(got[2.0 ** 40][0])) > 2.0 ** 30 and np.max(np.abs(got[0.0][0])) < 2.0 ** 20
    for a, b in zip(got[0.0][1:], got[2.0 ** 40][1:]):
        assert np.any(a != 0.0) and np.array_equal(a, b)


@pytest.mark.parametrize("nx,ny", [(64, 32), (96, 48), (256, 256), (384, 16)])
def test_range_ends_of_every_pass(ctx_of, nx, ny):
    """Values near both ends of the FP64 range through the filter, the derivatives, the 3/2 round trip and a divergence:
    every pass scales by powers of two, so the results are those at scale 1, times the scale."""
    c = ctx_of(nx, ny)
    nz = c.cfg.nz
    g = np.random.default_rng(9)
    f = g.standard_normal((nz, ny, nx))
    t = g.standard_normal((nz, ny, nx))
    mx, my = 3 * nx // 2, 3 * ny // 2

    def run(scale):
        pad = lambda a: np.concatenate([a * scale, np.zeros((nz, ny, 2))], axis=2)
        a, b, z = pad(f), pad(t), np.zeros((nz, ny, nx + 2))
        out = [a.copy()] + [np.zeros_like(a) for _ in range(6)]
        c.call("filt_da", out[0], out[1], out[2], ints=(nz,))
        c.call("ddxy", out[3], out[4], a, ints=(nz,))
        c.call("divstress_uv", out[5], a, b, z)
        big = np.zeros((nz, my, mx + 2))
        c.call("dealias1", a, big, ints=(nz,))
        c.call("dealias2", out[6], big, ints=(nz,))
        # the top level of a divergence is a constant
        return [q[:nz - 1, :, :nx].astype(np.longdouble) / np.longdouble(scale) for q in out] + \
            [big[:nz - 1, :, :mx].astype(np.longdouble) / np.longdouble(scale)]

    want = run(1.0)
    for scale in (2.0 ** -1005, 2.0 ** -980, 2.0 ** -900, 2.0 ** 900, 2.0 ** 990):
        for i, (a, b) in enumerate(zip(run(scale), want)):
            # the spectra carry 1/(nx ny): at the smallest scales their last bits are subnormal units of 2^-1074
            assert rel(a, b) < (8 * EPS if scale > 2.0 ** -1000 else 2.0 ** -46), (scale, i)


@pytest.mark.parametrize("nx,ny", [(64, 32), (96, 48), (256, 256)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_a_number_through_every_pass(ctx_of, nx, ny, bad):
    """Not-a-number or infinity in one plane: none of that plane is finite, all other planes keep their bits."""
    c = ctx_of(nx, ny)
    nz = c.cfg.nz
    g = np.random.default_rng(10)
    f, t = np.zeros((nz, ny, nx + 2)), np.zeros((nz, ny, nx + 2))
    f[:, :, :nx] = g.standard_normal((nz, ny, nx))
    t[:, :, :nx] = g.standard_normal((nz, ny, nx))
    mx, my = 3 * nx // 2, 3 * ny // 2

    def run(a, b):
        out = [a.copy()] + [np.zeros_like(a) for _ in range(6)]
        c.call("filt_da", out[0], out[1], out[2], ints=(nz,))
        c.call("ddxy", out[3], out[4], a, ints=(nz,))
        c.call("divstress_uv", out[5], a, b, np.zeros_like(a))
        big = np.zeros((nz, my, mx + 2))
        c.call("dealias1", a, big, ints=(nz,))
        c.call("dealias2", out[6], big, ints=(nz,))
        return [q[:, :, :nx] for q in out] + [big[:, :, :mx]]

    want = run(f, t)
    for which in (0, 1):
        a, b = f.copy(), t.copy()
        (a, b)[which][1, 3, 5] = bad
        got = run(a, b)
        for i, (q, w) in enumerate(zip(got, want)):
            others = [k for k in range(nz) if k != 1]
            assert np.array_equal(q[others], w[others]), i
            if which == 0 or i == 5:
                assert not np.any(np.isfinite(q[1])), i
            else:
                assert np.array_equal(q[1], w[1]), i
