"""The fixed-point nonlinear pass on the device: every class of transform
length and kernel form (lines per block and warps per line change with the
number and length of the lines), extreme magnitudes, non-finite lines, and
the grids of exactly 3 Nm points that a variable time step reads its velocity
maxima on.

The reference is a long-double FFT of the 3 Nm-point grid.  Tolerance against
it, relative to a product's norm over the line: the transforms' own error
(2^-52.8 each way, tests/test_fixed_point_fft.py, three transforms meet in a
product), the products' and outputs' rounding and the inputs' 2^-59: below 6 x
2^-52.8 < 1.0e-15."""
import numpy as np
import pytest
import scipy.fft

pytestmark = pytest.mark.gpu


def reference(nm, t, w, up, ur):
    p = 3 * nm
    g = [scipy.fft.irfft(np.asarray(x, np.clongdouble), n=p, axis=1, norm="forward") for x in (t, w, up, ur)]
    return [scipy.fft.rfft(a * b, axis=1, norm="forward")[:, :nm + 1]
            for a, b in ((g[2], g[0]), (g[3], g[0]), (g[2], g[1]), (g[3], g[1]))]


def fields(rng, nr, nm, scales=(1.0, 1e3, 1e2, 1e-3)):
    decay = np.exp(-6.0 * np.arange(nm + 1) / nm)
    out = [(rng.standard_normal((nr, nm + 1)) + 1j * rng.standard_normal((nr, nm + 1))) * decay * s for s in scales]
    for x in out:
        x[:, 0] = x[:, 0].real
    return out


def errors(got, ref):
    return [float(np.max(np.linalg.norm((g - r).astype(np.clongdouble), axis=1) /
                         np.maximum(np.linalg.norm(r, axis=1), np.finfo(float).tiny))) for g, r in zip(got, ref)]


# 40 lines: 8 warps a line; 330 lines: the forms of short, middle and long lines
@pytest.mark.parametrize("nr", [40, 330])
@pytest.mark.parametrize("nm", [1, 2, 3, 5, 10, 14, 21, 32, 42, 61, 85, 100, 128, 170, 209, 220, 256, 341, 384, 385,
                                512, 1365])
def test_lengths_and_forms(fg, nm, nr):
    ins = fields(np.random.default_rng(nm), nr, nm)
    rows = np.arange(nr % 11, nr, 11)  # the reference's long doubles are slow
    got = [g[rows] for g in fg.nonlin(nm, *ins)]
    assert max(errors(got, reference(nm, *[x[rows] for x in ins]))) < 1.0e-15


@pytest.mark.parametrize("nb", [1, 3, 61])
def test_batch_lines_equal_single_instances(fg, nb):
    """A line's result depends on that line only: a batch (odd sizes leave a
    block with fewer lines than it holds) equals its instances alone."""
    import torch
    nr, nm = 7, 42
    cols = [fields(np.random.default_rng(b), nr, nm) for b in range(nb)]
    dev = [torch.from_numpy(np.ascontiguousarray(np.stack([c[f] for c in cols], axis=-1))).cuda() for f in range(4)]
    outs = [torch.full_like(dev[0], float("nan")) for _ in range(4)]
    fg.check(fg.lib().falcon_nonlin_dev(nr, nm, nb, *[x.data_ptr() for x in dev + outs],
                                        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for b in range(nb):
        alone = fg.nonlin(nm, *cols[b])
        for o, q in zip(outs, alone):
            assert np.array_equal(o[:, :, b].cpu().numpy(), q)


@pytest.mark.parametrize("scales", [(1e-150, 1e-160, 1e-150, 1e-140), (1e140, 1e150, 1e150, 1e148),
                                    (1e-300, 1e300, 1e-200, 1e200), (5e-310, 1.0, 1e10, 1e-300)])
def test_magnitudes(fg, scales):
    nr, nm = 6, 42
    ins = fields(np.random.default_rng(7), nr, nm, scales)
    got, ref = fg.nonlin(nm, *ins), reference(nm, *ins)
    for g, r in zip(got, ref):
        if np.max(np.abs(r)) > np.finfo(float).max:  # beyond the doubles
            assert not np.isfinite(g).all()
            continue
        # a product below the normal numbers keeps their absolute spacing; fields
        # of subnormal numbers carry 2^-1074 each
        tol = 1e-15 * np.linalg.norm(r, axis=1) + 2.0 ** -1070 * (nm + 1)
        if min(scales) < 1e-305:
            tol = tol + 1e-12 * np.linalg.norm(r, axis=1)
        assert np.all(np.linalg.norm((g - r).astype(np.clongdouble), axis=1) <= tol)


def test_zero_and_single_mode_fields(fg):
    nr, nm = 5, 85
    t, w, up, ur = (np.zeros((nr, nm + 1), np.complex128) for _ in range(4))
    t[1, 3] = 0.25 + 0.5j
    w[2, 85] = 1e3 - 7j
    up[1:, 1] = 1.0 + 2.0j
    ur[1:, 85] = -3.0 + 1e-3j
    got, ref = fg.nonlin(nm, t, w, up, ur), reference(nm, t, w, up, ur)
    for g, r in zip(got, ref):
        assert np.all(np.linalg.norm((g - r).astype(np.clongdouble), axis=1) <= 1e-15 * np.linalg.norm(r, axis=1))
    assert all(np.all(g[0] == 0.0) for g in got)


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("field", [0, 1, 2, 3])
def test_nonfinite_lines_give_nan_and_stay_alone(fg, field, value):
    nr, nm = 9, 42
    ins = fields(np.random.default_rng(3), nr, nm)
    clean = fg.nonlin(nm, *ins)
    ins[field][4, 5] = value
    got = fg.nonlin(nm, *ins)
    for g, c in zip(got, clean):
        assert np.isnan(g[4].real).all() and np.isnan(g[4].imag).all()
        keep = np.arange(nr) != 4
        assert np.array_equal(g[keep], c[keep])


def test_overflowing_products_are_not_finite(fg):
    ins = fields(np.random.default_rng(4), 3, 42, (1e200, 1e200, 1e200, 1e200))
    assert not any(np.isfinite(g).any() for g in fg.nonlin(42, *ins))


# 3 Nm = 30 (6 x 5), 33, 39, 51 (radix 11, 13, 17 on the tensor cores), 57, 69,
# 87, 93 (19, 23, 29, 31), 48, 63 (twiddled), 99, 132, 111 (11, 11, 37 twiddled)
@pytest.mark.parametrize("nm", [10, 11, 13, 17, 19, 23, 29, 31, 16, 21, 33, 44, 37])
def test_variable_dt_reads_the_maxima_of_its_own_grid(fg, orc, nm):
    kw = dict(ra=1e6, dt=1e-5, vartimestep=True, cfl=0.3, dt_max=1e-4)
    p = fg.make_params(17, nm, "SBDF2", **kw)
    g, o = fg.Instance(p), orc.Sim(orc.make_params(17, nm, "SBDF2", **kw))
    g.init_noise(5, 1e-1)
    o.init_noise(5, 1e-1)
    for _ in range(6):
        g.step(1)
        o.step(1)
        assert abs(g.diagnostics()["dt"] - o.dt) <= 1e-12 * o.dt
    a, b = g.get_state(), o.get_state()
    for k in ("T", "omg", "up", "ur"):
        assert np.linalg.norm(a[k] - b[k]) < 1e-10 * np.linalg.norm(b[k])
    g.close()
