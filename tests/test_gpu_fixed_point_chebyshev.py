"""The Chebyshev transforms in fixed point (fx_columns_kernel of
falcon-dns_gb300/csrc/falcon_fxgemm.cu): odd and even sizes around its row
blocks (2, 4, 8, 64, 96, 128 output pairs) and chunks of 8 pairs, its largest
(257) and the dense form past it, column counts around both tiles.

Columns of the identity give the operator as the device holds it.  Random and
falling columns are then compared with that operator times them in extended
precision.  With B_i = sum_k |A_ik| |x_k|, an element read back is off by its
rounding (2^-53) and by the truncation of its row (2^-58 of the row's largest
scaled element), x by 2^-58 of the largest scaled x, a product by 2^-57 (its
low x low part), the sum is rounded once: |error| <= 2^-52 B_i +
4 n 2^-58 max_k |A_ik| 2^-w_k max_k |x_k| 2^w_k, and
n 2^-53 B_i + 2^-53 B_i for the dense form's FP64 sums.  The operators
themselves: the recursions over n degrees lose at most 4 n^2 roundings of an
element bound k^0, k^2, k^4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("falcon_cheb_fwd_dev", "falcon_cheb_inv_dev", "falcon_cheb_d1_dev", "falcon_cheb_d2_dev")


def call(fg, fn, n, x, outs=1):
    import torch
    xin = torch.from_numpy(np.ascontiguousarray(x).view(np.float64)).cuda()
    y = [torch.full_like(xin, 7.0) for _ in range(outs)]
    fg.check(getattr(fg.lib(), fn)(n, x.shape[0], xin.data_ptr(), *[o.data_ptr() for o in y], None))
    torch.cuda.synchronize()
    y = [o.cpu().numpy().view(np.complex128) for o in y]
    return y if outs > 1 else y[0]


def formula(n):
    k, C = np.arange(n), np.sqrt(2.0 / (n - 1))
    th = ((n - 1 - np.arange(n)) * np.longdouble(np.pi) / (n - 1)).astype(np.longdouble)[:, None]
    t = np.cos(k * th)
    half = np.where((k == 0) | (k == n - 1), 0.5, 1.0)
    return [t.T * (2 * half) / ((n - 1) * C), C * t * half]


@pytest.mark.parametrize("n,ncol", [(3, 1), (4, 9), (5, 2500), (9, 16), (16, 33), (17, 2432), (33, 1217), (64, 5),
                                    (65, 2433), (66, 1300), (127, 70), (128, 2440), (129, 2435), (130, 3),
                                    (95, 2440), (97, 300), (97, 2600), (192, 2432), (193, 2433), (256, 2434), (257, 20), (257, 2440), (258, 6)])
def test_fixed_point_chebyshev(fg, n, ncol):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((ncol, n)) + 1j * rng.standard_normal((ncol, n))
    x[::2] *= np.exp2(-0.25 * np.arange(n))
    ref = formula(n)
    eye = np.eye(n) + 0j
    for q, fn in enumerate(NAMES):
        A = call(fg, fn, n, eye).real.T.astype(np.longdouble)
        if q < 2:
            assert np.abs(A - ref[q]).max() <= 4 * n * n * 2.0 ** -53 * np.abs(ref[q]).max()
        y = call(fg, fn, n, x)
        w = np.frexp(np.abs(A).max(0).astype(float))[1] if q else np.zeros(n, int)
        scaled_a = np.abs(A * np.exp2(-w.astype(float))).max(1)
        for part in ("real", "imag"):
            some = np.unique(np.r_[np.arange(min(ncol, 20)), np.arange(max(ncol - 12, 0), ncol)])
            xp, yp = getattr(x, part)[some].astype(np.longdouble), getattr(y, part)[some]
            B = np.abs(xp) @ np.abs(A).T
            tol = 2.0 ** -52 * B + 4 * n * 2.0 ** -58 * np.outer(np.abs(xp * np.exp2(w.astype(float))).max(1), scaled_a)
            if n > 257:
                tol += n * 2.0 ** -53 * B
            assert (np.abs(yp - xp @ A.T) <= tol).all(), fn
    d1, d2 = call(fg, "falcon_cheb_d1d2_dev", n, x, 2)
    assert np.array_equal(d1, call(fg, NAMES[2], n, x)) and np.array_equal(d2, call(fg, NAMES[3], n, x))


def test_a_column_with_a_nan_is_alone(fg):
    rng = np.random.default_rng(1)
    x = rng.standard_normal((40, 33)) + 1j * rng.standard_normal((40, 33))
    good = call(fg, NAMES[0], 33, x)
    x[7, 5] = complex(np.nan, x[7, 5].imag)
    x[8] = 0.0
    y = call(fg, NAMES[0], 33, x)
    assert np.isnan(y[7].real).all() and np.array_equal(y[7].imag, good[7].imag) and (y[8] == 0).all()
    keep = np.r_[0:7, 9:40]
    assert np.array_equal(y[keep], good[keep])
