"""Chebyshev transforms row by row: the rows away from the walls, whose elements
are smaller by k (d1) and k^2 (d2) than the largest of their columns, are as
accurate as the others.

With w_k = floor(e_k / 2) (falcon-dns_gb300/csrc/falcon_fxgemm.cu; 0 for fwd),
an operator row and a column of X are rounded to 60 bits (59 for fwd, whose
points are added in pairs) at the power of two above their largest weighted
element, and the low halves' product is left out: for A_i and X the largest
weighted elements, 2^-59 A_i |x_k| 2^w_k + 2^-59 X |A_ik| 2^-w_k + 2^-59 A_i X
a term at most; the mirrored rows' differences (below 2^-36 A_i) in 24 bits of
30 bits of X: 2^-59 A_i X a term; the sum is rounded once, and so were the
operator's elements, read back as columns of the identity (2^-53 each, of
sum_k |A_ik x_k|).  So |error| <= 2^-52 sum_k |A_ik x_k| + 4 n 2^-59 A_i X."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG
from test_gpu_fixed_point_chebyshev import NAMES, call

pytestmark = pytest.mark.gpu


def operator(fg, n, fn):
    return call(fg, fn, n, np.eye(n) + 0j).real.T


@pytest.mark.parametrize("n", [17, 64, 65, 129, 257])
def test_every_row(fg, n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((60, n)) + 0j
    x[::3] *= np.exp2(-0.25 * np.arange(n))
    x[1::3] *= np.arange(n) + 1.0
    for q, fn in enumerate(NAMES):
        A = operator(fg, n, fn)
        top = np.abs(A).max(0)
        w = np.where(top > 0, np.floor_divide(np.frexp(top)[1], 2), -1000) if q else np.zeros(n, int)
        amax = np.abs(A * np.exp2(-np.maximum(w, -999).astype(float))).max(1)
        A, xp = A.astype(np.longdouble), x.real.astype(np.longdouble)
        xmax = np.abs(xp * np.exp2(w.astype(float))).max(1)
        tol = 2.0 ** -52 * (np.abs(xp) @ np.abs(A).T) + 4 * n * 2.0 ** -59 * np.outer(xmax, amax)
        err = np.abs(call(fg, fn, n, x).real - xp @ A.T)
        assert (err <= tol).all(), (fn, float((err / tol).max()))


@pytest.mark.parametrize("n", [17, 65, 128])
def test_a_constant_has_no_derivative(fg, n):
    """Coefficient 0 (and 1 in d2) meets a column of zeros: whatever it is, the
    others keep their digits; a NaN in it is one in the result."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((8, n)) + 1j * rng.standard_normal((8, n))
    for fn, count in ((NAMES[2], 1), (NAMES[3], 2)):
        x[:, :count] = 0.0
        want = call(fg, fn, n, x)
        x[:, :count] = 1e30
        assert np.array_equal(call(fg, fn, n, x), want), fn
        x[3, 0] = np.nan
        got = call(fg, fn, n, x)
        assert np.isnan(got[3].real).all() and np.array_equal(got[4], want[4])


@pytest.mark.parametrize("n,few", [(3, 1700), (3, 6666), (7, 1485), (9, 1155), (9, 2222), (13, 800),
                                   (13, 1538), (14, 40), (33, 20), (129, 43), (257, 128)])
def test_few_columns(fg, n, few):
    """Both sides of the rule that gives calls of up to 13 points to FP64 products,
    pairs shared out over blocks, and in place, which does neither:
    within the bound above, or (n + 1) 2^-53 sum_k |A_ik x_k| of an FP64 sum on
    top of it, of the same operator times the columns; d1 and d2 together as apart."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((few + 1, n)) + 1j * rng.standard_normal((few + 1, n))
    some = np.unique(np.r_[0:4, few - 4:few])
    for q, fn in enumerate(NAMES):
        A = operator(fg, n, fn)
        top = np.abs(A).max(0)
        w = np.where(top > 0, np.floor_divide(np.frexp(top)[1], 2), -1000) if q else np.zeros(n, int)
        amax = np.abs(A * np.exp2(-np.maximum(w, -999).astype(float))).max(1)
        xp = x[some]
        size = np.abs(xp.real) + np.abs(xp.imag)
        tol = (n + 4) * 2.0 ** -53 * (size @ np.abs(A).T) + 4 * n * 2.0 ** -59 * np.outer(
            (size * np.exp2(w.astype(float))).max(1), amax)
        want = xp.astype(np.clongdouble) @ A.astype(np.clongdouble).T
        for y in (call(fg, fn, n, x[:few]), call(fg, fn, n, x), in_place(fg, fn, n, x[:few])):
            assert (np.abs(y[some].real - want.real) <= tol).all() and (np.abs(y[some].imag - want.imag) <= tol).all(), fn
    for c in (few, few + 1):
        d1, d2 = call(fg, "falcon_cheb_d1d2_dev", n, x[:c], 2)
        assert np.array_equal(d1, call(fg, NAMES[2], n, x[:c])) and np.array_equal(d2, call(fg, NAMES[3], n, x[:c]))


def in_place(fg, fn, n, x):
    import torch
    y = torch.from_numpy(np.ascontiguousarray(x).view(np.float64)).cuda()
    fg.check(getattr(fg.lib(), fn)(n, x.shape[0], y.data_ptr(), y.data_ptr(), None))
    torch.cuda.synchronize()
    return y.cpu().numpy().view(np.complex128)


RESET = """
import ctypes
import numpy as np
import falcon_gpu as fg

rt = ctypes.CDLL("libcudart.so.13")
x = np.random.default_rng(2).standard_normal((40, 33, 2))

def run():
    a, b = ctypes.c_void_p(), ctypes.c_void_p()
    y = np.empty_like(x)
    for p in (a, b):
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(x.nbytes)) == 0
    assert rt.cudaMemcpy(a, x.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(x.nbytes), 1) == 0
    fg.check(fg.lib().falcon_cheb_d1_dev(33, 40, a, b, None))
    assert rt.cudaMemcpy(y.ctypes.data_as(ctypes.c_void_p), b, ctypes.c_size_t(x.nbytes), 2) == 0
    return y

first = run()
assert rt.cudaDeviceReset() == 0
spare = ctypes.c_void_p()
assert rt.cudaMalloc(ctypes.byref(spare), ctypes.c_size_t(1 << 20)) == 0
assert np.array_equal(run(), first)
print("ok")
"""


def test_after_a_device_reset(fg):
    """The operators go with their context: those of a size used before are made
    again in a new one."""
    r = subprocess.run([sys.executable, "-c", RESET], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=PKG))
    assert r.returncode == 0 and r.stdout.split()[-1] == "ok", (r.returncode, r.stdout, r.stderr[-2000:])
