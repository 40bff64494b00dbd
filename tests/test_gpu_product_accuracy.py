"""The fixed-point products (falcon-dns_gb300/csrc/falcon_fxgemm.cu) one by one
against extended precision and against the FP64 products (launch_gemm), through
their launchers: operators whose rows and columns are uneven (radial
derivatives, inverse Helmholtz operators), on even fields, on fields that vanish
at the walls and on fields that are large there.

Element bound: with w_k = floor(e_k / 2), e_k the exponent of column k's largest
element (|a| < 2^e_k), an operator row and an X column are rounded to 60 bits at
the power of two above their largest weighted element: 2^-60 of that element A_i
(or X_n) at most, each; the low halves' product that is left out is below
2^58 2^-120 (2 A_i)(2 X_n) = 2^-60 A_i X_n; the sum is rounded once.  So
|error| <= 3 K 2^-60 A_i X_n + 2^-53 |y| (a second time, for the factors of
2^-60 that the first two products share).

Norm bound: no more than FP64's own error on the same operands."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include <vector>
#include "falcon_internal.h"
using namespace falcon;
extern "C" int product(int fixed, int rows, int K, int N, int batch, const double* A, const double* X, double* Y) {
  const size_t na = (size_t)batch * rows * K, nx = (size_t)batch * K * N, ny = (size_t)batch * rows * N;
  double *a = nullptr, *x = nullptr, *y = nullptr;
  int2* fx = nullptr;
  int *ex = nullptr, *w = nullptr;
  cudaError_t e = cudaMalloc(&a, na * 8);
  if (!e) e = cudaMalloc(&x, nx * 8);
  if (!e) e = cudaMalloc(&y, ny * 8);
  if (!e) e = cudaMalloc(&fx, na * sizeof(int2));
  if (!e) e = cudaMalloc(&ex, (size_t)batch * rows * sizeof(int));
  if (!e) e = cudaMalloc(&w, (size_t)batch * K * sizeof(int));
  if (!e) e = cudaMemcpy(a, A, na * 8, cudaMemcpyHostToDevice);
  if (!e) e = cudaMemcpy(x, X, nx * 8, cudaMemcpyHostToDevice);
  GemmArgs g{};
  g.A = a; g.lda = rows; g.sA = (long)rows * K;
  g.X = x; g.ldx = N; g.sX = (long)K * N;
  g.Y = y; g.ldy = N; g.sY = (long)rows * N;
  g.rows = rows; g.K = K; g.N = N; g.batch = batch; g.alpha = 1.0;
  g.fx = fx; g.fx_ex = ex; g.fx_w = w;
  if (!e && fixed) e = launch_fx_operator(a, rows, g.sA, rows, K, batch, w, fx, ex, 0);
  if (!e) e = fixed ? launch_fx_gemm(g, 0) : launch_gemm(g, 0);
  if (!e) e = cudaDeviceSynchronize();
  if (!e) e = cudaMemcpy(Y, y, ny * 8, cudaMemcpyDeviceToHost);
  cudaFree(a); cudaFree(x); cudaFree(y); cudaFree(fx); cudaFree(ex); cudaFree(w);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def product(fg, tmp_path_factory):
    d = tmp_path_factory.mktemp("product")
    (d / "h.cpp").write_text(HARNESS)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    build = os.path.join(PKG, "_build")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(cuda, "include"), str(d / "h.cpp"), "-o", str(d / "h.so"), "-L" + build,
                    "-lfalcon_gpu", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + build],
                   check=True, timeout=300)
    lib = ctypes.CDLL(str(d / "h.so"))

    def run(fixed, A, X):
        """A [batch][rows][K], X [batch][K][N]"""
        batch, rows, K = A.shape
        N = X.shape[2]
        a = np.ascontiguousarray(A.transpose(0, 2, 1))
        x = np.ascontiguousarray(X)
        y = np.empty((batch, rows, N))
        p = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        assert lib.product(fixed, rows, K, N, batch, p(a), p(x), p(y)) == 0
        return y

    return run


def derivatives(n):
    """d/dr and the Laplacian of mode 0 by values at the Chebyshev points of an annulus of width 1."""
    x = np.cos((n - 1 - np.arange(n)) * np.pi / (n - 1))
    t, d, d2 = np.zeros((3, n, n))
    t[:, 0], t[:, 1], d[:, 1] = 1.0, x, 1.0
    for j in range(2, n):
        t[:, j] = 2 * x * t[:, j - 1] - t[:, j - 2]
        d[:, j] = 2 * t[:, j - 1] + 2 * x * d[:, j - 1] - d[:, j - 2]
        d2[:, j] = 4 * d[:, j - 1] + 2 * x * d2[:, j - 1] - d2[:, j - 2]
    h = np.ones(n)
    h[[0, -1]] = 0.5
    coef = h[:, None] * (t * (2 * h)[:, None]).T / (n - 1)
    r = 0.35 / 0.65 + 0.5 * (1 + x)
    d1 = 2 * d @ coef
    return x, r, d1, 4 * d2 @ coef + d1 / r[:, None]


def operators(n):
    x, r, d1, lap = derivatives(n)
    helm = np.eye(n) - 1e-5 * (lap - np.diag((20 / r) ** 2))
    helm[[0, -1]] = np.eye(n)[[0, -1]]
    solve = np.linalg.inv(helm)
    return x, {"d/dr": d1, "laplacian": lap, "solve": solve, "solve, d/dr": d1 @ solve}


def fields(x, ncol, rng):
    s = np.polynomial.chebyshev.chebval(x, rng.standard_normal((10, ncol)) * np.exp2(-np.arange(10))[:, None]).T
    wall = (1 - x * x)[:, None]
    return {"even": rng.standard_normal((len(x), ncol)), "smooth": s, "zero at the walls": s * wall,
            "with its slope": s * wall ** 2, "large at the walls": s / (0.01 + wall)}


@pytest.mark.parametrize("n", [17, 33, 65, 129, 257])
@pytest.mark.parametrize("ncol", [2, 8, 48])
def test_uneven_products(product, n, ncol):
    rng = np.random.default_rng(n + ncol)
    x, ops = operators(n)
    for op, A in ops.items():
        w = np.floor_divide(np.frexp(np.abs(A).max(0))[1], 2)
        amax = np.abs(A * np.exp2(-w.astype(float))).max(1)
        for kind, X in fields(x, 48, rng).items():
            X3 = np.ascontiguousarray(X.reshape(n, 48 // ncol, ncol).transpose(1, 0, 2))
            A3 = np.broadcast_to(A, (48 // ncol, n, n))
            flat = lambda y: y.transpose(1, 0, 2).reshape(n, 48)  # noqa: E731
            exact = A.astype(np.longdouble) @ X.astype(np.longdouble)
            y = flat(product(1, A3, X3))
            err = np.abs(y - exact)
            xmax = np.abs(X * np.exp2(w.astype(float))[:, None]).max(0)
            assert (err <= 3 * n * 2.0 ** -60 * np.outer(amax, xmax) + 2.0 ** -52 * np.abs(exact)).all(), (op, kind)
            if n <= 129:
                ref = np.abs(flat(product(0, A3, X3)) - exact)
                assert np.linalg.norm(err.astype(float)) <= np.linalg.norm(ref.astype(float)), (op, kind)


@pytest.mark.parametrize("ncol", [2, 7, 40])
@pytest.mark.parametrize("n", [3, 7, 8, 14, 15, 64, 129, 256, 257])
def test_largest_sums(product, n, ncol):
    """Every element the largest its scale holds, of one sign (columns 0), alternating
    (1) and with opposite low halves (the others): sums at the limit of the carries,
    within the element bound."""
    a = np.full((1, 33, n), 1.0 - 2.0 ** -53)
    x = np.full((1, n, ncol), -(1.0 - 2.0 ** -53))
    x[0, :, 1] *= np.where(np.arange(n) % 2, 1.0, -1.0)
    x[0, :, 2:] -= 2.0 ** -30 + 2.0 ** -31
    a[0, 1::2] -= 2.0 ** -31
    exact = a[0].astype(np.longdouble) @ x[0].astype(np.longdouble)
    err = np.abs(product(1, a, x)[0] - exact)
    w = np.floor_divide(np.frexp(np.abs(a[0]).max(0))[1], 2)
    assert (w == 0).all()
    assert (err <= 3 * n * 2.0 ** -60 * 1.01 + 2.0 ** -52 * np.abs(exact)).all()


@pytest.mark.parametrize("ncol", [2, 40])
def test_fp64_products(product, ncol):
    """launch_gemm, which modes 0 and 2 and operators without integers take: |error| <= (K + 1) 2^-53 sum |a x|."""
    rng = np.random.default_rng(3)
    for n in (33, 258, 300):
        A, X = rng.standard_normal((2, n + 1, n)), rng.standard_normal((2, n, ncol))
        al, xl = A.astype(np.longdouble), X.astype(np.longdouble)
        err = np.abs(product(0, A, X) - al @ xl)
        assert (err <= (n + 1) * 2.0 ** -53 * (np.abs(al) @ np.abs(xl))).all()
