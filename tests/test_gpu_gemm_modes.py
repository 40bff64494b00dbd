"""Which arithmetic a contraction mode stands for: mode 0 is FP64 (products and
what follows them in launches of their own), mode 5 the fixed-point integers, on
which the tests of tests/test_gpu_fixed_point_gemm.py and
tests/test_gpu_elementwise.py run here as well; a step's results differ by a
rounding (2^-53 an operation, amplified by the operators' condition: 4e-12 over
3 steps at Nr <= 131, as there)."""
import pytest

import test_gpu_elementwise as elementwise
import test_gpu_fixed_point_gemm as fixed
from conftest import rel

pytestmark = pytest.mark.gpu


class FixedPoint:
    """The library with mode 0 asked for answered by mode 5."""

    def __init__(self, fg):
        self._fg = fg

    def __getattr__(self, name):
        return getattr(self._fg, name)

    def set_gemm_mode(self, mode):
        prev = self._fg.set_gemm_mode(5 if mode == 0 else mode)
        return 0 if prev == 5 else prev


@pytest.mark.parametrize("R,Nm,scheme,B", [(33, 20, "CNAB2", 1), (65, 21, "SBDF3", 9), (49, 16, "ARS443", 2)])
def test_mode_0_is_fp64(fg, R, Nm, scheme, B):
    """Per step and stage at least: the radial products, the temperature solve, the
    buoyancy, three blocks of the vorticity solve, uphi_bar and the velocity, one
    launch each, the nonlinear pass and a right-hand side."""
    launches, out = {}, {}
    graphs = fg.lib().falcon_set_step_graphs(0)
    try:
        for mode in (0, 5):
            prev = fg.set_gemm_mode(mode)
            b = fg.Batch([fg.make_params(R, Nm, scheme, ra=1e5, dt=1e-6) for _ in range(B)])
            b.init_noise(range(B))
            b.step(1)
            n = fg.lib().falcon_launch_count()
            b.step(2)
            launches[mode] = (fg.lib().falcon_launch_count() - n) / 2
            out[mode] = b.get_state(B - 1)
            b.close()
            fg.set_gemm_mode(prev)
    finally:
        fg.lib().falcon_set_step_graphs(graphs)
    assert launches[0] >= 11 > launches[5] / (5 if scheme == "ARS443" else 1), launches
    assert max(rel(out[0][f], out[5][f]) for f in fixed.FIELDS) < 4e-12
    assert any((out[0][f] != out[5][f]).any() for f in fixed.FIELDS)


def _cases(test):
    return pytest.mark.parametrize(*next(m for m in test.pytestmark if m.name == "parametrize").args)


@_cases(fixed.test_fixed_point_contractions)
def test_fixed_point_contractions(fg, R, Nm, scheme, B):
    fixed.test_fixed_point_contractions(FixedPoint(fg), R, Nm, scheme, B)


@_cases(fixed.test_products_in_one_launch)
def test_products_in_one_launch(fg, R, Nm, scheme, B):
    fixed.test_products_in_one_launch(FixedPoint(fg), R, Nm, scheme, B)


@_cases(fixed.test_narrow_shares_and_what_follows)
def test_narrow_shares_and_what_follows(fg, R, Nm, scheme, B):
    fixed.test_narrow_shares_and_what_follows(FixedPoint(fg), R, Nm, scheme, B)


@_cases(fixed.test_products_of_several_prandtl_numbers)
def test_products_of_several_prandtl_numbers(fg, R, Nm, scheme, counts):
    fixed.test_products_of_several_prandtl_numbers(FixedPoint(fg), R, Nm, scheme, counts)


@pytest.mark.parametrize("scheme", ["CNAB2", "SBDF3", "ARS343", "RK4"])
def test_alone_and_in_a_batch(fg, scheme):
    elementwise.test_alone_and_in_a_batch(FixedPoint(fg), scheme, 33, 42, 33)


def test_longest_contraction(fg, orc):
    fixed.test_longest_contraction(FixedPoint(fg), orc)
