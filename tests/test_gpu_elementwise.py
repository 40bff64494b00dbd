"""The right-hand-side and stage kernels' grids and unrolled forms: an instance
steps to the same bits alone (blocks of 64) and in a batch whose rows end inside
a block of 128, for every number of history levels and stages that has a form of
its own and for one that has not; every kernel does the same FP64 operations per
element wherever the element lies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["CNAB2", "CNAB3", "SBDF2", "SBDF3", "SBDF4", "ARS222", "ARS343", "ARS443", "BPR353", "EUL111",
                                    "MARS343", "RK2", "RK4"])
@pytest.mark.parametrize("R,Nm,B", [(17, 9, 7), (33, 42, 33), (20, 21, 31)])
def test_alone_and_in_a_batch(fg, scheme, R, Nm, B):
    prev = fg.set_gemm_mode(0)
    try:
        ps = [fg.make_params(R, Nm, scheme, ra=1e4 * (1 + k), dt=1e-6) for k in range(B)]
        b = fg.Batch(ps)
        b.init_noise([5 + k for k in range(B)])
        b.step(5)
        for k in (0, B - 1):
            a = fg.Batch([ps[k]])
            a.init_noise([5 + k])
            a.step(5)
            x, y = a.get_state(0), b.get_state(k)
            assert all(np.array_equal(x[f], y[f]) for f in ("T", "omg", "up", "ur")), k
    finally:
        fg.set_gemm_mode(prev)
