"""Reading an instance's fields back (falcon_batch_get_state): into pageable,
page-locked, misaligned and missing arrays, any mixture of them in one call,
the same values."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,Nm,B", [(17, 4, 1), (33, 21, 5)])
def test_read_back_into_any_memory(fg, R, Nm, B):
    import torch
    b = fg.Batch([fg.make_params(R, Nm, "CNAB2", ra=1e5 * (1 + k), dt=1e-5) for k in range(B)])
    b.init_noise(range(B))
    b.step(3)
    n = R * (Nm + 1)
    ptr = ctypes.POINTER(ctypes.c_double)
    for i in (0, B - 1):
        want = b.get_state(i)
        names = ("T", "omg", "up", "ur", "psi")
        pinned = torch.full((2 * n,), float("nan"), dtype=torch.float64, pin_memory=True).numpy()
        tail = torch.full((2 * n + 1,), float("nan"), dtype=torch.float64, pin_memory=True).numpy()  # 8-byte aligned part
        pageable = np.full(2 * n, np.nan)
        into = [pinned, tail[1:], None, pageable, None]
        for turn in range(5):  # every kind of memory for every field
            args = [into[(k + turn) % 5] for k in range(5)]
            for a in (pinned, tail, pageable):
                a[:] = np.nan
            fg.check(fg.lib().falcon_batch_get_state(b.h, i, *[None if a is None else a.ctypes.data_as(ptr) for a in args]))
            for a, name in zip(args, names):
                if a is not None:
                    assert np.array_equal(a, want[name].view(np.float64).ravel()), (turn, name)
            assert np.isnan(tail[0])
    b.close()
