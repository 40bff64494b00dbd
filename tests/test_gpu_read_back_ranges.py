"""Reading back into arrays of which only a part is page-locked: the first and
the last page registered, the ones between not; and into registered memory."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 65536  # a multiple of the pages of x86-64 and of Arm


def test_partly_registered_arrays(fg):
    import torch
    torch.cuda.init()
    rt = ctypes.CDLL("libcudart.so.13")
    R, Nm = 65, 170
    b = fg.Batch([fg.make_params(R, Nm, "CNAB2", ra=1e5, dt=1e-6)])
    b.init_noise([1])
    b.step(2)
    want = b.get_state(0)
    n = 16 * R * (Nm + 1)
    pages = n // PAGE + 2
    assert pages >= 4
    raw = np.zeros((5, (pages + 1) * PAGE), np.uint8)
    ptr = ctypes.POINTER(ctypes.c_double)
    views, registered = [], []
    for k, a in enumerate(raw):
        first = -a.ctypes.data % PAGE
        # the field ends in the last registered page
        last = first + (pages - 1) * PAGE
        for at in ((first, last) if k < 4 else [first]):
            size = PAGE if k < 4 else pages * PAGE
            assert rt.cudaHostRegister(ctypes.c_void_p(a.ctypes.data + at), ctypes.c_size_t(size), 0) == 0
            registered.append(a.ctypes.data + at)
        end = last + 16
        views.append(a[end - n:end].view(np.float64))
        assert first <= end - n < first + PAGE
    try:
        for v in views:
            v[:] = np.nan
        fg.check(fg.lib().falcon_batch_get_state(b.h, 0, *[v.ctypes.data_as(ptr) for v in views]))
        for v, name in zip(views, ("T", "omg", "up", "ur", "psi")):
            assert np.array_equal(v, want[name].view(np.float64).ravel()), name
    finally:
        for at in registered:
            assert rt.cudaHostUnregister(ctypes.c_void_p(at)) == 0
        b.close()
