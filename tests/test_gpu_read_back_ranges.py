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


def test_overlapping_arrays(fg):
    """Two fields into one page-locked array: the later one's values, as with a copy per field."""
    import torch
    R, Nm = 65, 170
    n = 2 * R * (Nm + 1)
    b = fg.Batch([fg.make_params(R, Nm, "CNAB2", ra=1e5, dt=1e-6)])
    b.init_noise([1])
    b.step(2)
    want = {k: v.view(np.float64).ravel() for k, v in b.get_state(0).items()}
    ptr = ctypes.POINTER(ctypes.c_double)
    a = torch.zeros(n + n // 2, dtype=torch.float64, pin_memory=True).numpy()
    at = lambda v: v.ctypes.data_as(ptr)  # noqa: E731
    for _ in range(20):
        a[:] = np.nan
        fg.check(fg.lib().falcon_batch_get_state(b.h, 0, at(a), at(a), None, None, at(a)))
        assert np.array_equal(a[:n], want["psi"]) and np.isnan(a[n:]).all()
        fg.check(fg.lib().falcon_batch_get_state(b.h, 0, at(a[n // 2:]), None, at(a), None, None))
        assert np.array_equal(a[:n], want["up"]) and np.array_equal(a[n:], want["T"][n // 2:])
    b.close()
