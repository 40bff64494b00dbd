"""Kept transform tables (make_fft of falcon-dns_gb300/csrc/falcon_host.cpp, at
most 8): more sizes than are kept, in turn and from four threads on streams of
their own, give the bits of the allocation-free form, which copies its tables
on every call; a batch made before its tables were dropped from the kept ones
steps on with them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (5, 8, 11, 16, 21, 25, 33, 42, 64, 85, 100, 170)


def nonlin(fg, fn, Nm, dev, stream):
    import torch
    outs = [torch.zeros_like(dev[0]) for _ in range(4)]
    stream.synchronize()
    fg.check(getattr(fg.lib(), fn)(9, Nm, 2, *[x.data_ptr() for x in dev + outs], stream.cuda_stream))
    stream.synchronize()
    return torch.stack(outs)


def test_more_sizes_than_kept_from_several_threads(fg):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    main = torch.cuda.current_stream()
    dev = {n: [torch.randn(9 * (n + 1) * 2 * 2, generator=g, device="cuda", dtype=torch.float64) for _ in range(4)]
           for n in SIZES}
    ref = {n: nonlin(fg, "falcon_nonlin_noalloc_dev", n, dev[n], main) for n in SIZES}
    b = fg.Batch([fg.make_params(17, 12, "CNAB2", ra=1e5, dt=1e-6)])
    b.init_noise([1])
    bad, done = [], []

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for r in range(3):
                for n in np.roll(SIZES, 3 * k + r):
                    if not torch.equal(nonlin(fg, "falcon_nonlin_dev", int(n), dev[int(n)], s), ref[int(n)]):
                        bad.append(n)
        done.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(done) == 4 and not bad
    for n in SIZES:  # and with nothing at the same time
        assert torch.equal(nonlin(fg, "falcon_nonlin_dev", n, dev[n], main), ref[n])
    c = fg.Batch([fg.make_params(17, 12, "CNAB2", ra=1e5, dt=1e-6)])
    c.init_noise([1])
    b.step(3)
    c.step(3)
    assert np.array_equal(b.get_state(0)["T"], c.get_state(0)["T"])
