"""The error word of the tcgen05 contraction's bounded waits: set here from the
host, in place of a kernel whose wait ran out; and what else is kept per context."""
import ctypes
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "falcon_tc.h"
extern "C" int set_word(int v) {
  int* p = falcon::tc_error_word();
  if (p) *p = v;
  return p != nullptr;
}
"""


@pytest.fixture(scope="module")
def set_word(fg, tmp_path_factory):
    d = tmp_path_factory.mktemp("word")
    (d / "h.cpp").write_text(HARNESS)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    build = os.path.join(PKG, "_build")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(cuda, "include"), str(d / "h.cpp"), "-o", str(d / "h.so"), "-L" + build,
                    "-lfalcon_gpu", "-Wl,-rpath," + build], check=True, timeout=300)
    return ctypes.CDLL(str(d / "h.so")).set_word


def test_a_new_batch_or_server_leaves_it(fg, set_word):
    """A timeout in one batch's steps is reported by that batch, although another
    batch and a server were made in between; once."""
    a = fg.Batch([fg.make_params(17, 5)])
    a.init_noise([1])
    a.step(1)
    a.get_state(0)
    assert set_word(3)
    b = fg.Batch([fg.make_params(9, 5)])
    s = fg.Server(1 << 30)
    with pytest.raises(fg.FalconError, match="timed out .code 3."):
        a.get_state(0)
    a.get_state(0)
    a.close()
    b.close()
    del s


RESET = """
import ctypes
import numpy as np
import falcon_gpu as fg

def run(mode, nm=42):
    fg.set_gemm_mode(mode)
    b = fg.Batch([fg.make_params(65, nm, "SBDF3", ra=1e5 * (k + 1), dt=1e-6) for k in range(12)])
    b.init_noise(range(12))
    b.step(3)
    out = b.get_state(11)["omg"]
    b.close()
    return out

first = [run(m) for m in (0, 1, 3, 4, 5)]
assert ctypes.CDLL("libcudart.so.13").cudaDeviceReset() == 0
for m, x in zip((0, 1, 3, 4, 5), first):
    assert np.array_equal(run(m), x), m
run(4, 20)  # shapes that are measured anew
print("ok")
"""


def test_after_a_device_reset(fg):
    """The error word, the kernels' shared-memory limits and the autotuner's buffer
    go with their context: a device that was reset steps on, with the same bits."""
    r = subprocess.run([sys.executable, "-c", RESET], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=PKG))
    assert r.returncode == 0 and r.stdout.split()[-1] == "ok", (r.returncode, r.stdout, r.stderr[-2000:])
