"""The error word of the tcgen05 contraction's bounded waits: set here from the
host, in place of a kernel whose wait ran out."""
import ctypes
import os
import subprocess

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
