"""What the launcher of the fixed-point products refuses, on the host: operators of
more than 257 columns, products without integers, and a velocity product (whose
launch's whole grid makes mode 0) together with products of other widths."""
import os
import subprocess

from conftest import PKG

SOURCE = r"""
#include <stdio.h>
#include "falcon_internal.h"
using namespace falcon;
int main() {
  GemmArgs g{};
  g.rows = 99; g.K = 33; g.N = 8; g.batch = 4; g.lda = 99;
  auto say = [&](const char* what) { printf("%s %d\n", what, launch_fx_gemm(g, 0) == cudaErrorInvalidValue); };
  say("no_integers");
  g.fx = reinterpret_cast<const int2*>(16);
  g.K = 258;
  say("too_long");
  g.K = 33;
  g.follow.kind = kVelocity;
  g.nextra = 1;
  say("extra");
  g.nextra = 0;
  g.nsub = 2;
  say("sub");
  g.nsub = 0;
  g.njobs = 2;
  say("jobs");
  g.N = 0;
  printf("nothing %d\n", launch_fx_gemm(g, 0) == cudaSuccess);
}
"""


def test_refused_products(fg, tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    build = os.path.join(PKG, "_build")
    (tmp_path / "h.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(cuda, "include"),
                    str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h"), "-L" + build, "-lfalcon_gpu",
                    "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + build], check=True, timeout=300)
    r = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True, timeout=60, check=True,
                       env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    got = dict(line.split() for line in r.stdout.splitlines())
    assert got == dict.fromkeys(("no_integers", "too_long", "extra", "sub", "jobs", "nothing"), "1"), got
