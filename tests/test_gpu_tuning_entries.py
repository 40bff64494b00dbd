"""Decisions of a library whose tiles were other kernels (w = 6 or 7) are read
from a cache file and not used: the shapes are measured again; and those of the
environment's file are used from the first product on."""
import os
import subprocess
import sys

import pytest

from conftest import PKG
from test_gpu_tuning import read_cache, run, tuned  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


def test_earlier_decisions_are_not_used(fg, tuned, tmp_path):  # noqa: F811
    ps = [fg.make_params(33, 20, "SBDF3", ra=1e5 * (1 + k), dt=1e-5) for k in range(3)]
    run(fg, ps, range(3), 3)
    rows = read_cache(tuned)
    assert len(rows) == fg.tune_entries()[0] > 0
    old = tmp_path / "old.txt"
    with open(old, "w") as f:
        f.write("falcon-contraction-tuning 2\n")
        for dev, key, us in rows:
            key[4] %= 60
            key[7] = 0 if key[5] >= 2 else 1
            f.write(" ".join([dev, *map(str, key), *map(str, us)]) + "\n")
    fg.tune_clear()
    fg.set_tune_cache(old)
    n, measured = fg.tune_entries()
    assert n == len(rows)
    run(fg, ps, range(3), 3)
    assert fg.tune_entries()[1] - measured == len(rows)
    assert len(read_cache(old)) == 2 * len(rows)


CHILD = """
import falcon_gpu as fg
b = fg.Batch([fg.make_params(33, 20, "CNAB2", ra=1e5 * (1 + k), dt=1e-5) for k in range(3)])
b.init_noise(range(3))
b.step(5)
b.get_state(0)
print("measured", fg.tune_entries()[1])
"""


def test_the_environments_file_is_read_before_the_first_decision(fg, tmp_path):
    """A process that finds its shapes in FALCON_TUNE_CACHE measures none of them."""
    cache = tmp_path / "env.txt"
    env = dict(os.environ, PYTHONPATH=PKG, FALCON_TUNE_CACHE=str(cache))
    for turn in range(2):
        r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300, env=env)
        assert r.returncode == 0, r.stderr[-2000:]
        measured = int(r.stdout.split()[-1])
        if turn == 0:
            rows = read_cache(cache)
            assert measured == len(rows) > 0
        else:
            assert measured == 0 and read_cache(cache) == rows
