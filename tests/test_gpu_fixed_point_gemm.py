"""The fixed-point integer contractions (falcon-dns_gb300/csrc/falcon_fxgemm.cu,
falcon_set_gemm_mode(0)): every radial and per-mode product of a step, at
radial sizes around the kernels' row blocks, K chunks and k shares and at
batch sizes around their column tiles.

- an instance's bits do not depend on the batch it steps in (the narrow
  kernel alone, tiles of every width in batches: sums of integers);
- against the exact bf16 slices on mma.sync (mode 1).  Both keep 57 or more
  bits of a product relative to the largest of its row or column, so a
  contraction's outputs differ by at most sqrt(2 K) 2^-57 max|A| max|X|, the
  rounding of an FP64 product sum (K = 131: 2^-53); steps amplify a rounding
  by the operators' condition, 1e-12 over 20 steps at Nr = 65 for FP64 tiles,
  so 4e-12 over 3 steps at Nr <= 131."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

FIELDS = ("T", "omg", "up", "ur")


def states(fg, mode, R, Nm, scheme, B, nsteps=3):
    prev = fg.set_gemm_mode(mode)
    try:
        b = fg.Batch([fg.make_params(R, Nm, scheme, ra=1e5 * (1 + k), dt=1e-6) for k in range(B)])
        b.init_noise([70 + k for k in range(B)])
        b.step(nsteps)
        out = [b.get_state(i) for i in range(B)]
        b.close()
        return out
    finally:
        fg.set_gemm_mode(prev)


@pytest.mark.parametrize("R,Nm,scheme,B", [
    (17, 5, "CNAB2", 1), (16, 6, "SBDF2", 2), (31, 9, "SBDF3", 3), (32, 20, "CNAB2", 4), (33, 7, "ARS343", 5),
    (64, 12, "BPR353", 8), (65, 21, "SBDF3", 9), (66, 5, "CNAB2", 17), (97, 8, "ARS443", 33), (129, 10, "SBDF3", 1),
    (131, 5, "CNAB2", 16), (130, 4, "SBDF2", 40)])
def test_fixed_point_contractions(fg, R, Nm, scheme, B):
    got, ref = states(fg, 0, R, Nm, scheme, B), states(fg, 1, R, Nm, scheme, B)
    for g, r in zip(got, ref):
        assert max(rel(g[f], r[f]) for f in FIELDS) < 4e-12
    prev = fg.set_gemm_mode(0)
    try:
        a = fg.Instance(fg.make_params(R, Nm, scheme, ra=1e5 * B, dt=1e-6))
        a.init_noise(70 + B - 1)
        a.step(3)
        alone = a.get_state()
        a.close()
    finally:
        fg.set_gemm_mode(prev)
    for f in FIELDS:
        assert np.array_equal(alone[f], got[B - 1][f]), f


@pytest.mark.parametrize("R,Nm,scheme,B", [(17, 5, "RK2", 1), (33, 16, "RK4", 1), (33, 15, "RK4", 4), (65, 21, "RK2", 9),
                                           (33, 16, "CNAB2", 1), (65, 20, "SBDF2", 3)])
def test_products_in_one_launch(fg, R, Nm, scheme, B):
    """A stage's radial products as one launch (two, five or six of them, the
    last of twice the batch's columns, none a multiple of the tile): the same
    bound against mode 1 as above, and mode 4 repeats its own bits whichever
    way it decided."""
    got, ref = states(fg, 0, R, Nm, scheme, B), states(fg, 1, R, Nm, scheme, B)
    for g, r in zip(got, ref):
        assert max(rel(g[f], r[f]) for f in FIELDS) < 4e-12
    a, b = states(fg, 4, R, Nm, scheme, B), states(fg, 4, R, Nm, scheme, B)
    for g, h, r in zip(a, b, ref):
        assert all(np.array_equal(g[f], h[f]) for f in FIELDS)
        assert max(rel(g[f], r[f]) for f in FIELDS) < 4e-12


@pytest.mark.parametrize("R,Nm,scheme,B", [(97, 341, "CNAB2", 1), (65, 170, "SBDF2", 4), (65, 170, "CNAB2", 3),
                                           (49, 85, "BPR353", 2), (128, 64, "SBDF3", 3), (17, 512, "CNAB2", 2),
                                           (9, 3, "CNAB2", 1), (129, 85, "ARS222", 4)])
def test_narrow_shares_and_what_follows(fg, R, Nm, scheme, B):
    """Narrow products of one to eight k shares and one to many row blocks, with
    the buoyancy, u_r and mode 0 in the same launches: the same bound against
    mode 1, which does these in kernels of their own."""
    got, ref = states(fg, 0, R, Nm, scheme, B), states(fg, 1, R, Nm, scheme, B)
    for g, r in zip(got, ref):
        assert max(rel(g[f], r[f]) for f in FIELDS) < 4e-12


@pytest.mark.parametrize("R,Nm,scheme,counts", [(33, 42, "CNAB2", (2, 1, 1)), (33, 10, "SBDF3", (1, 5)),
                                                (65, 85, "BPR353", (1, 2, 1)), (17, 20, "CNAB2", (1,) * 10),
                                                (17, 20, "CNAB2", (1,) * 11), (48, 16, "SBDF2", (9, 2, 6))])
def test_products_of_several_prandtl_numbers(fg, R, Nm, scheme, counts):
    """The temperature products of a group's Prandtl numbers in one launch (uneven
    widths, up to the ten it takes, and one more): the bits of each instance
    alone, and the bound above against mode 1."""
    prs = [0.3 * 1.7 ** k for k, c in enumerate(counts) for _ in range(c)]

    def run(mode, which):
        prev = fg.set_gemm_mode(mode)
        try:
            b = fg.Batch([fg.make_params(R, Nm, scheme, ra=1e5 * (1 + k), pr=prs[k], dt=1e-6) for k in which])
            b.init_noise([70 + k for k in which])
            b.step(3)
            out = [b.get_state(i) for i in range(len(which))]
            b.close()
            return out
        finally:
            fg.set_gemm_mode(prev)

    every = range(len(prs))
    got, ref = run(0, every), run(1, every)
    for k in every:
        assert max(rel(got[k][f], ref[k][f]) for f in FIELDS) < 4e-12
    for k in (0, len(prs) - 1):
        alone = run(0, [k])[0]
        assert all(np.array_equal(alone[f], got[k][f]) for f in FIELDS)


def test_longest_contraction(fg, orc):
    """K = 257, the most the fixed-point sums hold."""
    prev = fg.set_gemm_mode(0)
    try:
        g = fg.Instance(fg.make_params(257, 4, "CNAB2", ra=1e5, dt=1e-7))
        o = orc.Sim(orc.make_params(257, 4, "CNAB2", ra=1e5, dt=1e-7))
        g.init_noise(1)
        o.init_noise(1)
        g.step(3)
        o.step(3)
        a, b = g.get_state(), o.get_state()
        for f in FIELDS:
            assert rel(a[f], b[f]) < 1e-8, f
        g.close()
    finally:
        fg.set_gemm_mode(prev)
