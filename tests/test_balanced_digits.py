"""The tensor-core butterflies' integer products (fx_mma_stage and
fx_mma_stage_wide of falcon-dns_gb300/csrc/falcon_fft.cuh) restated in exact
integers on the coefficient tables of falcon_fixed.h: seven balanced 9-bit
digits give back a constant and a value, the FP32 sums of every diagonal stay
exact above their start of 1.5 2^23, and what the accumulators' bits are put
together to is the product but for the digit pairs that are left out."""
import os
import random
import re

import pytest

from conftest import PKG

S, BIAS = 7, 256 * ((1 << 63) // 511)
MAGIC = 0x4B400000


def tables(p):
    src = open(os.path.join(PKG, "csrc", "falcon_fixed.h")).read()
    body = re.search(r"struct FxDft<%d> \{(.*?)\};\n\};" % p, src, re.S).group(1)
    c, s = (re.search(r"%s\[%d\] = \{(.*?)\}" % (k, p), body + "}", re.S).group(1) for k in "cs")
    return [[int(v) for v in re.findall(r"(-?\d+)LL", t)] for t in (c, s)]


def constant_digits(c):  # fx_digit
    out = []
    for i in range(S - 1, 0, -1):
        d = (c + 256) % 512 - 256
        out.append(d)
        c = (c - d) // 512
    return [c] + out[::-1]


def value_digits(v):  # fx_digits of the biased value
    u = (v + BIAS) % (1 << 64)
    return [(u >> 9 * (S - 1 - s) & 511) - 256 for s in range(S)]


def together(sums):  # fx_undigit: 64-bit integers, the last diagonal shifted down
    off = -sum(MAGIC << sh for sh in (46, 37, 28, 19, 10, 1)) - (MAGIC >> 8)
    bits = [MAGIC + q for q in sums]
    w = off + sum(b << sh for b, sh in zip(bits[:6], (46, 37, 28, 19, 10, 1))) + (bits[6] >> 8)
    return (w + (1 << 63)) % (1 << 64) - (1 << 63)


@pytest.mark.parametrize("p", [11, 13, 17, 19, 23, 29, 31])
def test_products_of_digits(p):
    rng = random.Random(p)
    h = (p - 1) // 2
    for table in tables(p):
        assert len(table) == p and max(map(abs, table)) <= 1 << 62
        digits = [constant_digits(c) for c in table]
        for c, d in zip(table, digits):
            assert sum(q * 512 ** (S - 1 - i) for i, q in enumerate(d)) == c and all(-256 <= q <= 255 for q in d[1:])
        # a diagonal's largest partial sum: |digits of the constants| times 256 (a leading digit's bound too)
        for j in range(1, h + 1):
            rows = [digits[j * q % p] for q in range(1, h + 1)]
            for d in range(S):
                assert 256 * sum(abs(r[s]) for r in rows for s in range(d + 1)) < 0.9 * 2 ** 22
        for _ in range(50):
            # |a_q| < 2^61 each, their products' sums below 2^61 as in the stages
            v = [rng.randrange(-(1 << 61) // h, (1 << 61) // h) for _ in range(h)]
            vd = [value_digits(x) for x in v]
            for x, d in zip(v, vd):
                assert sum(q * 512 ** (S - 1 - i) for i, q in enumerate(d)) == x
            j = rng.randrange(1, h + 1)
            sums = [sum(digits[j * q % p][s] * vd[q - 1][d - s] for q in range(1, h + 1) for s in range(d + 1))
                    for d in range(S)]
            exact = sum(table[j * q % p] * v[q - 1] for q in range(1, h + 1))  # in 2^-62
            # in units: the last diagonal's shift drops less than one; the pairs s + t = d > 6, of which there
            # are 13 - d a product, at most (13 - d) 2^16 512^(12 - d) 2^-62 each product
            dropped = sum((13 - d) << 16 + 9 * (12 - d) for d in range(S, 13))
            assert abs((together(sums) << 62) - exact) <= (1 << 62) + h * dropped
