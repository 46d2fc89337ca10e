"""Multi-exponentiations over carry-heavy operands (limbs of 0xFFFFFFFF and 0, halves whose sums carry) and lengths around the
blocks' and threads' shares, both representations, against Python integers.  Exact."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 257, 4099, 40000])
@pytest.mark.parametrize("fname", ["p32", "bls12_381_fr", "mnt4753_fr"])
def test_heavy_operands(gsn, cuda_device, fname, n, mode):
    f, rnd = gsn.FIELDS[fname], random.Random(n + 7 * mode)
    pool = [f.p - 1, f.p - 2, 1, (1 << (16 * f.limbs)) - 1, f.p - 1 - ((1 << (16 * f.limbs)) - 1)]
    pool += [sum((0xFFFFFFFF if rnd.random() < 0.85 else 0) << (32 * k) for k in range(f.limbs)) % f.p for _ in range(40)]
    pool += [rnd.randrange(f.p) for _ in range(20)]
    ia, ib = ([rnd.randrange(len(pool)) for _ in range(n)] for _ in range(2))
    table = f.ints_to_array(pool).reshape(len(pool), -1)
    a, b = gsn.to_device(table[ia]), gsn.to_device(table[ib])
    got = f.from_limbs(gsn.to_host(gsn.multiexp(f, a, b, mode=mode)))
    want = sum(pool[i] * pool[j] for i, j in zip(ia, ib)) % f.p
    assert got == (want if mode == 0 else want * pow(f.R, -1, f.p) % f.p)
