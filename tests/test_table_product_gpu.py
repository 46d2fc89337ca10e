"""Products by table constants at their edges, on the GPU: a two-point coset transform is x0 + s x1, x0 - s x1 for
any shift s, so its table product takes every pair of operands; the inverses divide by 2^k.  Exact."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(f, count, seed):
    rnd = random.Random(seed)
    heavy = [sum((0xFFFFFFFF if rnd.random() < 0.85 else 0) << (32 * k) for k in range(f.limbs)) % f.p
             for _ in range(count)]
    return [1, 2, f.p - 1, f.p - 2, f.p >> 1] + [rnd.randrange(1, f.p) for _ in range(count)] + [v or 1 for v in heavy]


@pytest.mark.parametrize("fname", ["p32", "bls12_381_fr", "mnt4753_fr"])
def test_two_point_coset_takes_any_operands(gsn, cuda_device, fname):
    f = gsn.FIELDS[fname]
    xs = [0] + _values(f, 5, 3)
    for s in _values(f, 5, 4):
        for x1 in xs:
            x0 = xs[(3 * x1 + s) % len(xs)]
            d = gsn.to_device(f.ints_to_array([x0, x1]))
            gsn.ntt(f, d, direction=gsn.COSET_FORWARD, shift=s)
            want = f.ints_to_array([(x0 + s * x1) % f.p, (x0 - s * x1) % f.p])
            assert np.array_equal(gsn.to_host(d).reshape(want.shape), want), (s, x0, x1)
            gsn.ntt(f, d, direction=gsn.COSET_INVERSE, shift=s)
            back = f.ints_to_array([x0, x1])
            assert np.array_equal(gsn.to_host(d).reshape(back.shape), back), (s, x0, x1)


@pytest.mark.parametrize("fname", ["p32", "bls12_381_fr", "mnt4753_fr"])
@pytest.mark.parametrize("log_n", range(0, 12))
def test_inverse_divides_extreme_values(gsn, cuda_device, fname, log_n):
    """The transform of a constant c is (n c, 0, ..., 0): its inverse is c everywhere, for extreme c n."""
    f = gsn.FIELDS[fname]
    n = 1 << log_n
    for v in (1, f.p - 1, n % f.p, (f.p - n) % f.p, f.p >> 1):
        d = gsn.to_device(f.ints_to_array([v] + [0] * (n - 1)))
        gsn.ntt(f, d, direction=gsn.INVERSE)
        want = f.ints_to_array([v * pow(n, -1, f.p) % f.p] * n)
        assert np.array_equal(gsn.to_host(d).reshape(want.shape), want), v
