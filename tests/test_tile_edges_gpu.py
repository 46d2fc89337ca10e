"""The multi-limb tile (kernel 0) at the edges of its values and shapes, through forced plans: radices 2^1..2^11 in one
pass, two to four passes, 1 to 8 columns, blocks from a warp to the register cap, all directions.  The inputs drive the
unreduced sums and differences to their bounds: all p - 1, 0 and p - 1 in turn at several distances, carry-heavy limbs.
Against the oracle, exact."""
import functools

import numpy as np
import pytest

import oracle as O
from forced_plans import forced, plan

pytestmark = pytest.mark.gpu

SHAPES = ([([r], 0, b) for r, b in zip(range(1, 12), (32, 32, 64, 32, 96, 128, 64, 256, 128, 512, 128))] +
          [([1, 10], 1, 128), ([10, 1], 0, 64), ([11, 1], 0, 256), ([1, 11], 0, 128), ([8, 3], 3, 128), ([5, 6], 3, 64),
           ([4, 5], 2, 32), ([7, 4], 1, 128), ([3, 4, 5], 2, 128), ([2, 7, 3], 3, 64), ([1, 1, 9], 1, 32),
           ([3, 1, 4], 3, 96), ([2, 3, 2, 3], 2, 128), ([4, 1, 1, 4], 3, 32)])


def _inputs(f, n):
    """Name -> array of n elements."""
    top = f.p - 1
    heavy = [v % f.p for v in (sum((0xFFFFFFFF if (j + k) % 3 else 0) << (32 * j) for j in range(f.limbs)) for k in range(3))]
    i = np.arange(n)
    return {"top": f.ints_to_array([top] * n),
            "turn 1": f.ints_to_array([top * int(v) for v in i & 1]),
            "turn n/2": f.ints_to_array([top * int(v) for v in (i >= n // 2)]),
            "turn 4": f.ints_to_array([0 if (int(v) >> 2) & 1 else top for v in i]),
            "heavy": f.ints_to_array([heavy[int(v) % 3] if v % 5 else 1 for v in i])}


@functools.lru_cache(maxsize=None)
def _wanted(fid, log_n):
    import gpusnarks_gb300 as g
    f = next(x for x in g.FIELDS.values() if x.fid == fid)
    out = []
    for name, x in _inputs(f, 1 << log_n).items():
        out.append((name, x, {g.FORWARD: O.ntt(fid, x), g.INVERSE: O.intt(fid, x),
                              g.COSET_FORWARD: O.coset_ntt(fid, x, O.GENERATORS[fid]),
                              g.COSET_INVERSE: O.coset_intt(fid, x, O.GENERATORS[fid])}))
    return out


@pytest.mark.parametrize("radix,lj,block", SHAPES)
@pytest.mark.parametrize("fname", ["bls12_381_fr", "mnt4753_fr"])
def test_extreme_values(gsn, cuda_device, tmp_path, fname, radix, lj, block):
    f, log_n = gsn.FIELDS[fname], sum(radix)
    with forced(gsn, tmp_path, plan(f.fid, radix, lj, block)):
        p = gsn.plan(f, log_n)
        assert p["kernel"] == 0 and p["radix_log"][:len(radix)] == radix and p["block"][0] == block
        for name, x, want in _wanted(f.fid, log_n):
            for direction, w in want.items():
                d = gsn.to_device(x)
                gsn.ntt(f, d, direction=direction)
                assert np.array_equal(gsn.to_host(d).reshape(x.shape), w.reshape(x.shape)), (name, direction)


@pytest.mark.parametrize("fname", ["bls12_381_fr", "mnt4753_fr"])
def test_two_point_products_on_the_tile(gsn, cuda_device, tmp_path, fname):
    """A two-point coset transform is x0 + s x1, x0 - s x1 for any shift s: the table product takes every pair of operands."""
    f = gsn.FIELDS[fname]
    p = f.p
    heavy = [sum((0xFFFFFFFF if (j + k) % 4 else 0) << (32 * j) for j in range(f.limbs)) % p for k in range(4)]
    values = [1, 2, p - 1, p - 2, p >> 1, (1 << 32) - 1, p >> 31] + heavy
    with forced(gsn, tmp_path, plan(f.fid, [1], 0, 32)):
        assert gsn.plan(f, 1)["kernel"] == 0
        for s in values:
            for x1 in [0] + values:
                x0 = values[(x1 + 3 * s) % len(values)]
                d = gsn.to_device(f.ints_to_array([x0, x1]))
                gsn.ntt(f, d, direction=gsn.COSET_FORWARD, shift=s)
                want = f.ints_to_array([(x0 + s * x1) % p, (x0 - s * x1) % p])
                assert np.array_equal(gsn.to_host(d).reshape(want.shape), want), (s, x0, x1)
                gsn.ntt(f, d, direction=gsn.COSET_INVERSE, shift=s)
                want = f.ints_to_array([x0, x1])
                assert np.array_equal(gsn.to_host(d).reshape(want.shape), want), (s, x0, x1)
