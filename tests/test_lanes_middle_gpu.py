"""Four-lane plans with a pass of radix 2 in the middle, which reads and writes the scratch in place: tiles of 2 to 16
outputs per column pair and more than one warp or loop round per tile, all directions, against the oracle.  Exact."""
import numpy as np
import pytest

import oracle as O
from forced_plans import forced, plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [32, 96, 128, 256])
@pytest.mark.parametrize("radix,lj", [([4, 1, 4], 3), ([4, 1, 5], 4), ([3, 1, 1, 3], 3), ([2, 1, 2], 2), ([1, 1, 5], 5),
                                      ([1, 1, 1], 1)])
def test_middle_pass_of_radix_two(gsn, cuda_device, tmp_path, radix, lj, block):
    f = gsn.MNT4_753
    x = f.random_array(1 << sum(radix), seed=0x5EED1300 + 16 * sum(radix) + lj)
    want = {gsn.FORWARD: O.ntt(2, x), gsn.INVERSE: O.intt(2, x),
            gsn.COSET_FORWARD: O.coset_ntt(2, x, O.GENERATORS[2]),
            gsn.COSET_INVERSE: O.coset_intt(2, x, O.GENERATORS[2])}
    with forced(gsn, tmp_path, plan(2, radix, lj, block, kernel=3)):
        p = gsn.plan(f, sum(radix))
        assert p["kernel"] == 3 and p["radix_log"][:len(radix)] == radix
        for direction, w in want.items():
            d = gsn.to_device(x)
            gsn.ntt(f, d, direction=direction)
            assert np.array_equal(gsn.to_host(d).reshape(x.shape), w.reshape(x.shape)), direction
