"""Plans with four lanes per product (kernel 3, 24 limbs): one to three passes, 1 to 4 columns, blocks that do not divide
a tile's outputs and groups past its end, extreme values, all directions, against the oracle.  Exact."""
import json

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lj", [0, 1, 2])
@pytest.mark.parametrize("radix,block", [([0], 32), ([1], 32), ([2], 32), ([3], 256), ([5], 96), ([7], 256), ([1, 1], 32),
                                         ([2, 3], 64), ([4, 4], 160), ([6, 6], 256), ([3, 2, 4], 128), ([5, 6], 1024)])
def test_lane_plans_match_oracle(gsn, cuda_device, tmp_path, radix, block, lj):
    from gpusnarks_gb300._lib import TUNING_FILE
    f = gsn.MNT4_753
    log_n, npass = sum(radix), len(radix)
    pad = lambda v: v + [0] * (4 - len(v))  # noqa: E731
    ljs = [min(lj, sum(radix[i + 1:]) if i < npass - 1 else (radix[0] if npass > 1 else 0)) for i in range(npass)]
    plan = {"field": 2, "mode": 0, "log_n": log_n, "kernel": 3, "e_log": 4, "npass": npass, "radix_log": pad(radix),
            "log_j": pad(ljs), "block": pad([block] * npass), "ms": 1.0}
    path = tmp_path / "plan.json"
    path.write_text(json.dumps({"device": "test", "plans": [plan]}))
    x = f.random_array(1 << log_n, seed=0x5EED1200 + 8 * log_n + lj)
    x[0] = f.to_limbs(f.p - 1)
    x[-1] = f.to_limbs(f.p - 1 if log_n else 0)
    try:
        gsn.clear_tuning()
        gsn.load_tuning(path)
        assert gsn.plan(f, log_n)["kernel"] == 3
        for direction, want in ((gsn.FORWARD, lambda: O.ntt(2, x)), (gsn.INVERSE, lambda: O.intt(2, x)),
                                (gsn.COSET_FORWARD, lambda: O.coset_ntt(2, x, O.GENERATORS[2])),
                                (gsn.COSET_INVERSE, lambda: O.coset_intt(2, x, O.GENERATORS[2]))):
            d = gsn.to_device(x)
            gsn.ntt(f, d, direction=direction)
            assert np.array_equal(gsn.to_host(d).reshape(x.shape), want().reshape(x.shape)), direction
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)
