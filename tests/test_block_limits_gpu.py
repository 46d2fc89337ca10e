"""Plans with blocks up to the largest that a table may name, and one-limb tiles of every radix and width (radix-4
sub-steps, odd and even): against the oracle.  Exact."""
import json

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _check(gsn, tmp_path, fid, radix, lj, block):
    from gpusnarks_gb300._lib import TUNING_FILE
    f = gsn.BY_ID[fid]
    log_n, npass = sum(radix), len(radix)
    pad = lambda v: v + [0] * (4 - len(v))  # noqa: E731
    ljs = [min(lj, sum(radix[i + 1:]) if i < npass - 1 else (radix[0] if npass > 1 else 0)) for i in range(npass)]
    plan = {"field": fid, "mode": 0, "log_n": log_n, "kernel": 0, "e_log": 4, "npass": npass, "radix_log": pad(radix),
            "log_j": pad(ljs), "block": pad([block] * npass), "ms": 1.0}
    path = tmp_path / "plan.json"
    path.write_text(json.dumps({"device": "test", "plans": [plan]}))
    x = f.random_array(1 << log_n, seed=0x5EED1100 + 16 * log_n + lj)
    try:
        gsn.clear_tuning()
        gsn.load_tuning(path)
        d = gsn.to_device(x)
        gsn.ntt(f, d)
        assert np.array_equal(gsn.to_host(d).reshape(x.shape), O.ntt(fid, x).reshape(x.shape))
        gsn.ntt(f, d, direction=gsn.INVERSE)
        assert np.array_equal(gsn.to_host(d).reshape(x.shape), x)
        gsn.ntt(f, d, direction=gsn.COSET_FORWARD)
        want = O.coset_ntt(fid, x, O.GENERATORS[fid]).reshape(x.shape)
        assert np.array_equal(gsn.to_host(d).reshape(x.shape), want)
        gsn.ntt(f, d, direction=gsn.COSET_INVERSE)
        assert np.array_equal(gsn.to_host(d).reshape(x.shape), x)
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)


@pytest.mark.parametrize("fid,block", [(0, 1024), (0, 32), (1, 1024), (2, 512), (2, 544), (2, 672)])
def test_largest_blocks(gsn, cuda_device, tmp_path, fid, block):
    _check(gsn, tmp_path, fid, [5, 6], 2, block)


@pytest.mark.parametrize("lj", [0, 1, 2, 3])
@pytest.mark.parametrize("radix", [[1], [2], [3], [8], [11], [1, 2], [2, 1], [4, 5], [8, 7], [9, 6], [10, 5], [3, 4, 6]])
def test_one_limb_tiles(gsn, cuda_device, tmp_path, radix, lj):
    _check(gsn, tmp_path, 0, radix, lj, 64)
