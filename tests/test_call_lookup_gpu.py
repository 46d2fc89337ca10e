"""Calls are resolved by the values of their arguments: other roots, shifts, directions, alignments and plans in turn,
refused ones among them, give what first calls give, also after the caches are released.  Exact."""
import json

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fname,log_n", [("p32", 9), ("bls12_381_fr", 6), ("mnt4753_fr", 5)])
def test_calls_in_turn(gsn, cuda_device, tmp_path, fname, log_n):
    import torch
    from gpusnarks_gb300._lib import TUNING_FILE
    f, n = gsn.FIELDS[fname], 1 << log_n
    x = f.random_array(n, seed=0x5EED0F00 + log_n)
    roots = [None] + [pow(f.root(log_n), e, f.p) for e in (1, 3, 5)]
    want = {}
    for i, w in enumerate(roots):
        wx = w if w is not None else f.root(log_n)
        want[i, 0] = O.ntt(f.fid, x, omega=O.to_limbs(f.fid, wx)).reshape(-1)
    bad = [pow(f.root(log_n), 2, f.p), 1, f.p]

    def go():
        for rep in range(2):
            for i, w in enumerate(roots):
                buf = torch.zeros(n * f.limbs + 1, dtype=torch.int32, device="cuda")
                d = buf[1:] if f.limbs == 1 and rep else buf[:-1]
                d.copy_(gsn.to_device(x).reshape(-1))
                gsn.ntt(f, d, omega=w)
                assert np.array_equal(gsn.to_host(d).reshape(-1), want[i, 0]), (i, rep)
                with pytest.raises(gsn.GsnError):
                    gsn.ntt(f, d, omega=bad[(i + rep) % 3])
                gsn.ntt(f, d, omega=w, direction=gsn.INVERSE)
                assert np.array_equal(gsn.to_host(d).reshape(-1), x.reshape(-1))
                with pytest.raises(gsn.GsnError):
                    gsn.ntt(f, d, omega=w, direction=gsn.COSET_FORWARD, shift=0)
                for s in (None, 2, 3):
                    gsn.ntt(f, d, omega=w, direction=gsn.COSET_FORWARD, shift=s)
                    gsn.ntt(f, d, omega=w, direction=gsn.COSET_INVERSE, shift=s)
                    assert np.array_equal(gsn.to_host(d).reshape(-1), x.reshape(-1))

    try:
        go()
        a, b = log_n // 2, log_n - log_n // 2
        plan = {"field": f.fid, "mode": 0, "log_n": log_n, "kernel": 0, "e_log": 4, "npass": 2,
                "radix_log": [a, b, 0, 0], "log_j": [1, 1, 0, 0], "block": [32, 32, 0, 0], "ms": 1.0}
        path = tmp_path / "plan.json"
        path.write_text(json.dumps({"device": "test", "plans": [plan]}))
        gsn.load_tuning(path)
        assert gsn.plan(f, log_n)["npass"] == 2
        go()
        assert gsn.load().gsn_release_caches() == 0
        go()
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)


def test_more_shifts_than_are_kept(gsn, cuda_device):
    import torch
    f = gsn.P32
    try:
        for shift in [*range(2, 4202), 2, 3]:
            d = torch.tensor([5, 7], dtype=torch.int32, device="cuda")
            gsn.ntt(f, d, direction=gsn.COSET_FORWARD, shift=shift)
            if shift < 4 or shift > 4090:  # x0 + x1 s, x0 - x1 s
                assert d.tolist() == [5 + 7 * shift, (5 - 7 * shift) % f.p - (1 << 32)], shift
    finally:
        assert gsn.load().gsn_release_caches() == 0
