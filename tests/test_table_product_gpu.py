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


@pytest.mark.parametrize("fname,radix", [("bls12_381_fr", [5, 4, 2]), ("mnt4753_fr", [3, 6])])
def test_capture_before_the_split_has_its_tables(gsn, cuda_device, tmp_path, fname, radix):
    """A plan whose pass tables do not exist yet is captured: the call reads the full table instead of building them,
    and gives what the uncaptured call gives afterwards."""
    import json

    import torch
    from gpusnarks_gb300._lib import TUNING_FILE
    from gpusnarks_gb300.batch import fill_random
    f = gsn.FIELDS[fname]
    log_n, npass = sum(radix), len(radix)
    pad = lambda v: v + [0] * (4 - len(v))  # noqa: E731
    x = torch.empty((1 << log_n) * f.limbs, dtype=torch.int32, device="cuda")
    fill_random(f, x, 0x5EED0C00)
    data, scratch, want = torch.empty_like(x), torch.empty_like(x), x.clone()
    gsn.ntt(f, want, direction=gsn.INVERSE)  # another split; builds the full table
    try:
        plan = {"field": f.fid, "mode": 0, "log_n": log_n, "kernel": 0, "e_log": 4, "npass": npass,
                "radix_log": pad(radix), "log_j": pad([1] * npass), "block": pad([64] * npass), "ms": 1.0}
        path = tmp_path / "plan.json"
        path.write_text(json.dumps({"device": "test", "plans": [plan]}))
        gsn.load_tuning(path)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            gsn.ntt(f, data, direction=gsn.INVERSE, scratch=scratch)
        data.copy_(x)
        graph.replay()
        assert torch.equal(data, want)
        data.copy_(x)
        gsn.ntt(f, data, direction=gsn.INVERSE, scratch=scratch)
        assert torch.equal(data, want)
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)
