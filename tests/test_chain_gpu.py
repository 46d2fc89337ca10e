"""Kernels that overlap their predecessor's end (chain.cuh): calls queued back to back between a caller's own kernels,
with no synchronisation, see each other's results.  Exact."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("fname,log_n", [("p32", 7), ("p32", 16), ("bls12_381_fr", 4), ("bls12_381_fr", 12),
                                         ("mnt4753_fr", 9)])
def test_queued_calls_see_their_predecessors(gsn, cuda_device, fname, log_n, side):
    import torch
    from gpusnarks_gb300.batch import fill_random
    f, n = gsn.FIELDS[fname], 1 << log_n
    x = torch.empty(n * f.limbs, dtype=torch.int32, device="cuda")
    fill_random(f, x, 0x5EED0D00 + log_n)
    ones = gsn.to_device(f.ints_to_array([1] * n)).reshape(-1)
    gsn.ntt(f, x.clone()), gsn.ntt(f, x.clone(), direction=gsn.INVERSE)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    with torch.cuda.stream(stream):
        buf, total = torch.empty_like(x), torch.zeros_like(x[:f.limbs])
        for i in range(40):
            want = torch.roll(x, i * f.limbs)
            buf.fill_(-1)
            buf.copy_(want)  # the caller's own kernel, then ours, with nothing between
            gsn.ntt(f, buf)
            gsn.pointwise_mul(f, buf, ones)
            gsn.ntt(f, buf, direction=gsn.INVERSE)
            gsn.multiexp(f, buf, ones, out=total)
            bad += (buf != want).sum()
            if i == 0:
                first = total.clone()
            bad += (total != first).sum()  # the sum of the elements does not depend on their order
    torch.cuda.synchronize()
    assert int(bad) == 0
