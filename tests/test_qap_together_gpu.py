"""The QAP computation's three polynomials in shared launches, against the same steps one call at a time: sizes on both
sides of the line where it goes one by one, several pass counts, arrays that only the generic 32-bit pass takes.  Exact."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fname,log_n", [("p32", 0), ("p32", 3), ("p32", 13), ("p32", 21), ("p32", 22),
                                         ("bls12_381_fr", 0), ("bls12_381_fr", 1), ("bls12_381_fr", 9),
                                         ("bls12_381_fr", 17), ("bls12_381_fr", 18), ("bls12_381_fr", 19),
                                         ("mnt4753_fr", 2), ("mnt4753_fr", 11), ("mnt4753_fr", 16),
                                         ("mnt4753_fr", 17)])
@pytest.mark.parametrize("offset", [0, 1])
def test_qap_equals_its_steps(gsn, cuda_device, fname, log_n, offset):
    import torch
    from gpusnarks_gb300.batch import fill_random
    f, n = gsn.FIELDS[fname], 1 << log_n
    if offset and f.limbs > 1:
        pytest.skip("16-byte alignment is required")
    polys = []
    for i in range(3):
        buf = torch.empty(n * f.limbs + 4, dtype=torch.int32, device="cuda")
        polys.append(buf[offset * (i % 2):][:n * f.limbs])  # 4-byte aligned: two arrays of three stay aligned
        fill_random(f, polys[i], 0x5EED0E00 + 8 * log_n + i)
    want = [x.clone() for x in polys]
    for x in want:
        gsn.ntt(f, x, direction=gsn.INVERSE)
        gsn.ntt(f, x, direction=gsn.COSET_FORWARD)
    gsn.coset_quotient(f, *want)
    gsn.ntt(f, want[0], direction=gsn.COSET_INVERSE)
    gsn.qap_h(f, *polys)
    for got, x in zip(polys, want):
        assert torch.equal(got, x)


def test_qap_refuses_what_its_steps_refuse(gsn, cuda_device):
    import torch
    f = gsn.BLS12_381
    a, b, c = (torch.zeros(8 * f.limbs + 1, dtype=torch.int32, device="cuda") for _ in range(3))
    with pytest.raises(gsn.GsnError):
        gsn.qap_h(f, a[1:], b[:-1], c[:-1])  # misaligned
    with pytest.raises(gsn.GsnError):
        gsn.qap_h(f, a[:-1], b[:-1], a[:-1])  # not distinct
    with pytest.raises(gsn.GsnError):
        gsn.qap_h(f, a[:-1], b[:-1], c[:-1], shift=1)  # Z vanishes on the coset
    with pytest.raises(gsn.GsnError):
        gsn.qap_h(f, a[:-1], b[:-1], c[:-1], shift=f.p)  # not canonical
