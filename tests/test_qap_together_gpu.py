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


@pytest.mark.parametrize("fname,log_n", [("p32", 13), ("bls12_381_fr", 12), ("mnt4753_fr", 10)])
@pytest.mark.parametrize("warm", [False, True])
def test_captured_calls_keep_their_scratch(gsn, cuda_device, fname, log_n, warm):
    """A QAP computation and a sum are captured on a stream that has a transform's scratch (`warm`: their own too), and
    eager ones after that leave the scratch of the captured transforms where it is."""
    import torch
    from gpusnarks_gb300.batch import fill_random
    f, n = gsn.FIELDS[fname], 1 << log_n
    x = [torch.empty(n * f.limbs, dtype=torch.int32, device="cuda") for _ in range(4)]
    for i, v in enumerate(x):
        fill_random(f, v, 0x5EED0E80 + 8 * log_n + i)
    want = [v.clone() for v in x]
    gsn.qap_h(f, *want[:3])
    gsn.ntt(f, want[3])
    total = gsn.multiexp(f, x[0], x[1]).clone()
    got, out = [v.clone() for v in x], torch.zeros_like(total)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def work():
        gsn.multiexp(f, got[0], got[1], out=out)
        gsn.qap_h(f, *got[:3])
        gsn.ntt(f, got[3])

    with torch.cuda.stream(stream):
        gsn.ntt(f, x[3].clone())
        if warm:
            work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        work()
    for rep in range(2):
        with torch.cuda.stream(stream):
            for v, w in zip(got, x):
                v.copy_(w)
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, total), rep
        assert torch.equal(got[3], want[3]) and torch.equal(got[0], want[0]), rep
        with torch.cuda.stream(stream):
            gsn.qap_h(f, *(v.clone() for v in x[:3]))
            gsn.multiexp(f, x[0], x[1])
        torch.cuda.synchronize()
