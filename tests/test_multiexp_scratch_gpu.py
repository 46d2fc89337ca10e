"""A captured transform keeps its scratch when a multi-exponentiation follows on its stream: also when that scratch is
smaller than one block's sums.  Exact."""
import numpy as np
import pytest

import oracle as O
from forced_plans import forced, plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fname,radix", [("p32", [1, 1]), ("p32", [2, 2]), ("bls12_381_fr", [1, 1]), ("mnt4753_fr", [1, 1])])
def test_captured_transform_keeps_its_scratch(gsn, cuda_device, tmp_path, fname, radix):
    import torch
    f, g = gsn.FIELDS[fname], gsn.MNT4_753
    log_n = sum(radix)
    x = f.random_array(1 << log_n, seed=0x5EED1500 + log_n)
    a, b = (gsn.to_device(g.random_array(3000, seed=0x5EED1501 + i)) for i in range(2))
    want_sum = gsn.to_host(gsn.multiexp(g, a, b))
    data, src = gsn.to_device(x), gsn.to_device(x)
    with forced(gsn, tmp_path, plan(f.fid, radix, 1, 32)):
        assert gsn.plan(f, log_n)["npass"] == 2
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            gsn.ntt(f, data)  # the stream's scratch
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            gsn.ntt(f, data)
        want = O.ntt(f.fid, x)
        for _ in range(2):
            with torch.cuda.stream(stream):
                got_sum = gsn.multiexp(g, a, b)
            torch.cuda.synchronize()
            data.copy_(src)
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(gsn.to_host(data).reshape(x.shape), want.reshape(x.shape))
            assert np.array_equal(gsn.to_host(got_sum), want_sum)
