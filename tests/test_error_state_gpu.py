"""A call that failed leaves nothing behind: the next one on the same thread succeeds."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_next_call_after_a_cuda_error(gsn, cuda_device):
    import torch
    from gpusnarks_gb300.batch import fill_random
    pageable = np.zeros(64, dtype=np.uint32)
    f = gsn.BLS12_381
    x = torch.empty(f.limbs << 6, dtype=torch.int32, device="cuda")
    assert gsn.load().gsn_host_free(ctypes.c_void_p(pageable.ctypes.data)) == 5  # GSN_ERR_CUDA: not page-locked
    fill_random(f, x, 1)
    want = x.clone()
    assert gsn.load().gsn_host_free(ctypes.c_void_p(pageable.ctypes.data)) == 5
    w = pow(f.generator, 5 * ((f.p - 1) >> 6), f.p)  # a root whose tables have to be built
    gsn.ntt(f, x, omega=w)
    gsn.ntt(f, x, direction=gsn.INVERSE, omega=w)
    assert torch.equal(x, want)
