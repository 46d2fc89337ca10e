"""The tuner keeps the pass tables of the plan it picks, not those of every candidate."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
def test_candidates_tables_are_freed(gsn, cuda_device, batched):
    import torch
    from gpusnarks_gb300._lib import TUNING_FILE
    from gpusnarks_gb300.batch import fill_random
    f, log_n = gsn.BLS12_381, 19
    x = torch.empty(f.limbs << log_n, dtype=torch.int32, device="cuda")
    fill_random(f, x, 0x5EED1700)
    want = x.clone()
    gsn.load().gsn_release_caches()
    gsn.clear_tuning()
    try:
        tune = gsn.load().gsn_autotune_batch if batched else gsn.load().gsn_autotune
        assert tune(f.fid, 5, 5, 1) == 0  # loads the kernels; builds the default root's table
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        assert tune(f.fid, log_n, log_n, 1) == 0
        kept = free - torch.cuda.mem_get_info()[0]
        assert kept <= 64 * 2**log_n * 3 // 2 + (16 << 20)  # the factors of one split
        gsn.ntt(f, x)
        gsn.ntt(f, x, direction=gsn.INVERSE)
        assert torch.equal(x, want)
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)
        gsn.load().gsn_release_caches()
