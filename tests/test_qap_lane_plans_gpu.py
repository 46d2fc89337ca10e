"""gsn_qap_h at sizes whose tuning table names four lanes per product: above 2^12 its last transform takes a split of its
own.  Up to the largest size of the field the result is that of the committed plans.  Exact."""
import pytest

from forced_plans import forced, plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radix", [[6, 7], [8, 8], [6, 6, 5], [8, 7, 7], [8, 7, 8], [8, 8, 8]])
def test_qap_under_lane_plans(gsn, cuda_device, tmp_path, radix):
    import torch
    from gpusnarks_gb300.batch import fill_random
    f, log_n = gsn.MNT4_753, sum(radix)
    polys = [torch.empty(f.limbs << log_n, dtype=torch.int32, device="cuda") for _ in range(3)]
    want = None
    try:
        for table in ([], [plan(2, radix, 1, 128, kernel=3)]):
            for i, x in enumerate(polys):
                fill_random(f, x, 0x5EED1400 + 4 * log_n + i)
            if not table:
                gsn.qap_h(f, *polys)
                want = [x.clone() for x in polys]
                continue
            with forced(gsn, tmp_path, *table):
                assert gsn.plan(f, log_n)["kernel"] == 3
                gsn.qap_h(f, *polys)
            for x, w in zip(polys, want):
                assert torch.equal(x, w)
    finally:
        gsn.load().gsn_release_caches()  # tens of GB of tables and scratch at 2^24
