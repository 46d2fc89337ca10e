"""A server's warm-up over sizes whose requests run by per-pass launches: four-lane, register-blocked 32-bit and generic
plans, then requests of each; sizes beyond the field's are refused.  Against the plain path, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fname,sizes", [("p32", (4, 12, 18)), ("bls12_381_fr", (3, 11)), ("mnt4753_fr", (2, 9, 15))])
def test_warm_up_of_per_pass_requests(gsn, cuda_device, fname, sizes):
    from gpusnarks_gb300.serve import Server
    f = gsn.FIELDS[fname]
    srv = Server(1 << 30, max_inflight=2, max_launch_work=1)
    try:
        srv.warmup(f, sizes[0], sizes[-1])
        with pytest.raises(gsn.GsnError):
            srv.warmup(f, 64, 64)
        for k in sizes:
            x = f.random_array(1 << k, seed=0x5EED1800 + k)
            out = np.empty_like(x)
            rid = srv.submit(f, x, gsn.INVERSE, host_out=out)
            srv.wait(rid)
            srv.release(rid)
            d = gsn.to_device(x)
            gsn.ntt(f, d, direction=gsn.INVERSE)
            assert np.array_equal(out.reshape(-1), gsn.to_host(d).reshape(-1)), k
    finally:
        srv.close()


_FRESH = """
import numpy as np, torch, gpusnarks_gb300 as g
from gpusnarks_gb300.serve import Server
f = g.FIELDS["{field}"]
busy = torch.empty(1 << 28, dtype=torch.float32, device="cuda")
srv = Server(1 << 30, max_inflight=2, max_launch_work=1)
srv.warmup(f, {k}, {k})
x = f.random_array(1 << {k}, seed=3)
out = np.empty_like(x)
busy.add_(1.0)
torch.cuda.synchronize()
for _ in range(300):  # some 90 ms of another stream's work
    busy.add_(1.0)
rid = srv.submit(f, x, 0, host_out=out)
srv.wait(rid)
srv.release(rid)
print(srv.stats()["step_max_s"][4])
srv.close()
"""


@pytest.mark.parametrize("field,k", [("p32", 18), ("mnt4753_fr", 9)])
def test_warm_up_loads_the_code(gsn, cuda_device, field, k):
    """In a fresh process the first launch after a warm-up does not wait for other streams' work to load its kernel."""
    import pathlib
    import subprocess
    import sys
    root = pathlib.Path(__file__).resolve().parent.parent
    run = subprocess.run([sys.executable, "-c", _FRESH.format(field=field, k=k)], cwd=root, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stderr
    assert float(run.stdout) < 0.02
