"""The first calls on a root of the caller's: the first builds the root's powers and stage twiddles, the second the
four-step factors, later ones nothing; prepared roots and batches have all at once.  Same results throughout, exact."""
import numpy as np
import pytest

import oracle as O
from forced_plans import forced, plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fname", ["bls12_381_fr", "mnt4753_fr"])
@pytest.mark.parametrize("radix", [[9], [5, 4], [3, 2, 4], [3, 3, 3]])
def test_tables_of_a_new_root(gsn, cuda_device, tmp_path, fname, radix):
    from gpusnarks_gb300.batch import Batch
    f, log_n = gsn.FIELDS[fname], sum(radix)
    count = gsn.load().gsn_kernel_launch_count
    roots = [pow(f.generator, (2 * i + 3) * ((f.p - 1) >> log_n), f.p) for i in range(2)]
    x = f.random_array(1 << log_n, seed=0x5EED1A00 + log_n + len(radix))
    plain = gsn.to_device(x)
    gsn.load().gsn_release_caches()
    with forced(gsn, tmp_path, plan(f.fid, radix, 1, 64)):
        gsn.ntt(f, plain)  # the default root's tables and the scratch
        built = []
        for _ in range(4):
            d = gsn.to_device(x)
            before = count()
            gsn.ntt(f, d, omega=roots[0])
            built.append(count() - before - len(radix))
            assert np.array_equal(gsn.to_host(d).reshape(x.shape), O.ntt(f.fid, x, roots[0]).reshape(x.shape))
        stages, factors = len(set(radix)), len(radix) - 1
        assert built == [1 + stages, factors, 0, 0]
        before = count()
        gsn.prepare(f, log_n, roots[1])
        assert count() - before == 1 + stages + factors
        d = gsn.to_device(x)
        before = count()
        gsn.ntt(f, d, omega=roots[1])
        assert count() - before == len(radix)
        Batch(f, [(d.data_ptr(), log_n, gsn.INVERSE, f.to_limbs(roots[1]), None)]).launch()
        assert np.array_equal(gsn.to_host(d).reshape(x.shape), x)
