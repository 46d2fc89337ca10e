"""Device tables when memory runs out: tables that nobody holds make room for what a call needs, and what a captured graph,
a batch or a running call holds stays.  Exact round trips."""
import contextlib
import threading

import pytest

pytestmark = pytest.mark.gpu

LOG_N = 20  # BLS12-381: 32 MB of data; 64 MB per table of a root or shift, and 64 MB of four-step factors per root


@contextlib.contextmanager
def memory_left(gsn, megabytes):
    """All device memory but this much taken, the library's caches empty."""
    import torch
    gsn.load().gsn_release_caches()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (megabytes << 20), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()
        gsn.load().gsn_release_caches()


def _root(f, i):
    return pow(f.generator, (2 * i + 3) * ((f.p - 1) >> LOG_N), f.p)


def _array(f, seed):
    import torch
    from gpusnarks_gb300.batch import fill_random
    x = torch.empty(f.limbs << LOG_N, dtype=torch.int32, device="cuda")
    fill_random(f, x, seed)
    return x


def _round_trip(gsn, f, x, want, w, shift, scratch=None):
    import torch
    gsn.ntt(f, x, direction=gsn.COSET_FORWARD, omega=w, shift=shift, scratch=scratch)
    gsn.ntt(f, x, direction=gsn.COSET_INVERSE, omega=w, shift=shift, scratch=scratch)
    torch.cuda.current_stream().synchronize()
    assert torch.equal(x, want)


def test_unused_tables_make_room(gsn, cuda_device):
    f = gsn.BLS12_381
    x = _array(f, 0x5EED1600)
    want = x.clone()
    _round_trip(gsn, f, x, want, _root(f, 90), 3)
    with memory_left(gsn, 1200):
        for i in range(24):  # 24 (64 + 64 + 2 * 64) MB of tables
            _round_trip(gsn, f, x, want, _root(f, i), 5 + i)


def test_calls_do_without_optional_tables(gsn, cuda_device):
    import torch
    f = gsn.BLS12_381
    x = _array(f, 0x5EED1601)
    want = x.clone()
    gsn.ntt(f, x, omega=_root(f, 1))
    image, got = x.clone(), x.clone()
    with memory_left(gsn, 112):  # the root's powers and the scratch fit, the four-step factors do not
        for _ in range(3):
            got.copy_(want)
            gsn.ntt(f, got, omega=_root(f, 1))
    assert torch.equal(got, image)


def test_prepare_builds_what_there_was_no_memory_for(gsn, cuda_device):
    import torch
    f = gsn.BLS12_381
    x = _array(f, 0x5EED1602)
    w = _root(f, 2)
    gsn.ntt(f, x, omega=w)
    gsn.load().gsn_release_caches()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (112 << 20), dtype=torch.uint8, device="cuda")
    try:
        gsn.ntt(f, x, omega=w, direction=gsn.INVERSE)
        torch.cuda.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()
    count = gsn.load().gsn_kernel_launch_count
    before = count()
    gsn.prepare(f, LOG_N, w)
    assert count() > before


def test_held_tables_stay(gsn, cuda_device):
    """A captured call, a batch and the prepared default tables keep theirs while others' are given back."""
    import torch
    from gpusnarks_gb300.batch import Batch
    f = gsn.BLS12_381
    x, y, z, scratch = _array(f, 0x5EED1603), _array(f, 0x5EED1604), _array(f, 0x5EED1605), _array(f, 1)
    src, want_y, want_z = x.clone(), y.clone(), z.clone()
    w, wb = _root(f, 40), _root(f, 41)
    _round_trip(gsn, f, z, want_z, _root(f, 90), 3, scratch)
    with memory_left(gsn, 1500):
        gsn.ntt(f, x, omega=w, scratch=scratch)
        image = x.clone()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            gsn.ntt(f, x, omega=w, scratch=scratch)
        batch = Batch(f, [(y.data_ptr(), LOG_N, gsn.FORWARD, f.to_limbs(wb), None)])
        gsn.ntt(f, y, omega=wb, direction=gsn.INVERSE, scratch=scratch)
        for i in range(16):
            _round_trip(gsn, f, z, want_z, _root(f, i), 5 + i, scratch)
            x.copy_(src)
            graph.replay()
            batch.launch()
            torch.cuda.synchronize()
            assert torch.equal(x, image) and torch.equal(y, want_y)
            gsn.ntt(f, y, omega=wb, direction=gsn.INVERSE, scratch=scratch)
        del batch, graph


def test_threads_under_pressure(gsn, cuda_device):
    import torch
    f, errors = gsn.BLS12_381, []
    arrays = [(_array(f, 0x5EED1610 + t), _array(f, 2)) for t in range(4)]
    wants = [x.clone() for x, _ in arrays]
    _round_trip(gsn, f, *arrays[0][:1], wants[0], _root(f, 90), 3, arrays[0][1])
    torch.cuda.synchronize()

    def work(t):
        try:
            x, scratch = arrays[t]
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(12):
                    _round_trip(gsn, f, x, wants[t], _root(f, 4 * i + t), 7 + 4 * i + t, scratch)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    with memory_left(gsn, 2400):
        threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(120)
        assert not any(t.is_alive() for t in threads)
    assert not errors, errors[0]


def test_tables_are_bounded(gsn, cuda_device):
    """A shift drawn anew for every call: what is kept of them stays within half of the device's memory."""
    import torch
    from gpusnarks_gb300.batch import fill_random
    f, log_n = gsn.BLS12_381, 24  # 1 GiB per shift
    x = torch.empty(f.limbs << log_n, dtype=torch.int32, device="cuda")
    fill_random(f, x, 0x5EED1620)
    want = x.clone()
    gsn.ntt(f, x)
    gsn.ntt(f, x, direction=gsn.INVERSE)
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    least = free
    try:
        for i in range((total >> 30) * 11 // 20):
            gsn.ntt(f, x, direction=gsn.COSET_FORWARD, shift=3 + i)
            least = min(least, torch.cuda.mem_get_info()[0])
        assert free - least <= total // 2 + (4 << 30)
        x.copy_(want)
        gsn.ntt(f, x, direction=gsn.COSET_FORWARD, shift=3)
        gsn.ntt(f, x, direction=gsn.COSET_INVERSE, shift=3)
        assert torch.equal(x, want)
    finally:
        gsn.load().gsn_release_caches()
