"""Host threads in the middle of their transforms while another loads and clears tuning tables: every call runs one plan
or the other, with that plan's tables and scratch.  Exact round trips."""
import json
import threading

import pytest

from forced_plans import plan

pytestmark = pytest.mark.gpu


def test_plans_change_under_running_threads(gsn, cuda_device, tmp_path):
    import torch
    from gpusnarks_gb300._lib import TUNING_FILE
    from gpusnarks_gb300.batch import fill_random
    tables = []
    for i, radices in enumerate((([5, 6], [4, 7], [3, 4, 4]), ([11], [6, 5], [2, 9]))):
        path = tmp_path / f"plans{i}.json"
        path.write_text(json.dumps({"device": "test", "plans": [plan(fid, r, 1, 64) for fid, r in enumerate(radices)]}))
        tables.append(path)
    errors, stop = [], threading.Event()

    def work(f, seed):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                x = torch.empty(f.limbs << 11, dtype=torch.int32, device="cuda")
                fill_random(f, x, seed)
                want = x.clone()
                w = pow(f.generator, 3 * ((f.p - 1) >> 11), f.p)
                for i in range(150):
                    own = {"omega": w} if i % 3 else {}
                    gsn.ntt(f, x, direction=gsn.COSET_FORWARD, **own)
                    gsn.ntt(f, x, direction=gsn.COSET_INVERSE, **own)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(x, want)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    def change():
        try:
            while not stop.is_set():
                for path in tables:
                    gsn.load_tuning(path)
                gsn.clear_tuning()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    changer = threading.Thread(target=change)
    threads = [threading.Thread(target=work, args=(f, 0x5EED1900 + i)) for i, f in enumerate([gsn.P32, gsn.BLS12_381, gsn.MNT4_753] * 2)]
    try:
        changer.start()
        for t in threads:
            t.start()
        for t in threads:
            t.join(120)
    finally:
        stop.set()
        changer.join(60)
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)
    assert not any(t.is_alive() for t in threads) and not errors, errors
