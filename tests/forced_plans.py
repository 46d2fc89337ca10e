"""A tuning table of the test's own: plans by radix, columns and block, loaded for a while in place of the committed one."""
import contextlib
import json


def plan(field, radix, lj, block, kernel=0, mode=0):
    """2^lj columns per tile where the pass's place allows them (make_split_plan's rule, runtime.cu)."""
    npass = len(radix)
    log_j = []
    for i in range(npass):
        last = i == npass - 1
        log_j.append((0 if npass == 1 else min(lj, radix[0])) if last else min(lj, sum(radix[i + 1:])))
    pad = lambda v: list(v) + [0] * (4 - len(v))  # noqa: E731
    return {"field": field, "mode": mode, "log_n": sum(radix), "kernel": kernel, "e_log": 4, "npass": npass,
            "radix_log": pad(radix), "log_j": pad(log_j), "block": pad([block] * npass), "ms": 1.0}


@contextlib.contextmanager
def forced(gsn, tmp_path, *plans):
    from gpusnarks_gb300._lib import TUNING_FILE
    path = tmp_path / "plans.json"
    path.write_text(json.dumps({"device": "test", "plans": plans}))
    try:
        gsn.clear_tuning()
        gsn.load_tuning(path)
        yield
    finally:
        gsn.clear_tuning()
        if TUNING_FILE.exists():
            gsn.load_tuning(TUNING_FILE)
