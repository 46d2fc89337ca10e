"""The calls that programs make of this framework, as cases to measure.

Sizes are those of the repository's own configurations, tests and benchmark: the 32-bit transform of 2^16 and the
2^20..2^28 sweep, the MNT4-753 transform of 2^18, batches of BLS12-381 transforms of 2^10..2^20, prover and serving
requests of both large fields, in every direction.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import gpusnarks_gb300 as g
from gpusnarks_gb300.batch import Batch

_DIRECTIONS = {"forward": g.FORWARD, "inverse": g.INVERSE, "coset_forward": g.COSET_FORWARD,
               "coset_inverse": g.COSET_INVERSE}


def listed():
    return [
        # The plain 32-bit transform of the first configuration: a small call, latency and launches count.
        {"name": "p32_fwd_2e16", "op": "ntt", "field": "p32", "log_n": 16, "dir": "forward", "root": "default"},
        # Product of two polynomials of 2^20 coefficients: two forward transforms, a product, an inverse.
        {"name": "p32_polymul_2e21", "op": "polymul", "field": "p32", "log_n": 21},
        # The large end of the 32-bit sweep, 256 MB resident.
        {"name": "p32_fwd_2e26", "op": "ntt", "field": "p32", "log_n": 26, "dir": "forward", "root": "default"},
        # Smallest batch-class polynomial on its own, back to coefficients: launch latency and an idle chip.
        {"name": "bls_inv_2e10", "op": "ntt", "field": "bls12_381_fr", "log_n": 10, "dir": "inverse",
         "root": "default"},
        # The common prover domain, evaluated with a root that the caller names (best_fft always passes one).
        {"name": "bls_fwd_2e20", "op": "ntt", "field": "bls12_381_fr", "log_n": 20, "dir": "forward", "root": "own"},
        # The prover's H polynomial: three inverses, three coset transforms, the quotient, a coset inverse.
        {"name": "bls_qap_2e16", "op": "qap", "field": "bls12_381_fr", "log_n": 16},
        # Many transforms of uneven sizes and all directions in one persistent launch.
        {"name": "bls_batch_256", "op": "batch", "field": "bls12_381_fr", "jobs": 256, "lo": 10, "hi": 16, "mix": 7},
        # A small serving request of the 753-bit field on a coset.
        {"name": "mnt4_coset_2e12", "op": "ntt", "field": "mnt4753_fr", "log_n": 12, "dir": "coset_forward",
         "root": "default"},
        # The headline: one forward transform of the reference's 768-bit field setup.
        {"name": "mnt4_fwd_2e18", "op": "ntt", "field": "mnt4753_fr", "log_n": 18, "dir": "forward",
         "root": "default"},
        # A large inverse of the same field.
        {"name": "mnt4_inv_2e20", "op": "ntt", "field": "mnt4753_fr", "log_n": 20, "dir": "inverse",
         "root": "default"},
        # The drop-in on host arrays: several polynomials in page-locked memory, copies in and out included.
        {"name": "mnt4_host_4x2e18", "op": "host", "field": "mnt4753_fr", "log_n": 18, "arrays": 4,
         "dir": "forward"},
        # The multi-exponentiation over field elements, a length that is no power of two.
        {"name": "mnt4_multiexp_1000003", "op": "multiexp", "field": "mnt4753_fr", "n": 1000003,
         "mode": "montgomery"},
    ]


_MAX_LOG = {"p32": 26, "bls12_381_fr": 22, "mnt4753_fr": 20}


def draw(rng: random.Random):
    op = rng.choices(["ntt", "qap", "polymul", "batch", "multiexp", "host"], [12, 3, 2, 3, 3, 1])[0]
    field = rng.choice(["p32", "bls12_381_fr", "mnt4753_fr"])
    limbs = g.FIELDS[field].limbs
    if op == "ntt":
        return {"op": op, "field": field, "log_n": rng.randint(4, _MAX_LOG[field]),
                "dir": rng.choice(sorted(_DIRECTIONS)), "root": rng.choice(["default", "own"])}
    if op == "qap":
        return {"op": op, "field": field, "log_n": rng.randint(6, _MAX_LOG[field] - 3)}
    if op == "polymul":
        return {"op": op, "field": field, "log_n": rng.randint(6, _MAX_LOG[field] - 2)}
    if op == "batch":
        lo = rng.randint(6, 11)
        return {"op": op, "field": field, "jobs": int(math.exp(rng.uniform(math.log(3), math.log(200)))), "lo": lo,
                "hi": min(lo + rng.randint(0, 5), {1: 16, 8: 16, 24: 13}[limbs]), "mix": rng.randint(0, 10**6)}
    if op == "multiexp":
        return {"op": op, "field": field, "n": int(math.exp(rng.uniform(math.log(200), math.log(1.6e8 / (4 * limbs))))),
                "mode": rng.choice(["canonical", "montgomery"])}
    return {"op": op, "field": field, "log_n": rng.randint(8, {1: 22, 8: 19, 24: 17}[limbs]),
            "arrays": rng.randint(1, 4), "dir": rng.choice(["forward", "inverse"])}


def _elements(f, n, gen):
    """n uniform elements as a device tensor of little-endian 32-bit limbs, the top limb below the modulus's."""
    top = (f.p >> (32 * (f.limbs - 1))) if f.limbs > 1 else f.p
    x = torch.randint(0, 1 << 32, (n, f.limbs), generator=gen, device="cuda", dtype=torch.int64)
    x[:, -1] = torch.randint(0, top, (n,), generator=gen, device="cuda", dtype=torch.int64)
    return torch.where(x >= 1 << 31, x - (1 << 32), x).to(torch.int32)


def _batch_jobs(case):
    """(log n, direction, first element) of each job and the elements of all."""
    rng = random.Random(case["mix"])
    jobs, at = [], 0
    for _ in range(case["jobs"]):
        k = rng.randint(case["lo"], case["hi"])
        jobs.append((k, rng.choice(sorted(_DIRECTIONS)), at))
        at += 1 << k
    return jobs, at


def _inputs(case, seed):
    f = g.FIELDS[case["field"]]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op = case["op"]
    if op == "ntt":
        return [_elements(f, 1 << case["log_n"], gen)]
    if op == "qap":
        return [_elements(f, 1 << case["log_n"], gen) for _ in range(3)]
    if op == "polymul":
        out = []
        for _ in range(2):  # coefficients in the lower half: the cyclic product is the product
            x = _elements(f, 1 << case["log_n"], gen)
            x[x.shape[0] // 2:] = 0
            out.append(x)
        return out
    if op == "batch":
        return [_elements(f, _batch_jobs(case)[1], gen)]
    if op == "multiexp":
        return [_elements(f, case["n"], gen) for _ in range(2)]
    return [_elements(f, 1 << case["log_n"], gen) for _ in range(case["arrays"])]


def _root(f, log_n):
    return pow(f.generator, (f.p - 1) >> log_n, f.p)


def _own_root(case):
    """The caller's own primitive root (an odd power of the default one), or None."""
    if case.get("root") != "own":
        return None
    f = g.FIELDS[case["field"]]
    return pow(_root(f, case["log_n"]), 5, f.p)


def prepare(case, seed):
    f = g.FIELDS[case["field"]]
    op = case["op"]
    data = _inputs(case, seed)
    state = {"op": op, "field": f, "data": data}
    if op == "ntt":
        w = _own_root(case)
        state["omega"] = None if w is None else f.to_limbs(w)
        state["dir"] = _DIRECTIONS[case["dir"]]
        g.prepare(f, case["log_n"], state["omega"])
    elif op == "batch":
        base, size = data[0].data_ptr(), 4 * f.limbs
        jobs = [(base + at * size, k, _DIRECTIONS[d], None, None) for k, d, at in _batch_jobs(case)[0]]
        state["batch"] = Batch(f, jobs)
    elif op == "multiexp":
        state["mode"] = g.MULTIEXP_MONTGOMERY if case["mode"] == "montgomery" else g.MULTIEXP_CANONICAL
    elif op == "host":
        state["data"] = [x.cpu().pin_memory() for x in data]
        state["log_n"] = case["log_n"]
        state["dir"] = _DIRECTIONS[case["dir"]]
    torch.cuda.synchronize()
    return state


def run(state):
    op, f, data = state["op"], state["field"], state["data"]
    if op == "ntt":
        return g.ntt(f, data[0], direction=state["dir"], omega=state["omega"])
    if op == "qap":
        g.qap_h(f, *data)
        return data
    if op == "polymul":
        for x in data:
            g.ntt(f, x)
        g.pointwise_mul(f, data[0], data[1])
        return [g.ntt(f, data[0], direction=g.INVERSE), data[1]]
    if op == "batch":
        state["batch"].launch()
        return data[0]
    if op == "multiexp":
        return g.multiexp(f, data[0], data[1], mode=state["mode"])
    g.best_fft_many([(x.data_ptr(), state["log_n"]) for x in data], field=f, direction=state["dir"])
    return data


def _products(log_n):
    return (log_n << log_n) // 2


def work(case):
    """Inputs read and outputs written once; each product counted as its limb products, two operations each."""
    limbs = g.FIELDS[case["field"]].limbs
    op, size = case["op"], 4 * limbs
    n = 1 << case.get("log_n", 0)
    if op == "ntt":
        moved, products = 2 * n * size, _products(case["log_n"])
    elif op == "qap":
        moved, products = 6 * n * size, 7 * _products(case["log_n"]) + 6 * n
    elif op == "polymul":
        moved, products = 4 * n * size, 3 * _products(case["log_n"]) + n
    elif op == "batch":
        jobs, total = _batch_jobs(case)
        moved, products = 2 * total * size, sum(_products(k) for k, _, _ in jobs)
    elif op == "multiexp":
        moved, products = 2 * case["n"] * size + size, case["n"]
    else:
        moved, products = 2 * case["arrays"] * n * size, case["arrays"] * _products(case["log_n"])
    return {"bytes": moved, "flops": 2 * limbs * limbs * products}


# --- the same results in plain integers --------------------------------------------------------------------------

def _ints(f, x):
    a = np.ascontiguousarray(x.cpu().numpy()).tobytes()
    size = 4 * f.limbs
    return [int.from_bytes(a[i:i + size], "little") for i in range(0, len(a), size)]


def _tensor(f, xs):
    size = 4 * f.limbs
    a = np.frombuffer(b"".join(int(x).to_bytes(size, "little") for x in xs), dtype=np.int32)
    return torch.from_numpy(a.reshape(-1, f.limbs).copy())


def _dft32(x, w, p):
    """Radix-2 transform of uint64 values below a 32-bit p (products below 2^64)."""
    n = len(x)
    log_n = n.bit_length() - 1
    tw = np.ones(max(1, n // 2), dtype=np.uint64)
    for k in range(log_n - 1):
        tw[1 << k:2 << k] = tw[:1 << k] * np.uint64(pow(w, 1 << k, p)) % np.uint64(p)
    p64, x = np.uint64(p), x.copy()
    for s in range(log_n):  # natural order in, bit-reversed out
        v = x.reshape(1 << s, 2, -1)
        a, b = v[:, 0].copy(), v[:, 1].copy()
        v[:, 0] = (a + b) % p64
        v[:, 1] = (a + p64 - b) % p64 * tw[::1 << s] % p64
    rev = np.zeros(1, dtype=np.int64)
    for _ in range(log_n):
        rev = np.concatenate([2 * rev, 2 * rev + 1])
    return x[rev]


def _dft(x, w, p):
    if len(x) == 1:
        return x
    tw, t = [1], 1
    for _ in range(len(x) // 2 - 1):
        t = t * w % p
        tw.append(t)

    def go(a, step):
        if len(a) == 1:
            return a
        e, o = go(a[::2], 2 * step), go(a[1::2], 2 * step)
        o = [u * v % p for u, v in zip(o, tw[::step])]
        return [(u + v) % p for u, v in zip(e, o)] + [(u - v) % p for u, v in zip(e, o)]

    return go(x, 1)


def _transform(f, x, direction, w=None):
    """Canonical integers (uint64 array for the 32-bit field), the direction's definition."""
    p, n = f.p, len(x)
    w = _root(f, n.bit_length() - 1) if w is None else w
    inverse = direction in ("inverse", "coset_inverse")
    s = f.generator if not inverse else pow(f.generator, -1, p)
    scale, c = [], 1 if not inverse else pow(n, -1, p)
    for _ in range(n):
        scale.append(c)
        c = c * s % p if direction.startswith("coset") else c
    dft = _dft32 if f.limbs == 1 else _dft
    if f.limbs == 1:
        scale = np.array(scale, dtype=np.uint64)
        mul = lambda a: a * scale % np.uint64(p)  # noqa: E731
    else:
        mul = lambda a: [u * v % p for u, v in zip(a, scale)]  # noqa: E731
    return mul(dft(x, pow(w, -1, p), p)) if inverse else dft(mul(x), w, p)


def exact(case, seed):
    f = g.FIELDS[case["field"]]
    p, op = f.p, case["op"]
    steps = work(case)["flops"] / (2 * f.limbs * f.limbs)
    if steps > (3e7 if f.limbs == 1 else 4.5e6):
        return None
    if f.limbs == 1:
        data = [x.cpu().numpy().reshape(-1).view(np.uint32).astype(np.uint64) for x in _inputs(case, seed)]
        out = lambda a: torch.from_numpy(a.astype(np.uint32).view(np.int32).reshape(-1, 1))  # noqa: E731
        times = lambda a, b: a * b % np.uint64(p)  # noqa: E731
    else:
        data = [_ints(f, x) for x in _inputs(case, seed)]
        out = lambda a: _tensor(f, a)  # noqa: E731
        times = lambda a, b: [u * v % p for u, v in zip(a, b)]  # noqa: E731
    if op == "ntt":
        return out(_transform(f, data[0], case["dir"], _own_root(case)))
    if op == "qap":
        a, b, c = (_transform(f, _transform(f, x, "inverse"), "coset_forward") for x in data)
        z = pow(pow(f.generator, len(a), p) - 1, -1, p)
        h = [(int(u) * int(v) - int(t)) * z % p for u, v, t in zip(a, b, c)]
        h = np.array(h, dtype=np.uint64) if f.limbs == 1 else h
        return [out(_transform(f, h, "coset_inverse")), out(b), out(c)]
    if op == "polymul":
        a, b = (_transform(f, x, "forward") for x in data)
        return [out(_transform(f, times(a, b), "inverse")), out(b)]
    if op == "batch":
        parts = [_transform(f, data[0][at:at + (1 << k)], d) for k, d, at in _batch_jobs(case)[0]]
        return torch.cat([out(x) for x in parts])
    if op == "multiexp":
        total = sum(int(u) * int(v) for u, v in zip(*data)) % p
        if case["mode"] == "montgomery":
            total = total * pow(1 << (32 * f.limbs), -1, p) % p
        return _tensor(f, [total]).reshape(-1)
    return [out(_transform(f, x, case["dir"])) for x in data]
