"""CPU emulation of the multi-exponentiation's last step (multiexp.cuh): column sums reduced by Montgomery word steps, a lane
per column, and the product by the representation constant in the same form, against Python integers; the totals reach the
largest that the entry points admit.  Every lane's column stays below 2^64."""
import random

import pytest

import oracle as O

M = 0xFFFFFFFF


def _lane_step(acc, p_lane, pinv, hi, enter):
    m = (acc[0] & M) * pinv & M
    prod = [m * v for v in p_lane]
    acc = [a + (q & M) for a, q in zip(acc, prod)]
    assert acc[0] & M == 0 and max(acc) < 1 << 64
    up = acc[1:] + [enter]
    out = [u + (q >> 32) + h for u, q, h in zip(up, prod, hi)]
    out[0] += acc[0] >> 32
    assert max(out) < 1 << 64
    return out


def _value(cols):
    return sum(c << (32 * k) for k, c in enumerate(cols))


def finish(cols, p, n, fix):
    pinv = (-pow(p, -1, 1 << 32)) & M
    p_lane = [(p >> (32 * j)) & M if j < n else 0 for j in range(32)]
    f_lane = [(fix >> (32 * j)) & M if j < n else 0 for j in range(32)]
    rows = n + 2
    cols = list(cols) + [0] * (rows + 32 - len(cols))
    acc = cols[:32]
    for r in range(rows):
        acc = _lane_step(acc, p_lane, pinv, [0] * 32, cols[r + 32])
    assert _value(acc) < 2 * p and not any(acc[n + 1:])
    x = _value(acc) % p
    acc = [0] * 32
    for i in range(n):
        prod = [((x >> (32 * i)) & M) * v for v in f_lane]
        acc = [a + (q & M) for a, q in zip(acc, prod)]
        acc = _lane_step(acc, p_lane, pinv, [q >> 32 for q in prod], 0)
    assert _value(acc) < 2 * p
    return _value(acc) % p


@pytest.mark.parametrize("fid", [0, 1, 2])
def test_columns_reduce_to_the_sum(fid):
    p, n, rnd = O.MODULI[fid], O.LIMBS[fid], random.Random(91 + fid)
    w = 2 * n + 1
    canonical, mont = pow(2, 32 * (2 * n + 2), p), pow(2, 32 * (n + 2), p)
    rinv = pow(1 << (32 * n), -1, p)
    totals = [0, 1, p, p * p, (p - 1) ** 2, (1 << 40) * (p - 1) ** 2] + [rnd.randrange(p * p << 39) for _ in range(20)]
    for total in totals:
        # the same total in wide columns: what sums over threads and blocks leave
        cols, left = [0] * w, total
        for k in range(w):
            cols[k] = left & M if k < w - 1 else left
            left = left >> 32 if k < w - 1 else 0
        for k in range(w - 1):  # move weight down: columns of up to 51 bits
            move = min(cols[k + 1], rnd.randrange(1 << 18))
            cols[k + 1] -= move
            cols[k] += move << 32
        if max(cols) >= 1 << 60:
            continue
        assert _value(cols) == total
        assert finish(cols, p, n, canonical) == total % p
        assert finish(cols, p, n, mont) == total * rinv % p
