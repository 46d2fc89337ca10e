"""CPU emulation of the product by a table constant (arith.cuh fe_mul_tw, fe_store_tw) and of the division by a
power of two (fe_div_pow2), word by word with an explicit carry flag, against Python integers on random and
carry-heavy operands: the row schedules lose no carry, the quotient estimate leaves the product below 2p, and both
results are canonical.  The device code runs these schedules in this order."""
import random

import pytest

import oracle as O

M = 0xFFFFFFFF


def _limbs(x, n):
    return [(x >> (32 * k)) & M for k in range(n)]


def _value(words):
    return sum(v << (32 * k) for k, v in enumerate(words))


def _chain(acc, at, prods):
    """One carry chain of wide multiply-adds into acc[at], acc[at + 2], ...; returns the carry out."""
    c = 0
    for k, prod in enumerate(prods):
        s = acc[at + 2 * k] + (prod & M) + c
        acc[at + 2 * k], c = s & M, s >> 32
        s = acc[at + 2 * k + 1] + (prod >> 32) + c
        acc[at + 2 * k + 1], c = s & M, s >> 32
    return c


def _low_row(E, Od, x, i, y, n, jmin=0):
    je, jo = jmin + ((i + jmin) & 1), jmin + ((i + jmin + 1) & 1)
    _chain(E, i + je, [x[j] * y for j in range(je, n - 1 - i, 2)])
    c = _chain(Od, i + jo - 1, [x[j] * y for j in range(jo, n - 2 - i, 2)])
    jt = n - 1 - i
    if jt >= jo:
        Od[n - 2] = (Od[n - 2] + x[jt] * y + c) & M


def _high_row(E, Od, x, i, y, n):
    for acc, j0, base, top in ((E, n - 2 - i if i <= n - 2 else 1, n - 2, n + 1), (Od, n - 1 - i, n - 1, n)):
        js = list(range(j0, n, 2))
        c = _chain(acc, i + j0 - base, [x[j] * y for j in js])
        k = i + js[-1] - base + 2
        if k <= top:
            acc[k] += c
            assert acc[k] <= M, "a carry was lost"
        else:
            assert c == 0, "the product overflowed its words"


def mul_tw(x, w, wp, p, n):
    R = 1 << (32 * n)
    xl = _limbs(x, n)
    E, Od = [0] * (n + 2), [0] * (n + 2)
    for i, y in enumerate(_limbs(wp, n)):
        _high_row(E, Od, xl, i, y, n)
    q = (_value(E) + (_value(Od) << 32)) >> 64
    assert x * wp // R - 1 <= q <= x * wp // R
    E, Od = [0] * n, [0] * n
    for i, y in enumerate(_limbs(w, n)):
        _low_row(E, Od, xl, i, y, n)
    by_adds = p & ((1 << 64) - 1) == 1 + (M << 32)
    by_shift = p & M == (1 << 30) + 1
    neg = _limbs(R - p, n)
    if by_shift:
        neg[1] = -(p >> 32) & M
        assert _value(neg[1:]) == R // (1 << 32) - (p >> 32)
    for i, y in enumerate(_limbs(q, n)):
        _low_row(E, Od, neg, i, y, n, 2 if by_adds else 1 if by_shift else 0)
    t = _value(E) + (_value(Od[:n - 1]) << 32)
    if by_adds:
        t += (q << 32) - q
    if by_shift:
        t -= q + (q << 30)
    t %= R
    assert t < 2 * p
    return t - p if t >= p else t


def _operands(fid, count, seed):
    p, n, rnd = O.MODULI[fid], O.LIMBS[fid], random.Random(seed)
    vals = [0, 1, 2, p - 1, p - 2, p >> 1, (p >> 1) + 1] + [rnd.randrange(p) for _ in range(count)]
    return vals + [sum((M if rnd.random() < 0.85 else 0) << (32 * k) for k in range(n)) % p for _ in range(count)]


@pytest.mark.parametrize("fid", [1, 2])
def test_product_by_a_table_constant(fid):
    p, n = O.MODULI[fid], O.LIMBS[fid]
    for w in _operands(fid, 12, 31 + fid):
        wp = (w << (32 * n)) // p
        for x in _operands(fid, 20, 41 + fid):
            assert mul_tw(x, w, wp, p, n) == x * w % p


def mul_lanes(x, w, wp, p, n):
    """Four lanes per product (ntt_lanes.cuh): lane g takes limbs 4c + g of the constants, its operand shifted up g words."""
    R = 1 << (32 * n)
    wl, ql, neg = _limbs(w, n), _limbs(wp, n), _limbs(R - p, n)
    h = 0
    for g in range(4):
        xs = _limbs(x << (32 * g), n + 3)
        E, Od = [0] * (n + 2), [0] * (n + 2)
        for c in range(n // 4):
            i, y = 4 * c, ql[4 * c + g]
            for acc, j0, base, last, top in ((E, max(0, n - 2 - i), n - 2, n + 2, n + 1),
                                             (Od, n - 1 - i if i < n - 1 else 1, n - 1, n + 1, n)):
                js = list(range(j0, last + 1, 2))
                cy = _chain(acc, i + j0 - base, [xs[j] * y for j in js])
                k = i + js[-1] - base + 2
                if k <= top:
                    acc[k] += cy
                    assert acc[k] <= M, "a carry was lost"
                else:
                    assert cy == 0, "the product overflowed its words"
        h += _value(E) + (_value(Od[:n + 1]) << 32)
        assert Od[n + 1] == 0
    assert h < 1 << (32 * (n + 2))
    q = h >> 64
    assert x * wp // R - 1 <= q <= x * wp // R
    t = 0
    for g in range(4):
        xs, qs = _limbs(x << (32 * g), n), _limbs(q << (32 * g), n)
        E, Od = [0] * n, [0] * n
        for c in range(n // 4):
            _low_row(E, Od, xs, 4 * c, wl[4 * c + g], n)
        for c in range(n // 4):
            _low_row(E, Od, qs, 4 * c, neg[4 * c + g], n)
        t += _value(E) + (_value(Od[:n - 1]) << 32)
    t %= R
    assert t < 2 * p
    return t % p


def test_product_shared_by_four_lanes():
    p, n = O.MODULI[2], O.LIMBS[2]
    for w in _operands(2, 8, 71):
        wp = (w << (32 * n)) // p
        for x in _operands(2, 12, 81) + [2 * p - 1, p, p + 1]:  # values below 2p enter
            assert mul_lanes(x, w, wp, p, n) == x * w % p


def test_products_and_reduction_of_unreduced_values():
    """MNT4-753: values up to 2^13 p enter products and the last pass's reduction by the top word."""
    p, n = O.MODULI[2], O.LIMBS[2]
    rnd = random.Random(101)
    top = (1 << 13) * p
    xs = [0, p, top - 1, top - p, (1 << 12) * p] + [rnd.randrange(top) for _ in range(40)]
    xs += [m * p + d for m in (1, 2, 3, 4095, 8191) for d in (-1, 0, 1)]
    inv = (1 << 48) // ((p >> 736) + 1)
    for x in xs:
        q = (x >> 736) * inv >> 48
        assert 0 <= x - q * p < 2 * p
        for w in (1, p - 1, rnd.randrange(p)):
            assert mul_tw(x, w, (w << (32 * n)) // p, p, n) == x * w % p


@pytest.mark.parametrize("fid", [1, 2])
def test_table_entry_from_the_montgomery_form(fid):
    p, n = O.MODULI[fid], O.LIMBS[fid]
    pinv, pl = (-pow(p, -1, 1 << 32)) & M, _limbs(p, n)
    for w in _operands(fid, 40, 51 + fid):
        m = (w << (32 * n)) % p
        E, Od, q, f = _limbs(m, n) + [0], [0] * (n + 1), 0, []
        for _ in range(n):
            f.append(E[0] * pinv & M)
            for acc, off in ((E, 0), (Od, 1)):
                c = _chain(acc, 0, [pl[j] * f[-1] for j in range(off, n, 2)])
                acc[n] += c
                assert acc[n] <= M
            assert E[0] == 0
            s = Od[0] + E[1]
            e0, c = s & M, s >> 32
            s = Od[1] + q + c
            e1, q = s & M, s >> 32
            E, Od = [e0, e1] + Od[2:], E[2:] + [0, 0]
        assert _value(E) + (_value(Od) << 32) + (q << 64) == w
        assert _value(f) == (w << (32 * n)) // p


@pytest.mark.parametrize("fid", [0, 1, 2])
@pytest.mark.parametrize("k", [1, 2, 13, 28, 31])
def test_division_by_a_power_of_two(fid, k):
    p = O.MODULI[fid]
    pinv = (-pow(p, -1, 1 << 32)) & M
    for x in _operands(fid, 40, 61 + fid):
        f = ((x & M) * pinv) & ((1 << k) - 1)
        assert (x + f * p) % (1 << k) == 0
        assert (x + f * p) >> k == x * pow(1 << k, -1, p) % p
