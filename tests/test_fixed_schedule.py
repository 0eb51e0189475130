"""Scaling of the fixed-point sweeps, restated on the CPU: for every
combination of butterfly levels per stage, no component or partial product
can leave 63 bits, and the coarsest step stays below 2^-51 of a tile's norm.
Also the exchange layouts: every stage covers the tile once, without bank
conflicts."""
import itertools

import pytest

E, LIM = 3, 5


def schedule(m, cost, backward):
    """(norm bounds in half bits above 2^60 at every step, B), as fix_schedule."""
    levels, seen = sum(m), []
    if cost and not backward:
        B, h = 62, 0
    else:
        up = (LIM - levels) // 2 if levels <= LIM else -((levels - LIM + 1) // 2)
        B = 60 + max(-2, min(2, up))
        h = 2 * (B - 60)
    seen.append(h)

    def room(mm):
        nonlocal h
        over = h + mm - LIM
        h += mm - 2 * ((over + 1) // 2 if over > 0 else 0)
        seen.append(h)

    h += m[0]
    seen.append(h)
    for x in m[1:]:
        room(x)
    h -= 8
    seen.append(h)
    for x in m[::-1]:
        room(x)
    return seen, B


@pytest.mark.parametrize("cost,backward", [(False, False), (True, False), (False, True), (True, True)])
def test_norms_stay_in_range(cost, backward):
    for stages in range(1, 5):
        for m in itertools.product(range(E + 1), repeat=stages):
            seen, B = schedule(m, cost, backward)
            assert max(seen) <= LIM  # norm <= 2^62.5: |component| < 2^63
            assert min(seen) >= -8 and 58 <= B <= 62  # >= 2^56: steps of at most 2^-56 of the norm
            # a product's middle sum: |x_h| |d_l| + |x_l| |d_h| over both components
            norm = 2.0 ** (60 + max(seen) / 2)
            assert 2 ** 0.5 * norm * 2.0 ** -32 * 2.0 ** 31 + 2 ** 0.5 * 2.0 ** 31 * 2.0 ** 30 < 2.0 ** 63


def eoff(T, s, c):
    lo = T - E * (s + 1)
    if lo >= 0:
        return c << lo
    r = E + lo
    return (c & ((1 << r) - 1)) | ((c >> r) << (T + lo))


def ebase(T, s, t):
    lo = T - E * (s + 1)
    if lo >= 0:
        return (t & ((1 << lo) - 1)) | ((t >> lo) << (lo + E))
    return t << (E + lo)


def sw(e):
    return e ^ ((e >> 3) & 7)


@pytest.mark.parametrize("T", [9, 10, 11, 12])
def test_exchange_layouts(T):
    threads = 1 << (T - E)
    for s in range((T + E - 1) // E):
        seen = set()
        for c in range(1 << E):
            o = sw(eoff(T, s, c))
            slots = [(sw(ebase(T, s, t)) ^ (o & 7)) + (o & ~7) for t in range(threads)]
            assert slots == [sw(ebase(T, s, t) | eoff(T, s, c)) for t in range(threads)]
            seen.update(slots)
            for q in range(0, threads, 8):  # a quarter warp's 16-byte accesses
                assert len({x & 7 for x in slots[q:q + 8]}) == 8
        assert seen == set(range(1 << T))
