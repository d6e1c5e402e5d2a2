"""What the search reads of a key without computing it: eight columns of byte
sums, as fill_group_table weighs the bytes and test_group adds the columns up.
Checked on the CPU in Python integers, with the six values' bytes at their ends
and unreduced."""
import random

import pytest

P = 2**255 - 19
ENDS = [0, 1, 19, P - 1, P, P + 1, 2 * P, 2**255, 2**256 - 38, 2**256 - 1, 2**224 - 1, 2**256 - 2**224]
ALL = (1 << 24) - 1


def columns(values, coefficients):
    """The sums of one key: column n < 3 of byte n of the low 24 bits of
    rho = c 2^(8 j) mod p, column 3 + n of byte n of the top 41 bits of rho."""
    col = [0] * 8
    for v, c in zip(values, coefficients):
        for j in range(32):
            byte, rho = v >> 8 * j & 255, (c << 8 * j) % P
            for n in range(3):
                col[n] += byte * (rho >> 8 * n & 255)
            for n in range(5):
                col[3 + n] += byte * (rho >> 215 + 8 * n & 255)
    return col


def read(k):
    """test_group's reading: the low limb (24 bits of it), K's bits 16..39, and
    whether those leave the quotient open."""
    assert all(0 <= c < 2**32 for c in k)
    t0 = k[4] + (k[3] >> 8)
    t1 = k[5] + (t0 >> 8)
    t2 = k[6] + (t1 >> 8)
    t3 = k[7] + (t2 >> 8)
    assert t3 < 2**32
    low = (k[0] + (k[1] << 8) + (k[2] << 16) + 19 * (t3 >> 8)) & ALL
    return low, (t3 & 255) << 16 | (t2 & 255) << 8 | (t1 & 255), t1 & t2 & t3 & 255 == 255


def check(values, coefficients):
    key = sum(v * c for v, c in zip(values, coefficients)) % P
    low, top, open_ = read(columns(values, coefficients))
    if open_:  # only next to a multiple of p: the sum is short by less than one of bit 16
        assert key >> 231 in (0, ALL)
        return False
    assert low == key & ALL
    # bits 231..254, or one less
    assert key >> 231 in (top, (top + 1) & ALL)
    return True


def test_ends():
    rng = random.Random(1)
    for a in ENDS:
        for c in ENDS[:5] + [rng.randrange(P) for _ in range(3)]:
            check([a] * 6, [c % P] * 6)
            check([a, 0, ENDS[3], 0, a, 1], [c % P, 1, P - 1, 0, -c % P, 5])


def test_random_values():
    rng = random.Random(2)
    n = 1500
    sure = sum(check([rng.getrandbits(256) for _ in range(6)], [rng.randrange(P) for _ in range(6)]) for _ in range(n))
    assert sure >= n - 2  # open in one of 2^24


def test_the_sum_is_short_by_less_than_its_lowest_sixteen_bits():
    """K = 2^40 T / p less an error of 192 x 255 at most, the largest with every
    byte 255: so bits 16..39 all ones are the only open case."""
    rng = random.Random(3)
    for values in [[2**256 - 1] * 6] + [[rng.getrandbits(256) for _ in range(6)] for _ in range(300)]:
        coefficients = [rng.randrange(P) for _ in range(6)]
        k = columns(values, coefficients)
        total = sum((v >> 8 * j & 255) * ((c << 8 * j) % P) for v, c in zip(values, coefficients) for j in range(32))
        got = sum(c << 8 * n for n, c in enumerate(k[3:]))
        assert 0 <= (total << 40) / P - got < 192 * 255 + 1
        assert 0 <= (total << 40) // P - got < 2**16


@pytest.mark.parametrize("above", [0, 1, 2**215 - 1])
def test_a_sum_just_below_a_multiple_is_open(above):
    """T = k p - 1 - above: its quotient is k - 1, which the sums cannot tell
    from k; they say so."""
    v, c = 1, P - 1 - above
    low, top, open_ = read(columns([v, 0, 0, 0, 0, 0], [c, 0, 0, 0, 0, 0]))
    assert open_ and top == ALL
