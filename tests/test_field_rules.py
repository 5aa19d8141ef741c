"""The GF(2^31-1) reduction of a sum of two products (red31p in m2_field.cuh),
restated with its 32-bit wrap-arounds and checked at the ends of its range."""
import random

P31 = (1 << 31) - 1


def red31p(x):
    b = x >> 31
    assert b < 1 << 32
    s = (x & P31) + (b & P31) + (b >> 31)
    assert s < 1 << 32
    return min(s, (s - P31) % (1 << 32))


def test_red31p_range_and_value():
    top = 2 * P31 * P31
    rng = random.Random(31)
    xs = [0, 1, P31 - 1, P31, P31 + 1, 2 * P31, (1 << 32) - 1, 1 << 32, (1 << 62) - 1, 1 << 62, top - 1, top]
    xs += [a * b + c * d for a in (0, 1, P31 - 1, P31) for b in (P31 - 1, P31) for c in (0, P31) for d in (1, P31)]
    xs += [k * P31 + r for k in (1, 2, P31 - 1, P31, P31 + 1, 2 * P31 - 1) for r in (-1, 0, 1)]
    xs += [rng.randrange(top + 1) for _ in range(20000)]
    for x in xs:
        r = red31p(x)
        assert 0 <= r <= P31 and r % P31 == x % P31, x
