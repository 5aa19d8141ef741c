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


P61 = (1 << 61) - 1
M64 = (1 << 64) - 1


def fold61(t):
    assert 0 <= t <= M64
    return (t & P61) + (t >> 61)


def part61(x):
    assert 0 <= x < 1 << 128
    r = (x & P61) + (x >> 61)
    assert r <= M64                      # the device's 64-bit sum does not wrap
    return r


def u64(v):
    assert 0 <= v <= M64                 # every intermediate is non-negative and fits
    return v


def products(a0, a1, b0, b1):
    k2_61, k4_61 = 2 * P61, 4 * P61
    k1 = part61(u64(a0 + a1) * b0)
    d, s = u64(b1 + (k2_61 - b0)), u64(b0 + b1)
    k2, k3 = part61(a0 * d), part61(a1 * s)
    mul = fold61(u64(k1 + u64(k4_61 - k3))), fold61(u64(k1 + k2))
    k2, k3 = part61(a1 * d), part61(a0 * s)
    conj = fold61(u64(k1 + k2)), fold61(u64(k1 + u64(k4_61 - k3)))
    sqr = fold61(part61(u64(a0 + a1) * u64(a0 + (k2_61 - a1)))), fold61(u64(part61(a0 * a1) << 1))
    return mul, conj, sqr


def test_gf61_products_range_and_value():
    """cmul61, cmulconj61 and csqr61 of m2_field.cuh for coordinates in
    [0, 2^61 + 7]: no 64-bit step wraps, results are the products and stay in
    that range."""
    top = (1 << 61) + 7
    edge = (0, 1, 2, P61 - 1, P61, P61 + 1, top - 1, top, 1 << 60)
    rng = random.Random(61)
    cases = [(a, b, c, d) for a in edge for b in edge for c in edge for d in edge]
    cases += [tuple(rng.randrange(top + 1) for _ in range(4)) for _ in range(20000)]
    for a0, a1, b0, b1 in cases:
        mul, conj, sqr = products(a0, a1, b0, b1)
        for got, want in ((mul, (a0 * b0 - a1 * b1, a0 * b1 + a1 * b0)), (conj, (a0 * b0 + a1 * b1, a1 * b0 - a0 * b1)),
                          (sqr, (a0 * a0 - a1 * a1, 2 * a0 * a1))):
            assert all(0 <= g <= top and g % P61 == w % P61 for g, w in zip(got, want))
