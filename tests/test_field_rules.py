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


def scale61(x):
    return u64(((u64(x) & ((1 << 31) - 1)) << 30) + (x >> 31))


def radix8(u):
    """dif8_adds of m2_split.cuh in GF(P61^2), every step as there."""
    k2, k4 = 2 * P61, 4 * P61
    add = lambda x, y: tuple(fold61(u64(p + q)) for p, q in zip(x, y))
    lsub = lambda x, y: tuple(u64(p + u64(k2 - q)) for p, q in zip(x, y))
    sub = lambda x, y: tuple(fold61(t) for t in lsub(x, y))
    times_i = lambda x: (u64(k2 - x[1]), x[0])

    def eighth_of_diff(x, y):
        d = lsub(x, y)
        return scale61(d[0] + u64(k4 - d[1])), scale61(d[0] + d[1])

    def dif_adds(x, u1, u2, u3):
        v0, v1 = tuple(u64(p + q) for p, q in zip(x, u2)), tuple(u64(p + q) for p, q in zip(u1, u3))
        v2, v3 = lsub(x, u2), lsub(u1, u3)
        fadd, fsub = lambda p, q: fold61(u64(p + q)), lambda p, q: fold61(u64(p + u64(k4 - q)))
        return [(fadd(v0[0], v1[0]), fadd(v0[1], v1[1])), (fsub(v0[0], v1[0]), fsub(v0[1], v1[1])),
                (fsub(v2[0], v3[1]), fadd(v2[1], v3[0])), (fadd(v2[0], v3[1]), fsub(v2[1], v3[0]))]

    a = [add(u[m], u[m + 4]) for m in range(4)]
    b = [sub(u[0], u[4]), eighth_of_diff(u[1], u[5]), times_i(sub(u[2], u[6])), times_i(eighth_of_diff(u[3], u[7]))]
    return dif_adds(*a) + dif_adds(*b)


def unradix8(y):
    """dit8_adds of m2_split.cuh in GF(P61^2)."""
    k2, k4 = 2 * P61, 4 * P61
    add = lambda x, z: tuple(fold61(u64(p + q)) for p, q in zip(x, z))
    lsub = lambda x, z: tuple(u64(p + u64(k2 - q)) for p, q in zip(x, z))
    sub = lambda x, z: tuple(fold61(t) for t in lsub(x, z))
    times_i = lambda x: (u64(k2 - x[1]), x[0])
    eighth_conj = lambda x: (scale61(x[0] + x[1]), scale61(x[1] + u64(k2 - x[0])))

    def dit_adds(x):
        v0, v1 = tuple(u64(p + q) for p, q in zip(x[0], x[1])), lsub(x[0], x[1])
        v2, v3 = tuple(u64(p + q) for p, q in zip(x[2], x[3])), lsub(x[3], x[2])
        fadd, fsub = lambda p, q: fold61(u64(p + q)), lambda p, q: fold61(u64(p + u64(k4 - q)))
        return [(fadd(v0[0], v2[0]), fadd(v0[1], v2[1])), (fsub(v1[0], v3[1]), fadd(v1[1], v3[0])),
                (fsub(v0[0], v2[0]), fsub(v0[1], v2[1])), (fadd(v1[0], v3[1]), fsub(v1[1], v3[0]))]

    a, b = dit_adds(y[:4]), dit_adds(y[4:])
    b = [b[0], eighth_conj(b[1]), times_i(b[2]), times_i(eighth_conj(b[3]))]
    return [add(a[0], b[0]), add(a[1], b[1]), sub(a[2], b[2]), sub(a[3], b[3]),
            sub(a[0], b[0]), sub(a[1], b[1]), add(a[2], b[2]), add(a[3], b[3])]


def test_radix8_ranges_and_value():
    w = [(1, 0)]
    for _ in range(7):
        p, q = w[-1]
        w.append(((p - q << 30) % P61, (p + q << 30) % P61))
    assert w[2] == (0, 1)
    rng = random.Random(8)
    ends = (0, 1, P61, P61 + 8)
    cases = [[(rng.choice(ends), rng.choice(ends)) for _ in range(8)] for _ in range(4000)]
    cases += [[(rng.randrange(P61 + 9), rng.randrange(P61 + 9)) for _ in range(8)] for _ in range(1000)]
    for u in cases:
        y = radix8(u)
        for k, e in enumerate((0, 4, 2, 6, 1, 5, 3, 7)):
            re = sum(u[m][0] * w[m * e % 8][0] - u[m][1] * w[m * e % 8][1] for m in range(8))
            im = sum(u[m][0] * w[m * e % 8][1] + u[m][1] * w[m * e % 8][0] for m in range(8))
            assert y[k][0] <= P61 + 8 and y[k][1] <= P61 + 8
            assert (y[k][0] - re) % P61 == 0 and (y[k][1] - im) % P61 == 0
        x = unradix8(y)
        for m in range(8):
            for c in range(2):
                assert x[m][c] <= P61 + 8 and (x[m][c] - 8 * u[m][c]) % P61 == 0
        unradix8(u)                          # ranges alone


def test_weight_shift_at_every_transform_size(tmp_path):
    """The device's shifts n^-1 (n - p j mod n) mod 61 and 31 up to n = 2^30, from
    the header that the table kernel includes, against whole numbers."""
    import os
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mersenne2gpu_gb300", "csrc")
    src = tmp_path / "s.cpp"
    src.write_text('#include "m2_host.hpp"\n#include <cstdio>\nint main() { unsigned lr, x, m;\n'
                   'while (std::scanf("%u %u %u", &lr, &x, &m) == 3) std::printf("%u\\n", m2::weight_shift(lr, x, m)); }\n')
    exe = tmp_path / "s"
    subprocess.run(["g++", "-std=c++17", "-I", csrc, "-o", str(exe), str(src)], check=True)
    rng = random.Random(61)
    cases = []
    for ln in range(3, 31):
        n = 1 << ln
        for m in (61, 31):
            lr = (1 << (m - 1 - ln)) % m
            assert lr * n % m == 1
            cases += [(lr, x, m) for x in [1, 2, n // 2, n - 1, n] + [rng.randrange(1, n + 1) for _ in range(40)]]
    out = subprocess.run([str(exe)], input="\n".join("%d %d %d" % c for c in cases), capture_output=True, text=True, check=True).stdout
    assert [int(v) for v in out.split()] == [lr * x % m for lr, x, m in cases]
    # the product as it was, in 32 bits, is wrong from n = 2^27 on
    wrong = min(x for lr, x, m in cases if lr * x % (1 << 32) % m != lr * x % m)
    assert wrong > 1 << 26
