"""The one-element-per-thread kernel of lone small tests (m2_lane.cu, path AUTO)
against the one-CTA kernel (path SMALL), exact integers and the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (log2 n, smallest and largest odd exponent of that transform), both fields and GF(P61^2) alone
SIZES = {0: [(5, 689, 1375), (6, 1377, 2687), (7, 2689, 5375), (8, 5377, 10495), (9, 10497, 20991), (10, 20993, 40959)],
         1: [(5, 449, 863), (6, 865, 1727), (7, 1729, 3327), (8, 3329, 6655), (9, 6657, 12799), (10, 12801, 25599)]}


def _compare(m2, p, mode, fields, ln):
    _, n, w = m2.layout(p, fields)
    assert n == 1 << ln
    full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    start = np.random.default_rng(p + mode).integers(0, 1 << 62, n, dtype=np.uint64) & full
    extreme = full.copy()
    extreme[0] -= np.uint64(1)               # M_p - 1: every digit but one all ones
    with m2.Engine(p, mode, fields=fields) as a, m2.Engine(p, mode, fields=fields, path=m2.PATH_SMALL) as b:
        assert a.info().path == m2.PATH_SMALL   # a carry span of 3 (p = 12801, GF(P61^2) alone) keeps the one-CTA kernel
        for state in (start, extreme):
            a.set_digits(state, 0)
            b.set_digits(state, 0)
            for k in (1, 2, 200):
                a.iterate(k)
                b.iterate(k)
                assert np.array_equal(a.digits(), b.digits()), (p, mode, fields, k)


@pytest.mark.parametrize("fields,ln,lo,hi", [(f, *s) for f in (0, 1) for s in SIZES[f]])
def test_lane_matches_one_cta(m2, fields, ln, lo, hi):
    for p in (lo, hi):
        for mode in (0, 1, 2):
            _compare(m2, p, mode, fields, ln)


@pytest.mark.parametrize("p", [1279, 2203, 4423, 9941, 19937, 23209])
def test_lane_matches_oracle(m2, oracle_mod, p):
    """Mersenne prime exponents: state after 700 squarings, LL and PRP."""
    for mode in (0, 1):
        with m2.Engine(p, mode) as e:
            e.iterate(699)
            e.iterate(1)
            got = e.digits()
        o = oracle_mod.Oracle(p, mode)
        o.iterate(700)
        assert np.array_equal(got, o.digits()), (p, mode)


@pytest.mark.parametrize("p,prime", [(1279, True), (2203, True), (1283, False)])
def test_lane_full_run_verdict(m2, p, prime):
    for mode in (0, 1):
        with m2.Engine(p, mode) as e:
            assert e.run() is prime
