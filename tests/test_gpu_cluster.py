"""The thread-block cluster kernel of lone tests of n = 2^9 ... 2^13
(m2_cluster.cu, path AUTO) against the one-CTA kernel (path SMALL), the oracle
and its own bounded wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (fields, log2 n, smallest and largest odd exponent of that transform); GF(P61^2) alone keeps
# another kernel where its carry span is 3 (the smallest exponents of a size)
SIZES = [(0, 9, 10497, 20991), (0, 10, 20993, 40959), (0, 11, 40961, 81919), (0, 12, 81929, 159739), (0, 13, 159763, 319483),
         (1, 9, 6657, 12799), (1, 10, 12801, 25599), (1, 11, 25601, 49151), (1, 12, 49153, 98303), (1, 13, 98305, 188415)]


@pytest.mark.parametrize("fields,ln,lo,hi", SIZES)
def test_cluster_matches_one_cta(m2, fields, ln, lo, hi):
    for p in (lo, hi):
        _, n, w = m2.layout(p, fields)
        assert n == 1 << ln
        full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
        start = np.random.default_rng(p).integers(0, 1 << 62, n, dtype=np.uint64) & full
        extreme = full.copy()
        extreme[0] -= np.uint64(1)               # M_p - 1: every digit but one all ones
        for mode in (0, 1, 2):
            with m2.Engine(p, mode, fields=fields) as a, m2.Engine(p, mode, fields=fields, path=m2.PATH_SMALL) as b:
                for state in (start, extreme):
                    a.set_digits(state, 0)
                    b.set_digits(state, 0)
                    for k in (1, 2, 100):
                        a.iterate(k)
                        b.iterate(k)
                        assert np.array_equal(a.digits(), b.digits()), (p, mode, fields, k)


@pytest.mark.parametrize("p", [19937, 23209, 44497, 86243, 216091])
def test_cluster_matches_oracle(m2, oracle_mod, p):
    for mode in (0, 1):
        with m2.Engine(p, mode) as e:
            e.iterate(399)
            e.iterate(1)
            got = e.digits()
        o = oracle_mod.Oracle(p, mode)
        o.iterate(400)
        assert np.array_equal(got, o.digits()), (p, mode)


@pytest.mark.parametrize("p", [19937, 44497, 216091])
def test_cluster_wait_runs_out_and_reports_timeout(m2, oracle_mod, p):
    """Failure detection without a GPU fault: CTA 0 waits for one carry more
    than there are; the launch ends, m2_sync reports M2_ETIMEOUT, and after a
    reload the context computes correct results again."""
    with m2.Engine(p, 1) as e:
        start = e.digits()
        assert e._L.m2_test_stall_fused(e._h) == 0
        e.iterate(3)
        with pytest.raises(m2.M2Error, match=r"\(-4\)"):
            e.sync()
        e.set_digits(start, 0)
        e.iterate(3)
        got = e.digits()
    o = oracle_mod.Oracle(p, 1)
    o.iterate(3)
    assert np.array_equal(got, o.digits())


def test_clusters_share_the_gpu(m2):
    """Many clusters in flight on streams of their own end where each ends alone."""
    ps = (19937, 44497, 86243, 216091) * 4
    alone = {}
    for p in set(ps):
        with m2.Engine(p, 1) as e:
            e.iterate(3000)
            alone[p] = e.res64()
    es = [m2.Engine(p, 1) for p in ps]
    for e in es:
        e.iterate(3000)
    assert [e.res64() for e in es] == [alone[p] for p in ps]
    for e in es:
        e.close()
