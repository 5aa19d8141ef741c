"""The one-launch kernel of lone mid-size tests (m2_flow.cu, path AUTO) against
the three-pass kernels (path LARGE), the oracle and its own bounded wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (log2 n, smallest and largest exponent of that transform)
DUAL = [(12, 81929, 159739), (13, 159763, 319483), (14, 319489, 622577), (15, 622603, 1245169), (16, 1245187, 2424827),
        (17, 2424833, 4849651), (18, 4849681, 9437179), (19, 9437185, 18874367), (20, 18874369, 36700159)]

GF61 = [(12, 49153, 98303), (13, 98305, 188415), (14, 188417, 376831), (15, 376833, 720895), (16, 720897, 1441791),
        (17, 1441793, 2752511), (18, 2752513, 5505023), (19, 5505025, 10485759), (20, 10485761, 20971519)]


def _random_state(m2, p, fields, seed):
    _, n, w = m2.layout(p, fields)
    full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    return np.random.default_rng(seed).integers(0, 1 << 62, n, dtype=np.uint64) & full, full


def _compare(m2, p, mode, fields, ln):
    start, full = _random_state(m2, p, fields, p + mode)
    extreme = full.copy()
    extreme[0] -= np.uint64(1)               # M_p - 1: every digit but one all ones
    with m2.Engine(p, mode, fields=fields) as a, m2.Engine(p, mode, fields=fields, path=m2.PATH_LARGE) as b:
        assert a.info().ln == ln and a.info().path == m2.PATH_LARGE
        # the kernel under test is the one that runs, but for a carry span beyond its segments of 4 digits
        # (the smallest GF(P61^2)-only exponents of n = 2^18 and up, which keep the three-pass kernels)
        assert (a.launches_for(7) == 1) == (a.info().span <= 3)
        for state in (start, extreme):
            a.set_digits(state, 0)
            b.set_digits(state, 0)
            for k in (1, 2, 64):
                a.iterate(k)
                b.iterate(k)
                assert np.array_equal(a.digits(), b.digits()), (p, mode, fields, k)


@pytest.mark.parametrize("ln,lo,hi", DUAL)
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_flow_matches_three_pass(m2, ln, lo, hi, mode):
    for p in (lo, hi):
        _compare(m2, p, mode, m2.FIELDS_DUAL, ln)


@pytest.mark.parametrize("ln,lo,hi", GF61)
def test_flow_matches_three_pass_gf61(m2, ln, lo, hi):
    for p in (lo, hi):
        _compare(m2, p, 1, m2.FIELDS_GF61, ln)


@pytest.mark.parametrize("p,iters", [(86243, 1300), (216091, 300), (1257787, 60)])
def test_flow_matches_oracle(m2, oracle_mod, p, iters):
    """From the start value, over more than one launch (1300 squarings)."""
    with m2.Engine(p, 1) as e:
        e.iterate(iters)
        got = e.digits()
    o = oracle_mod.Oracle(p, 1)
    o.iterate(iters)
    assert np.array_equal(got, o.digits())


def test_flow_follows_three_pass_stages(m2, oracle_mod):
    """A context whose three-pass stages ran (pending segment carries, untagged
    elements) goes on in the one-launch kernel from that state."""
    p = 216091
    with m2.Engine(p, 0) as e:
        e.iterate(5)
        e.profile(3)
        e.iterate(6)
        for stage in (0, 1, 2):
            e.test_stage(stage)
        e.iterate(5)
        got = e.digits()
    o = oracle_mod.Oracle(p, 0)
    o.iterate(20)
    assert np.array_equal(got, o.digits())


@pytest.mark.parametrize("p", [132049, 6972593])
def test_flow_wait_runs_out_and_reports_timeout(m2, oracle_mod, p):
    """Failure detection without a GPU fault: column group 0 waits for a carry
    tag that no word has; the launch ends, m2_sync reports M2_ETIMEOUT, and
    after a reload the context computes correct results again."""
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


def test_flow_contexts_share_the_gpu(m2):
    """Contexts whose launches are in flight together on streams of their own
    (more CTAs than the GPU holds at once) end where each ends alone."""
    ps = (216091, 1257787, 6972593, 13466917, 24036583, 13466917)
    alone = []
    for p in ps:
        with m2.Engine(p, 1) as e:
            e.iterate(1500)
            alone.append(e.res64())
    es = [m2.Engine(p, 1) for p in ps]
    for e in es:
        e.iterate(1500)
    assert [e.res64() for e in es] == alone
    for e in es:
        e.close()
