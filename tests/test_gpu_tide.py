"""The one-launch kernel of large lone tests (m2_tide.cu, path AUTO, n = 2^21
and 2^22) against the three-pass kernels (path LARGE) and its own bounded wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _states(m2, p, fields):
    _, n, w = m2.layout(p, fields)
    full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    extreme = full.copy()
    extreme[0] -= np.uint64(1)               # M_p - 1: every digit but one all ones
    return np.random.default_rng(p).integers(0, 1 << 62, n, dtype=np.uint64) & full, extreme


# smallest and largest exponents of both sizes and field sets; a carry span above 3 keeps the three-pass kernels
@pytest.mark.parametrize("p,mode,fields,ln", [
    (36700161, 1, 0, 21), (73400319, 0, 0, 21), (73400321, 2, 0, 22), (142606335, 1, 0, 22),
    (20971521, 0, 1, 21), (39845887, 1, 1, 21), (39845889, 1, 1, 22), (79691775, 2, 1, 22)])
def test_tide_matches_three_pass(m2, p, mode, fields, ln):
    start, extreme = _states(m2, p, fields)
    with m2.Engine(p, mode, fields=fields) as a, m2.Engine(p, mode, fields=fields, path=m2.PATH_LARGE) as b:
        assert a.info().ln == ln
        assert (a.launches_for(250) == 1) == (a.info().span <= 3)
        for state, ks in ((start, (1, 2, 253)), (extreme, (3,))):
            a.set_digits(state, 0)
            b.set_digits(state, 0)
            for k in ks:
                a.iterate(k)
                b.iterate(k)
                assert np.array_equal(a.digits(), b.digits()), (p, mode, fields, k)


@pytest.mark.parametrize("p", [57885161, 115640321])
def test_tide_follows_three_pass_stages(m2, p):
    """A context whose three-pass stages ran (pending segment carries, untagged
    elements) goes on in the one-launch kernel from that state."""
    with m2.Engine(p, 0) as a, m2.Engine(p, 0, path=m2.PATH_LARGE) as b:
        a.iterate(2)
        for stage in (0, 1, 2):
            a.test_stage(stage)
        a.iterate(2)
        b.iterate(5)
        assert a.info().iteration == 5 and np.array_equal(a.digits(), b.digits())


@pytest.mark.parametrize("p", [57885161, 115640321])
def test_tide_wait_runs_out_and_reports_timeout(m2, p):
    """Failure detection without a GPU fault: the first CTA waits for a carry
    tag that no word has; the launch ends, m2_sync reports M2_ETIMEOUT, and
    after a reload the context computes correct results again."""
    with m2.Engine(p, 1) as e, m2.Engine(p, 1, path=m2.PATH_LARGE) as b:
        start = e.digits()
        assert e._L.m2_test_stall_fused(e._h) == 0
        e.iterate(3)
        with pytest.raises(m2.M2Error, match=r"\(-4\)"):
            e.sync()
        e.set_digits(start, 0)
        e.iterate(3)
        b.iterate(3)
        assert np.array_equal(e.digits(), b.digits())


def test_tide_contexts_share_the_gpu(m2):
    """Contexts of several sizes in flight together end where each ends alone."""
    ps = (57885161, 13466917, 57885161, 216091)
    alone = {}
    for p in set(ps):
        with m2.Engine(p, 1) as e:
            e.iterate(600)
            alone[p] = e.res64()
    es = [m2.Engine(p, 1) for p in ps]
    for e in es:
        e.iterate(600)
    assert [e.res64() for e in es] == [alone[p] for p in ps]
    for e in es:
        e.close()


def test_one_launch_and_three_pass_contexts_take_turns(m2):
    """Contexts whose kernels wait between their CTAs -- one-launch ones and
    three-pass ones with the fused column pass by tickets and cooperative --
    in flight together: none starves another until its wait runs out."""
    jobs = [(115640321, m2.PATH_LARGE, 300), (57885161, m2.PATH_AUTO, 500), (13466917, m2.PATH_LARGE, 1000),
            (1257787, m2.PATH_LARGE, 1000), (6972593, m2.PATH_AUTO, 1000)]
    want = []
    for p, path, k in jobs:
        with m2.Engine(p, 1, path=path) as e:
            e.iterate(k)
            want.append(e.res64())
    es = [m2.Engine(p, 1, path=path) for p, path, _ in jobs]
    for part in range(2):
        for e, (_, _, k) in zip(es, jobs):
            e.iterate(k // 2)
    assert [e.res64() for e in es] == want
    for e in es:
        e.close()
