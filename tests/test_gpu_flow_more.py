"""The one-launch kernel of mid-size tests (m2_flow.cu) where the exponents of
test_gpu_flow.py run in a cluster: every test here asserts the kernel it is about."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel(e):
    """Name of the kernel of the context's squarings (one squaring is run)."""
    return e.profile(1)[0]["name"]


@pytest.mark.parametrize("p", [622577, 1257787, 6972593, 18874379])
def test_pending_carries_of_three_pass_stages(m2, p):
    """k_flow starts from pending segment carries and untagged elements, clears the
    carries, and goes on from its own state afterwards."""
    with m2.Engine(p, 0) as a, m2.Engine(p, 0, path=m2.PATH_LARGE) as b:
        assert _kernel(a) == "k_flow"
        a.iterate(4)
        for _ in range(2):
            for stage in (0, 1, 2):
                a.test_stage(stage)
        a.iterate(5)
        a.iterate(3)
        b.iterate(1 + 4 + 2 + 5 + 3)
        assert a.info().iteration == 15 and np.array_equal(a.digits(), b.digits())


@pytest.mark.parametrize("p", [622577, 2976221, 13466917, 18874379])
def test_wait_runs_out(m2, p):
    """Column group 0 waits for a carry tag that no word has: the launch ends,
    m2_sync reports M2_ETIMEOUT, and a reload computes correctly again."""
    with m2.Engine(p, 1) as e, m2.Engine(p, 1, path=m2.PATH_LARGE) as b:
        start = e.digits()
        assert _kernel(e) == "k_flow"
        assert e._L.m2_test_stall_fused(e._h) == 0
        e.iterate(3)
        with pytest.raises(m2.M2Error, match=r"\(-4\)"):
            e.sync()
        e.set_digits(start, 0)
        e.iterate(3)
        b.iterate(3)
        assert np.array_equal(e.digits(), b.digits())


@pytest.mark.parametrize("p", [622577, 1257787, 13466917])
def test_state_handed_from_launch_to_launch(m2, p):
    """More than one launch (1000 squarings each) in a call, and odd and even
    numbers of squarings in a row, against the three-pass kernels."""
    with m2.Engine(p, 2) as a, m2.Engine(p, 2, path=m2.PATH_LARGE) as b:
        assert _kernel(a) == "k_flow" and a.launches_for(2301) == 3
        b.iterate(1)
        for k in (2301, 1, 2, 1000, 999):
            a.iterate(k)
            b.iterate(k)
        assert np.array_equal(a.digits(), b.digits())


def test_against_oracle(m2, oracle_mod):
    p = 622577
    with m2.Engine(p, 1) as e:
        assert _kernel(e) == "k_flow"
        e.iterate(1150)
        got = e.digits()
    o = oracle_mod.Oracle(p, 1)
    o.iterate(1151)
    assert np.array_equal(got, o.digits())


# the shapes of n = 2^12 and 2^13, which serve carry spans of 3 (GF(P61^2) alone)
@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("p", [49157, 49999, 98317, 99991])
def test_smallest_shapes(m2, p, mode):
    _, n, w = m2.layout(p, m2.FIELDS_GF61)
    full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    state = np.random.default_rng(p + mode).integers(0, 1 << 62, n, dtype=np.uint64) & full
    with m2.Engine(p, mode, fields=m2.FIELDS_GF61) as a, m2.Engine(p, mode, fields=m2.FIELDS_GF61, path=m2.PATH_LARGE) as b:
        assert a.info().span == 3 and _kernel(a) == "k_flow"
        for start in (state, full - np.uint64(1)):
            a.set_digits(start, 0)
            b.set_digits(start, 0)
            for k in (1, 2, 1003):
                a.iterate(k)
                b.iterate(k)
                assert np.array_equal(a.digits(), b.digits()), (p, mode, k)
