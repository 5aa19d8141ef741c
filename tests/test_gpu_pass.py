"""The three-pass kernels with the fields in turn (m2_pass.cu): the server's tests
of n = 2^15 ... 2^20, and path LARGE up to n = 2^18, against the same tests on
the kernels of path AUTO."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# smallest and largest odd exponents of n = 2^15 ... 2^20
ENDS = [622593, 1245183, 1245185, 2424831, 2424833, 4849663, 4849665, 9437183, 9437185, 18874367, 18874369, 36700159]


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_server_matches_alone(m2, mode):
    from mersenne2gpu_gb300.serve import Server
    got = {}
    with Server(budget_bytes=4 << 30, quantum=17) as srv:
        for p in ENDS:
            srv.submit(p, p, mode, 40)
        for _ in range(10000):
            srv.step()
            for r in srv.poll():
                got[r.id] = r
            if len(got) == len(ENDS):
                break
    for p in ENDS:
        with m2.Engine(p, mode) as e:
            e.iterate(40)
            assert got[p].status == 0 and got[p].res64 == e.res64(), (p, mode)


def test_server_small_tests_beside_waiting_lanes(m2):
    """One-CTA tests that hold whole SMs, more of them than that allows, and
    larger tests whose column CTAs wait for each other."""
    from mersenne2gpu_gb300.serve import Server
    small = [20993, 40961, 81929, 159745, 319487] * 9
    for large in ([], [57885161, 115640321], [57885161] * 2 + small * 3):
        jobs = small + large
        got = {}
        with Server(budget_bytes=8 << 30, quantum=23) as srv:
            for i, p in enumerate(jobs):
                srv.submit(i, p, 1, 60)
            for _ in range(100000):
                srv.step()
                for r in srv.poll():
                    got[r.id] = r
                if len(got) == len(jobs):
                    break
        want = {}
        for i, p in enumerate(jobs):
            if p not in want:
                with m2.Engine(p, 1) as e:
                    e.iterate(60)
                    want[p] = e.res64()
            assert got[i].status == 0 and got[i].res64 == want[p], p


@pytest.mark.parametrize("fields", [0, 1])
@pytest.mark.parametrize("p", [159745, 319487, 622589, 1245183, 2424831, 4849663, 9437183])
def test_path_large_matches_auto(m2, p, fields):
    _, n, w = m2.layout(p, fields)
    full = (np.uint64(1) << w.astype(np.uint64)) - np.uint64(1)
    extreme = full.copy()
    extreme[0] -= np.uint64(1)               # M_p - 1: every digit but one all ones
    start = np.random.default_rng(p).integers(0, 1 << 62, n, dtype=np.uint64) & full
    with m2.Engine(p, 0, fields=fields, path=m2.PATH_LARGE) as a, m2.Engine(p, 0, fields=fields) as b:
        for state in (start, extreme):
            a.set_digits(state, 0)
            b.set_digits(state, 0)
            for k in (1, 3, 60):
                a.iterate(k)
                b.iterate(k)
                assert np.array_equal(a.digits(), b.digits()), (p, fields, k)
