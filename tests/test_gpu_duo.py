"""The fields-in-turn kernel of shared launches (m2_duo.cu: batches and the
server, n = 2^8 ... 2^14) against the same tests run alone."""
import pytest

pytestmark = pytest.mark.gpu

# (log2 n, smallest and largest odd exponent of that transform)
SIZES = [(8, 5377, 10495), (9, 10497, 20991), (10, 20993, 40959), (11, 40961, 81919), (12, 81921, 159743), (13, 159745, 319487),
         (14, 319489, 622591)]


@pytest.mark.parametrize("ln,lo,hi", SIZES)
def test_batch_matches_alone(m2, ln, lo, hi):
    # 160 tests and more fill the GPU: this kernel's launches (and the queue's second round)
    ps, modes, iters = [], [], []
    for k in range(240):
        ps.append((lo, hi)[k & 1])
        modes.append(k // 2 % 3)
        iters.append((1, 2, 3, 61)[k // 6 % 4])
    r = m2.batch_run(ps, modes=modes, iters=iters)
    assert m2.batch_tuning(ln)["carry_blocks"] >= 1
    alone = {}
    for p, mode, it, got in zip(ps, modes, iters, r.res64):
        if (p, mode, it) not in alone:
            with m2.Engine(p, mode) as e:
                assert e.n == 1 << ln
                e.iterate(it)
                alone[p, mode, it] = e.res64()
        assert alone[p, mode, it] == int(got), (p, mode, it)


def test_server_matches_alone(m2):
    from mersenne2gpu_gb300.serve import Server
    jobs = [(p, mode, 95) for _, lo, hi in SIZES for p in (lo, hi) for mode in (0, 1, 2)]
    got = {}
    with Server(budget_bytes=1 << 30, quantum=31) as srv:
        for i, (p, mode, iters) in enumerate(jobs):
            srv.submit(i, p, mode, iters)
        for _ in range(10000):
            srv.step()
            for r in srv.poll():
                got[r.id] = r
            if len(got) == len(jobs):
                break
    assert len(got) == len(jobs)
    for i, (p, mode, iters) in enumerate(jobs):
        with m2.Engine(p, mode) as e:
            e.iterate(iters)
            assert got[i].status == 0 and got[i].res64 == e.res64(), (p, mode)
