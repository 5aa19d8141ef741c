"""Lone tests beside other work of the same process on the GPU."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


class _Busy(threading.Thread):
    """`work` in a thread of its own."""

    def __init__(self, work):
        super().__init__()
        self.work = work

    def run(self):
        self.result = self.work()

    def __enter__(self):
        self.start()
        time.sleep(0.2)
        return self

    def __exit__(self, *a):
        self.join()


def _batch(m2, iters):
    """100 tests of n = 2^14, one to an SM (about 75 us a squaring)."""
    return m2.batch_run([622577] * 100, iters=[iters] * 100)


def _quick_calls(m2):
    t0 = time.time()
    with m2.Engine(9941, 1) as e:
        e.iterate(100)
        e.res64()
    return time.time() - t0


# a batch of 2.2 s, and results of a test of about 1.5 s (in pageable memory) that are waited for
@pytest.mark.parametrize("case", ["batch", "res64", "verdict", "digits"])
def test_calls_of_other_threads_go_on(m2, case):
    _batch(m2, 2)                             # tables and tuning
    _quick_calls(m2)
    with m2.Engine(6972593, 1) as e:
        if case != "batch":
            e.iterate(100000)
        with _Busy(lambda: _batch(m2, 30000) if case == "batch" else getattr(e, case)()) as busy:
            took = _quick_calls(m2)
            assert busy.is_alive() and took < 0.5


def _res64(m2, p, iters, **kw):
    with m2.Engine(p, 1, **kw) as e:
        e.iterate(iters)
        return e.res64()


# a second context beside one whose call takes about 2 s: one-launch kernels, passes, passes whose CTAs wait for
# each other, one CTA (alone these take 0.01 to 0.1 s)
@pytest.mark.parametrize("pa,ka", [(57885161, 20000), (6972593, 130000)])
@pytest.mark.parametrize("p,path,k", [(1257787, 0, 2000), (1257787, 2, 2000), (57885161, 0, 500), (57885161, 2, 500), (9941, 0, 2000)])
def test_second_context_gets_on(m2, pa, ka, p, path, k):
    want = _res64(m2, pa, ka), _res64(m2, p, k, path=path)
    with m2.Engine(pa, 1) as a, m2.Engine(p, 1, path=path) as b:
        a.iterate(ka)
        t0 = time.time()
        b.iterate(k)
        got = b.res64()
        took = time.time() - t0
        assert took < 0.8 and (a.res64(), got) == want


def test_many_contexts_share_the_gpu(m2):
    """16 contexts of one size with calls in flight together take about as long as
    on the three-pass kernels (2 to 5 times as long one after the other)."""
    for p in (622609, 1245197):
        took = {}
        for path in (m2.PATH_LARGE, m2.PATH_AUTO):
            es = [m2.Engine(p, 1, path=path) for _ in range(16)]
            for _ in range(3):
                t0 = time.time()
                for e in es:
                    e.iterate(600)
                for e in es:
                    e.sync()
                took[path] = time.time() - t0
            assert len({e.res64() for e in es}) == 1
            for e in es:
                e.close()
        assert took[m2.PATH_AUTO] < 1.3 * took[m2.PATH_LARGE]


@pytest.mark.parametrize("p", [1257787, 24036583, 36700201])
def test_lone_test_beside_a_batch(m2, p):
    """A batch holds 100 SMs for 2.2 s: a lone test beside it goes on."""
    want = _res64(m2, p, 150)
    _batch(m2, 2)
    with m2.Engine(p, 1) as e, _Busy(lambda: _batch(m2, 30000)) as busy:
        t0 = time.time()
        e.iterate(150)
        assert e.res64() == want and busy.is_alive() and time.time() - t0 < 1.0


def test_enqueueing_thread_holds_up_nobody(m2):
    """A call of more launches than the stream's queue takes blocks its own thread,
    not the calls of others."""
    with m2.Engine(622577, 1) as a, m2.Engine(6972593, 1) as b:
        b.iterate(10)
        with _Busy(lambda: a.iterate(1100000)):
            t0 = time.time()
            b.iterate(100)
            b.sync()
            assert time.time() - t0 < 1.0
        a.sync()


def test_lone_test_beside_a_busy_server(m2):
    from mersenne2gpu_gb300.serve import Server
    small = [20993, 40961, 5381, 10499, 81929] * 60
    want = _res64(m2, 6972593, 3000), _res64(m2, 57885161, 300)
    with Server(budget_bytes=8 << 30, quantum=500) as srv, m2.Engine(6972593, 1) as e, m2.Engine(57885161, 1) as f:
        for i, p in enumerate(small):
            srv.submit(i, p, 1, 2000)
        srv.submit(1000, 1257787, 1, 3000)
        done = {}

        def serve():
            while len(done) < 301:
                srv.step()
                for r in srv.poll():
                    done[r.id] = r

        with _Busy(serve):
            e.iterate(3000)
            f.iterate(300)
            assert (e.res64(), f.res64()) == want
    ref = {p: _res64(m2, p, 2000) for p in set(small)}
    assert all(done[i].status == 0 and done[i].res64 == ref[p] for i, p in enumerate(small))
    assert done[1000].status == 0 and done[1000].res64 == _res64(m2, 1257787, 3000)


def test_state_after_launches_were_called_off(m2):
    """What reads or replaces the state of a context whose queued launches gave
    way: stages, profiles, a new state, the error check, capture."""
    p, q = 57885161, 1257787
    want = _res64(m2, p, 5011)
    with m2.Engine(p, 1) as a, m2.Engine(q, 1, path=m2.PATH_LARGE) as b:
        start = a.digits()
        for read in ("stages", "profile", "replace"):
            a.set_digits(start, 0)
            a.iterate(5000)
            b.iterate(2000)                   # calls off what of a's is queued
            if read == "stages":
                for stage in (0, 1, 2):
                    a.test_stage(stage)
                a.iterate(10)
            elif read == "profile":
                a.profile(10)
                a.iterate(1)
            else:
                a.set_digits(start, 0)
                a.iterate(5011)
            assert a.info().iteration == 5011 and a.res64() == want
            b.sync()
        want = _res64(m2, p, 1250)
        a.set_digits(start, 0)
        with m2.Gec(a, 600) as g:
            for k in (500, 750):
                b.iterate(3000)
                g.iterate(k)
            b.iterate(3000)
            assert g.check() and g.verified()[1] == 1250 and a.res64() == want


def test_captured_launches_beside_other_runs(m2):
    """Graphs of one-launch contexts replayed on two streams at once, and after
    their contexts ran beside others in passes."""
    import torch
    ps = (6972593, 57885161)
    want = [_res64(m2, p, 2 + 6 * 200 + 300) for p in ps]
    with m2.Engine(1257787, 1, path=m2.PATH_LARGE) as other:
        es, gs, ss = [], [], []
        for p in ps:
            s = torch.cuda.Stream()
            e = m2.Engine(p, 1, stream=s.cuda_stream)
            e.iterate(2)
            e.sync()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                e.iterate(200)
            es.append(e)
            gs.append(g)
            ss.append(s)
        for i in range(6):
            if i % 2:
                other.iterate(1000)
                for e in es:
                    e.iterate(100)
            for g, s in zip(gs, ss):
                with torch.cuda.stream(s):
                    g.replay()
        assert [e.res64() for e in es] == want
        for e in es:
            e.close()
