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
