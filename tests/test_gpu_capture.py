"""Launches whose CTAs wait for each other, on streams that their caller captures
(every kernel that a lone test may take) and after contexts that are gone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the one-element-per-thread CTA, the cluster, and the cooperative kernels of mid-size and large transforms
@pytest.mark.parametrize("p", [9941, 21701, 216091, 1257787, 24036583, 57885161])
def test_captured_squarings_replay(m2, p):
    import torch
    s = torch.cuda.Stream()
    with m2.Engine(p, 0, stream=s.cuda_stream) as e, m2.Engine(p, 0) as ref:
        e.iterate(3)
        e.sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            e.iterate(5)                 # recorded, not run
        for _ in range(3):
            with torch.cuda.stream(s):
                g.replay()
        s.synchronize()
        e.iterate(2)
        ref.iterate(3 + 3 * 5 + 2)
        assert np.array_equal(e.digits(), ref.digits())


def test_contexts_destroyed_with_work_in_flight(m2):
    """Launches whose CTAs wait for each other take turns also after a context
    that is gone: its work in flight comes first."""
    want = []
    for p in (1257787, 57885161):
        with m2.Engine(p, 1) as e:
            e.iterate(40)
            want.append(e.res64())
    for path in (m2.PATH_LARGE, m2.PATH_AUTO):
        for p in (285212449, 115640321):          # groups by arrival ticket
            with m2.Engine(p, 1, path=path) as e:
                e.iterate(30)                     # not synchronised
            got = []
            for q in (1257787, 57885161):
                with m2.Engine(q, 1) as e:
                    e.iterate(40)
                    got.append(e.res64())
            assert got == want


@pytest.mark.parametrize("p", [9941, 216091, 1257787, 57885161])
def test_nothing_is_created_under_capture(m2, p):
    """A context on a stream that is being captured is refused, as is a read that
    has no buffer yet: their memory would be the graph's.  The capture goes on."""
    import torch
    s = torch.cuda.Stream()
    with m2.Engine(p, 1, stream=s.cuda_stream) as e, m2.Engine(p, 1) as ref:
        e.iterate(3)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            with pytest.raises(m2.M2Error, match=r"\(-3\)"):
                m2.Engine(p, 1, stream=s.cuda_stream)
            with pytest.raises(m2.M2Error, match=r"\(-3\)"):
                e.digits()
            e.iterate(4)
        with torch.cuda.stream(s):
            g.replay()
        s.synchronize()
        ref.iterate(7)
        assert np.array_equal(e.digits(), ref.digits())


@pytest.mark.parametrize("p", [216091, 1257787, 57885161])
def test_capture_after_three_pass_stages(m2, p):
    """Squarings recorded while the state is as three-pass stages left it: for the
    replays, and for calls that come before any."""
    import torch
    s = torch.cuda.Stream()
    with m2.Engine(p, 1, stream=s.cuda_stream) as e, m2.Engine(p, 1) as ref:
        for stage in (0, 1, 2):
            e.test_stage(stage)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            e.iterate(2)
        e.iterate(3)
        for _ in range(2):
            with torch.cuda.stream(s):
                g.replay()
        s.synchronize()
        e.iterate(1)
        ref.iterate(1 + 3 + 2 * 2 + 1)
        assert np.array_equal(e.digits(), ref.digits())
