"""Device memory that a call needed only for itself is given back."""
import pytest

pytestmark = pytest.mark.gpu


def test_batch_gives_its_memory_back(m2):
    """20000 tests of n = 2^14 hold 3 GiB: afterwards other allocators have it again."""
    import torch
    m2.batch_run([622577] * 4, iters=[1] * 4)
    before = torch.cuda.mem_get_info()[0]
    r = m2.batch_run([622577] * 20000, iters=[1] * 20000)
    assert len(set(r.res64.tolist())) == 1
    assert before - torch.cuda.mem_get_info()[0] <= 512 << 20
