"""What the batch autotuner remembers: a choice per transform size for a full GPU,
and one for fewer tests than that."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_small_first_batch_does_not_decide_for_large_ones(m2):
    for ln, p in ((9, 19937), (11, 77291)):
        few = m2.batch_run([p] * 8, iters=[20] * 8)
        if m2.batch_tuning(ln)["ns_per_test_squaring"] < 100:
            continue                          # a full GPU of this size was timed before in this process
        many = m2.batch_run([p] * 300, iters=[20] * 300)
        # 300 tests of n = 512 take 13 ns a test-squaring, 8 of them 800
        assert m2.batch_tuning(ln)["ns_per_test_squaring"] < 100
        assert set(many.res64.tolist()) == set(few.res64.tolist())
        again = m2.batch_run([p] * 8, iters=[20] * 8)
        assert (again.res64 == few.res64).all()


@pytest.mark.parametrize("ln,p", [(8, 7001), (9, 19937), (10, 39983), (11, 77291), (12, 132049), (13, 300007), (14, 600011)])
def test_a_full_gpu_takes_the_kernel_with_the_fields_in_turn(m2, ln, p):
    """The kernel that the comparisons with lone tests are about (10 to 30% faster
    than the other's best at every size)."""
    r = m2.batch_run([p] * 240, iters=[7] * 240)
    assert m2.batch_tuning(ln)["kernel"] == "k_duo"
    with m2.Engine(p, 1) as e:
        assert e.n == 1 << ln
        e.iterate(7)
        assert set(r.res64.tolist()) == {e.res64()}
