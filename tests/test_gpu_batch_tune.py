"""The autotuner starts from what the batch launches, so a tuned batch is never slower
than the untuned one by its own log."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [None, (128, 256, 128, 0, 0), (32, 1024, 64, 1, 0)])
def test_the_launched_shape_is_the_first_candidate(lib_built, first):
    from fierro_gb300 import problems, sgh
    ps = [problems.sedov(n, jitter=0.1, seed=n, permute=True, cycles=20) for n in (6, 9)]
    with sgh.Batch(ps) as b:
        assert b.shape() == (128, 256, 128, 0, 0)  # the documented default
        if first:
            b.set_shape(*first)
        for i, p in enumerate(ps):
            b.set_state(i, sgh.setup(p))
        chosen, log = b.autotune(cycles=2)
        # a small batch without a shape of its own launches one-warp blocks
        assert tuple(log[0][0]) == (first or (32, 64, 32, 0, 0))
        assert chosen == min(log, key=lambda r: r[1])[0] and b.shape() == chosen
