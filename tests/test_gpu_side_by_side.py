"""Boxes of different size on one GPU at the same time: a short run beside a long one."""
import pytest

from gpu_util import make_args

pytestmark = pytest.mark.gpu


def _box(N, les=0.0, precision=1, priority=0):
    from spns_b200.hit import HIT
    h = HIT(make_args(0, nu=1e-3, Ns=N, les=les), precision=precision, k41_ranks=-1, stream_priority=priority)
    h.seed_field(3, 3.0)
    h.New_Fractional_Step_Method(3)
    return h


@pytest.mark.parametrize("les", [0.0, 0.17])
def test_closing_a_box_leaves_the_others_running(les):
    """A box is released in the order of its own stream: one with captured steps of either form is
    closed while 600 ms of another's steps are in flight, and those are not waited for."""
    for _ in range(3):
        long_run, short = _box((256, 256, 256)), _box((64, 64, 64), les)
        for h in (long_run, short):
            h.New_Fractional_Step_Method(4)        # captured
        long_run.step_async(300)
        short.step_async(5)
        short.synchronize()
        short.close()
        running = not long_run.query()
        long_run.synchronize()
        long_run.close()
        if running:
            return
    pytest.fail("closing a 64^3 box waited for 300 steps of a 256^3 box, three times of three")
