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


@pytest.mark.parametrize("N, les, precision", [((256, 256, 512), 0.17, 1), ((256, 256, 512), 0.17, 0), ((512, 256, 512), 0.0, 1)])
def test_short_steps_do_not_wait_for_whole_z_passes(N, les, precision):
    """Steps of a 32^3 box of high priority, one after another, beside a box whose z pass takes
    milliseconds.  If blocks of that pass stayed to its end, one short step in each long one would wait
    for nearly the whole pass; at most one in four may wait for half of it."""
    import time

    import numpy as np
    long_run, short = _box(N, les, precision), _box((32, 32, 32), 0.17, 1, -5)
    for h in (long_run, short):
        h.New_Fractional_Step_Method(4)            # captured
    long_run.profile_begin(3)
    long_run.New_Fractional_Step_Method(3)
    names, ms = long_run.profile_read(3)
    z_pass = 1e-3 * float(np.median(ms[:, names.index("k3_z")]))
    steps, waits = 40, []
    long_run.step_async(steps)
    while not long_run.query():
        t = time.perf_counter()
        short.step_async(1)
        short.synchronize()
        waits.append(time.perf_counter() - t)
    long_run.synchronize()
    short.close()
    long_run.close()
    assert len(waits) > steps and np.sum(np.array(waits) > 0.5 * z_pass) <= steps // 4


@pytest.mark.parametrize("My, Mz, wide", [(48, 384, 256), (48, 192, 128), (72, 384, 256)])
def test_threads_with_boxes_of_one_z_length(My, Mz, wide, monkeypatch):
    """Two host threads launch steps of boxes with the same z length and 17 and `wide` / 2 + 1 modes
    along it (staged z pass, and k3_z at 192): the shared memory that the kernels of the
    one need does not depend on what the other launched last."""
    import threading

    import numpy as np

    from spns_b200.hit import HIT
    monkeypatch.setenv("SPNS_NO_GRAPHS", "1")
    boxes = []
    for Nz in (32, wide):
        args = make_args(0, nu=1e-3, Ns=(32, My * 2 // 3, Nz))
        args.Mx, args.My, args.Mz = 48, My, Mz
        h = HIT(args, k41_ranks=-1)
        h.seed_field(3, 3.0)
        boxes.append(h)
    errors = []

    def run(h):
        try:
            for _ in range(60):
                h.step_async(100)
                h.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(str(e))

    threads = [threading.Thread(target=run, args=(h,)) for h in boxes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert all(np.isfinite(h.get_compact()).all() for h in boxes)
