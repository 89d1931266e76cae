"""The staged rotational z pass (k3_rot_staged): waits that give up, and boxes side by side."""
import numpy as np
import pytest

from gpu_util import broadband_field, make_args

pytestmark = pytest.mark.gpu


def _box(N=(64, 64, 512), precision=0, U0=None):
    from spns_b200.hit import HIT
    h = HIT(make_args(0, nu=2e-3, Ns=N), precision=precision, k41_ranks=-1)
    h.set_compact(broadband_field(*N, seed=7) if U0 is None else U0)
    h.Recalculate_Velocity_Antitransform()
    h.Recalculate_TimeStep()
    return h


@pytest.mark.parametrize("precision", [0, 1])
def test_a_wait_that_gives_up_is_reported(precision, monkeypatch):
    """Every wait for a staged pair gives up at once: the step reports it, the copies are waited for
    before the blocks end, and boxes stepped before, beside and after it are not touched."""
    from spns_b200.hit import SpnsError
    alone = _box(precision=precision)
    alone.New_Fractional_Step_Method(4)
    beside = _box(precision=precision)
    with monkeypatch.context() as m:
        m.setenv("SPNS_STAGE_POLLS", "0")
        h = _box(precision=precision)
    beside.step_async(4)
    with pytest.raises(SpnsError, match="status -7.*bulk copies"):
        h.New_Fractional_Step_Method(1)
    beside.synchronize()
    h.close()
    after = _box(precision=precision)
    after.New_Fractional_Step_Method(4)
    for b in (beside, after):
        assert np.array_equal(b.get_compact(), alone.get_compact())
