"""The staged rotational z pass (k3_rot_staged): waits that give up, parity at the unit shape and the grids
that tests/test_gpu_pass_edges.py does not reach, boxes side by side, and states that are not finite."""
import numpy as np
import pytest

from gpu_util import broadband_field, make_args, rel_l2

pytestmark = pytest.mark.gpu


def _args(N, M=None, les=0.0):
    args = make_args(0, nu=2e-3, Ns=N, les=les)
    if M:
        args.Mx, args.My, args.Mz = M
    return args


def _box(N=(64, 64, 512), precision=0, U0=None, M=None, les=0.0):
    from spns_b200.hit import HIT
    h = HIT(_args(N, M, les), precision=precision, k41_ranks=-1)
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


def _staged(N, M, precision, monkeypatch):
    """Whether the box's z pass is the staged one: with waits that give up, its step says so."""
    from spns_b200.hit import SpnsError
    with monkeypatch.context() as m:
        m.setenv("SPNS_STAGE_POLLS", "0")
        h = _box(N, precision, M=M)
    try:
        h.New_Fractional_Step_Method(1)
        return False
    except SpnsError as e:
        assert "status -7" in str(e)
        return True
    finally:
        h.close()


# modes, FFT lengths, precision, whether the pass is the staged one.  Relative L2 of the state after 3
# steps <= 1e-12 in double, 5e-6 in single precision, as at the other sizes.
PARITY = {
    "z144_kz49": ((96, 96, 96), (144, 144, 144), 0, True),       # 12 threads a pencil, eight of them in three warps
    "z144_kz48": ((96, 96, 94), (144, 144, 144), 0, True),
    "z144_few": ((32, 32, 96), (48, 48, 144), 0, False),         # too few pencils
    "z768_waves": ((96, 96, 511), (144, 144, 768), 0, True),     # more than 16 rounds: several waves of blocks
    "z1536_waves": ((96, 96, 1023), (144, 144, 1536), 1, True),
}


@pytest.mark.parametrize("box", PARITY)
def test_parity(box, monkeypatch):
    import oracle as O
    N, M, precision, staged = PARITY[box]
    assert _staged(N, M, precision, monkeypatch) == staged
    U0 = broadband_field(*N, seed=7)
    gpu = _box(N, precision, U0, M)
    ref = O.OracleHIT(_args(N, M), k41_ranks=1)
    ref.set_compact(U0)
    ref.Recalculate_Velocity_Antitransform()
    ref.Recalculate_TimeStep()
    for h in (gpu, ref):
        for _ in range(3):
            h.New_Fractional_Step_Method()
    assert rel_l2(gpu.get_compact(), ref.get_compact()) <= (5e-6 if precision else 1e-12)


# several boxes of one z length with other mode and pencil counts (other dynamic shared memory of one
# kernel), and boxes of other lengths; 72 x 72 pencils of 96 give blocks of half an SM's threads
SIDE_BY_SIDE = {
    0: [((128, 96, 125), (192, 144, 192)), ((64, 64, 96), (96, 96, 192)), ((64, 64, 256), (96, 96, 384)),
        ((48, 48, 64), (72, 72, 96)), ((48, 48, 63), (72, 72, 96))],
    1: [((128, 128, 125), (192, 192, 192)), ((128, 192, 96), (192, 288, 192)), ((96, 96, 256), (144, 144, 384))],
}


@pytest.mark.parametrize("precision", SIDE_BY_SIDE)
def test_staged_boxes_side_by_side(precision, monkeypatch):
    """Boxes whose z passes each take an SM's tensor memory, stepped concurrently on the streams of one
    ensemble, reach bit for bit the states they reach alone."""
    from spns_b200.hit import Ensemble
    for N, M in SIDE_BY_SIDE[precision]:
        assert _staged(N, M, precision, monkeypatch)
    start = [broadband_field(*N, seed=9) for N, _ in SIDE_BY_SIDE[precision]]
    members, alone = ([_box(N, precision, U0, M) for (N, M), U0 in zip(SIDE_BY_SIDE[precision], start)] for _ in range(2))
    for h in alone:
        h.New_Fractional_Step_Method(4)
    ens = Ensemble(members)
    ens.step(4)
    for h, a in zip(members, alone):
        assert np.array_equal(h.get_compact(), a.get_compact())
    ens.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("les", [0.0, 0.17])
def test_a_state_that_is_not_finite_is_reported(les, precision, bad, monkeypatch):
    """One mode of the state set to NaN or infinity: the running maxima of the staged pass (in tensor
    memory, over many pencils) and of k3_field (LES) report it."""
    from spns_b200.hit import SpnsError
    N = (64, 64, 512)
    if not les:
        assert _staged(N, None, precision, monkeypatch)
    h = _box(N, precision, les=les)
    h.New_Fractional_Step_Method(2)
    U = h.get_compact()
    U[1, 5, 7, 100] = bad
    h.set_compact(U)
    with pytest.raises(SpnsError, match="status -5"):
        h.New_Fractional_Step_Method(1)
