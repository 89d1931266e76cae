"""GPU step against the oracle at the sizes where the passes' dispatch and tiles change.

Kz is the number of kz modes of a row: tiles of the x/y passes are one 128-byte line of a row
(8 columns double, 16 single, or pairs of columns), rows of 1 KB and more have a pitch of whole
lines, a z pass takes pencils one by one or in pairs.  So: Kz at and around a tile, at and around
1 KB (64 in double, 128 in single precision), odd and even; boxes on both sides of 4 blocks per
SM in the x/y passes (fields spread over blocks or one after another); mode counts below 2/3 of
the FFT length, odd ones among them.

Bar: relative L2 of the state <= 1e-12 after 3 steps in double, as at the other sizes.  Single
precision: a step adds dt R with |dt R| <= C |u| (C = 0.35 C_At, the CFL number) and R of relative
error below 1e-5 (float transforms along three axes and products), so 3 steps stay within 5e-6.
"""
import numpy as np
import pytest

from gpu_util import broadband_field, make_args, rel_l2

pytestmark = pytest.mark.gpu

# modes per axis and FFT lengths
BOXES = {
    "kz9": ((17, 32, 17), (48, 48, 48)),           # one tile and a column
    "kz16": ((32, 31, 31), (48, 48, 48)),
    "kz63": ((32, 32, 125), (48, 48, 192)),        # below 1 KB a row in double
    "kz64": ((32, 21, 127), (48, 48, 192)),
    "kz65": ((32, 32, 128), (48, 48, 192)),
    "kz127": ((32, 32, 253), (48, 48, 384)),       # the same in single precision
    "kz128": ((32, 32, 255), (48, 48, 384)),
    "kz129": ((21, 32, 256), (48, 48, 384)),
    "y96": ((48, 64, 64), (72, 96, 96)),           # fields over blocks
    "y192": ((128, 96, 64), (192, 144, 96)),       # one after another
    "x288": ((192, 32, 33), (288, 48, 72)),
}
# boxes with pencils enough for the persistent z pass in single precision too: one to four warps
# a unit, several pencils of one, a last round that is not full
STAGED = {
    "z192": ((128, 128, 125), (192, 192, 192)),
    "z288": ((96, 96, 191), (144, 144, 288)),
    "z384": ((96, 96, 256), (144, 144, 384)),
    "z768": ((64, 64, 511), (96, 96, 768)),
    "z1536": ((48, 48, 1024), (72, 72, 1536)),
}
FORMS = {
    "rotational": (0, dict(self_adaptive=True), dict(eps_forcing=0.1)),
    "advective": (2, dict(), dict()),
    "les": (0, dict(les=0.17, rotating=(0.0, 0.0, 1.0)), dict()),
}


def _states(box, form_name, precision):
    import oracle as O
    from spns_b200.hit import HIT
    N, M = {**BOXES, **STAGED}[box]
    form, aopt, hopt = FORMS[form_name]
    args = make_args(0, nu=3.283e-4, Ns=N, **aopt)
    args.Mx, args.My, args.Mz = M
    gpu = HIT(args, k41_ranks=-1, nonlinear_form=form, precision=precision, **hopt)
    ref = O.OracleHIT(args, k41_ranks=1, **hopt)
    U0 = broadband_field(*N, seed=5)
    for h in (gpu, ref):
        h.set_compact(U0)
        h.Recalculate_Velocity_Antitransform()
        h.Recalculate_TimeStep()
        for _ in range(3):
            h.New_Fractional_Step_Method()
    out = gpu.get_compact(), ref.get_compact()
    gpu.close()
    return out


@pytest.mark.parametrize("form_name", FORMS)
@pytest.mark.parametrize("box", BOXES)
def test_double_at_the_edges(box, form_name):
    from spns_b200.hit import SPNS_FP64
    a, b = _states(box, form_name, SPNS_FP64)
    assert rel_l2(a, b) <= 1e-12


@pytest.mark.parametrize("form_name", FORMS)
@pytest.mark.parametrize("box", BOXES)
def test_single_at_the_edges(box, form_name):
    from spns_b200.hit import SPNS_FP32_HILO
    a, b = _states(box, form_name, SPNS_FP32_HILO)
    assert rel_l2(a, b) <= 5e-6


def test_ensemble_names_the_member_that_failed():
    from spns_b200.hit import HIT, Ensemble, SpnsError
    members = [HIT(make_args(n, nu=1e-2), k41_ranks=1) for n in (32, 48, 32)]
    ens = Ensemble(members)
    ens.step(2)
    bad = members[1].get_compact()
    bad[0, 1, 1, 1] = np.nan
    members[1].set_compact(bad)
    with pytest.raises(SpnsError, match="member 1"):
        ens.step(2)
    assert np.isfinite(members[0].get_compact()).all() and np.isfinite(members[2].get_compact()).all()
    ens.close()
    for h in members:
        h.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("box", STAGED)
def test_persistent_z_pass(box, precision):
    a, b = _states(box, "rotational", precision)
    assert rel_l2(a, b) <= (5e-6 if precision else 1e-12)


@pytest.mark.parametrize("precision", [0, 1])
def test_rotational_members_side_by_side(precision):
    """The persistent z pass takes an SM's tensor memory whole: boxes stepped concurrently, on
    streams of one ensemble, reach bit for bit the states they reach alone."""
    from spns_b200.hit import HIT, Ensemble
    members, alone = [], []
    for i, N in enumerate([(64, 64, 64), (64, 32, 128), (32, 32, 128), (64, 64, 64)]):
        args = make_args(0, nu=2e-3, Ns=N)
        h = HIT(args, precision=precision, k41_ranks=-1)
        h.seed_field(40 + i, 3.0)
        a = HIT(args, precision=precision, k41_ranks=-1)
        a.checkpoint_load(h.checkpoint_save())
        members.append(h)
        alone.append(a)
    for a in alone:
        a.New_Fractional_Step_Method(4)
    ens = Ensemble(members)
    ens.step(4)
    for h, a in zip(members, alone):
        assert np.array_equal(h.get_compact(), a.get_compact())
    ens.close()
