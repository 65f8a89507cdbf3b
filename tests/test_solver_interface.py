"""Parts of the solver's interface that a host program relies on, without a GPU: the comparison of two states accepts
the required reduction as a host that screens energies passes it, and a state has a band, zero for float64
differences."""
import types

from seq_vp_3d_b200.solver import EPS, Registration, State


def evaluated(eval_id, differences=None):
    return State(theta=None, u=None, warped=None, energy=[1., .5, .25, .125, .0625], certificate=None, eval_id=eval_id,
                 differences=differences)


def test_state_has_a_band():
    assert evaluated(1).band == 0.


def test_stable_reductions_takes_the_required_reduction():
    reg = Registration.__new__(Registration)
    reg._reference_version = 0
    reg.pair = types.SimpleNamespace(energy_difference=lambda *a: (-.75, -.5))
    base, own = evaluated(1), evaluated(2, differences=((1, 0), (-.25, -.125)))
    for args in ((), (None,), (.1,)):
        (dE, rE), (dF, rF) = reg.stable_reductions(base, own, *args)
        assert (dE, dF) == (.25, .125) and rE == 16 * EPS * base.total and rF == 16 * EPS * base.outer
        (dE, _), (dF, _) = reg.stable_reductions(base, evaluated(3), *args)
        assert (dE, dF) == (.75, .5)
    assert reg.stable_reductions(base, own, required=.1)[0][0] == .25
