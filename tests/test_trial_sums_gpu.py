"""What the one-pass trial promises about the separate calls, on states whose active cells differ from the base's and
with J on the barrier's thresholds."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import q1 as Q

pytestmark = pytest.mark.gpu
W = dict(lam=1e-4, mu=.03, nu=.03, kappa=.002)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def compressed(shape, lo, hi, rng):
    """Noise, and the cells lo <= x < hi compressed to J about 0.03."""
    u = rng.normal(size=shape + (3,)) * .003
    u[..., 0] -= .97 * (np.clip(np.arange(shape[2]), lo, hi) - (lo + hi) / 2)
    return u


@pytest.mark.parametrize("shape", [(5, 6, 7), (5, 6, 24), (40, 44, 48)])
def test_trial_terms_are_the_energys(shape):
    """Energy terms bitwise those of energy() and differences those of energy_difference(), where the base's active
    cells are others than the trial's: the trial's sums must not depend on which cells are evaluated beside them."""
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    rng = np.random.default_rng(8)
    P = DevicePair(grid_from_shape(shape, (1., 1., 1.)), rng.random(shape), rng.random(shape),
                   rng.normal(size=shape + (3,)) * .003, **W)
    for k in range(24):
        trial = dev(compressed(shape, 1, 4, rng))
        wt = P.warp(trial)[0]
        terms, bad = P.energy(trial, wt)
        base = dev(compressed(shape, *((1, 4), (0, 6), (3, 6), (4, 5))[k % 4], rng))
        wb = P.warp(base)[0]
        _, _, tterms, tbad, diff, _ = P.trial_energy(base, wb, trial)
        assert same_bits(tterms, terms) and tbad == bad, k
        assert same_bits(np.array(diff), np.array(P.energy_difference(base, wb, trial, wt)))


def test_screened_counts_and_masks_on_the_thresholds():
    """The screened trial's barrier, violation count and activity mask are the float64 trial's, with the activation and delta on
    values that J takes (up to rounding)."""
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    shape = (7, 9, 12)
    rng = np.random.default_rng(2)
    grid = grid_from_shape(shape, (.9, 1.1, 1.3))
    og = Q.make_grid(shape, (.9, 1.1, 1.3))
    fixed, moving = rng.random(shape), rng.random(shape)
    ref, base = rng.normal(size=shape + (3,)) * .003, rng.normal(size=shape + (3,)) * .08
    trial = base + rng.normal(size=shape + (3,)) * .02
    J = np.sort(Q.geometry(Q.local(trial, og), Q.ops(og, "closed27_uniform"))[2].ravel())
    J = J[(J > 0) & (J < 1)]
    for k in range(24):
        delta, act = float(J[3 * k]), float(J[3 * k + 200])
        P = DevicePair(grid, fixed, moving, ref, **W, activation=act, delta=delta)
        bd, td = dev(base), dev(trial)
        wb = P.warp(bd)[0]
        a, b = P.trial_energy(bd, wb, td), P.trial_energy_screened(bd, wb, td)
        assert a[3] == b[3] and torch.equal(a[5], b[5]), k
        assert a[2][4] == b[2][4]
