"""The cell kernels on the closed27 points (energies, stable differences) against the oracle's Gauss27 sums, on grids
whose cell counts leave remainders in every tile: the smallest grid the library takes, odd and uneven axes,
anisotropic voxels, a compressed region where the barrier is active.

Tolerance: the float64 contract's 1e-12 relative.  Both forms sum the same integrals exactly up to rounding; with
residuals no smaller than 1e-3 of |grad u| the rounding of J (1e-16) stays below 1e-12 of a cell's residual."""
import numpy as np
import pytest
import torch

from oracle import q1 as Q

pytestmark = pytest.mark.gpu
TOL = 1e-12
GRIDS = [((5, 5, 5), (1., 1., 1.)), ((6, 9, 7), (.9, 1.1, 1.3)), ((9, 33, 18), (1., .8, 1.)),
         ((12, 7, 66), (1.25, 1., .9))]


def states(shape, spacing, seed=3):
    """(fixed, moving, reference, base, trial): random smooth-free fields, one x layer compressed to J about 0.03."""
    rng = np.random.default_rng(seed)
    h = np.array(spacing)
    noise = lambda a: rng.normal(size=shape + (3,)) * a * h
    base = noise(.004)
    k = shape[2] // 2
    base[2:-2, 2:-2, :k, 0] += .97 * h[0] / 2
    base[2:-2, 2:-2, k:, 0] -= .97 * h[0] / 2
    ref, trial = base + noise(.003), base + noise(.002)
    for v in (base, ref, trial):
        v[[0, -1]] = 0.
        v[:, [0, -1]] = 0.
        v[:, :, [0, -1]] = 0.
    return rng.random(shape), rng.random(shape), ref, base, trial


@pytest.fixture(scope="module", params=GRIDS, ids=[str(g[0]) for g in GRIDS])
def problem(request):
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    shape, spacing = request.param
    fixed, moving, ref, base, trial = states(shape, spacing)
    w = dict(lam=1e-4, mu=.03, nu=.03, kappa=.002)
    P = DevicePair(grid_from_shape(shape, spacing), fixed, moving, ref, **w)
    OP = Q.make_problem(Q.make_grid(shape, spacing), fixed, moving, ref, w["lam"], w["mu"], w["nu"], w["kappa"])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return P, OP, dev(base), dev(trial), base, trial


def test_energies_and_differences(problem):
    P, OP, bd, td, base, trial = problem
    wb, wt = P.warp(bd)[0], P.warp(td)[0]
    ob, ot = Q.warp(OP, base)[0], Q.warp(OP, trial)[0]
    ref = np.array(Q.energy(OP, trial, ot)[:5])
    terms, bad = P.energy(td, wt)
    assert bad == 0 and np.all(np.abs(terms - ref) <= TOL * np.abs(ref)), (terms, ref)
    dE, dF = Q.differences(OP, base, ob, trial, ot)
    scale = np.array(Q.energy(OP, base, ob)[:5]) + ref      # a difference rounds relative to what it subtracts
    got = P.energy_difference(bd, wb, td, wt)
    assert abs(got[0] - dE) <= TOL * scale.sum() and abs(got[1] - dF) <= TOL * (scale[0] + scale[4])


@pytest.mark.parametrize("term", ["total", "jd", "curl", "barrier", "outer"])
def test_gradients(problem, term):
    P, OP, bd, td, base, trial = problem
    w, g = P.warp(bd, with_gradient=True)
    ow, og = Q.warp(OP, base, True)
    ref = Q.gradient(OP, base, ow, og, term)
    got = P.gradient(bd, w, g, term).cpu().numpy()
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


def test_outer_gradients(problem):
    P, OP, bd, td, base, trial = problem
    w, g = P.warp(bd, with_gradient=True)
    ow, og = Q.warp(OP, base, True)
    active = P.trial_energy(td, P.warp(td)[0], bd)[5]
    assert 0 < int(active.sum())
    for mask in (None, active):
        for got, term in zip(P.outer_gradients(bd, w, g, mask), ("outer", "image", "total")):
            ref = Q.gradient(OP, base, ow, og, term)
            assert np.linalg.norm(got.cpu().numpy() - ref) <= TOL * np.linalg.norm(ref)


def test_ggn_diagonal(problem):
    P, OP, bd, td, base, trial = problem
    _, g = P.warp(bd, with_gradient=True)
    _, og = Q.warp(OP, base, True)
    active = P.trial_energy(td, P.warp(td)[0], bd)[5]
    ref = Q.ggn_diagonal(OP, base, og)
    for mask in (None, active):
        got = P.ggn_diagonal(bd, g, mask).cpu().numpy()
        assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("term", ["total", "jd", "curl"])
def test_mixed_gradients(problem, term):
    """The float32 soft gradient on the same grids against the float64 one: within 1e-4 (J and curl of the two fields
    round at 1e-7 to 2e-7 each, the residuals between them are no smaller than 4e-3)."""
    P, OP, bd, td, base, trial = problem
    w, g = P.warp(bd, with_gradient=True)
    ref = P.gradient(bd, w, g, term)
    P.precision = "mixed"
    from seq_vp_3d_b200 import _lib
    _lib.call("svp_pair_set_precision", P._h, 1)
    try:
        got = P.gradient(bd, w, g, term)
    finally:
        _lib.call("svp_pair_set_precision", P._h, 0)
        P.precision = "plain"
    assert float((got - ref).norm()) <= 1e-4 * float(ref.norm())
