"""The localized barrier and the node JD measure where cells are compressed far below the activation, against the
oracle: J near 1e-3 and 1e-6 along one axis and along three, and 2^-60.  The barrier's slope goes like 1/J and its
curvature like 1/J^2, so J has to keep its relative accuracy.

Spacing 1 and displacements on a dyadic lattice, so that F is exact in both; what is left is the rounding of J's
products, a few 1e-16 of J.  Tolerance: the float64 contract's 1e-12 relative."""
import numpy as np
import pytest
import torch

from oracle import q1 as Q

pytestmark = pytest.mark.gpu
TOL = 1e-12
SHAPE = (7, 8, 9)
W = dict(lam=1e-4, mu=.03, nu=.03, kappa=.002)
# (length left of a compressed edge, compressed axes): J about 1e-3, 1e-6, 1e-3, 1e-6, 2^-60
CASES = [(2. ** -10, 1), (2. ** -20, 1), (51 / 512, 3), (41 / 4096, 3), (2. ** -20, 3)]


def states(t, axes, seed=4):
    """(reference, base, trial): every cell compressed to t along the first `axes` axes, with noise of t / 64."""
    rng = np.random.default_rng(seed)
    lattice = 2. ** -46
    noise = lambda a: np.round(rng.normal(size=SHAPE + (3,)) * a / lattice) * lattice
    ident = Q.make_grid(SHAPE, (1., 1., 1.)).identity()
    field = np.zeros(SHAPE + (3,))
    for k in range(axes):
        field[..., k] = (t - 1) * (ident[..., k] - (SHAPE[2 - k] - 1) / 2)
    base = field + noise(t / 64)
    return noise(.003), base, base + noise(t / 64)


@pytest.fixture(scope="module", params=CASES, ids=[f"{t:.3g}-{a}" for t, a in CASES])
def problem(request):
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    ref, base, trial = states(*request.param)
    rng = np.random.default_rng(1)
    fixed, moving = rng.random(SHAPE), rng.random(SHAPE)
    P = DevicePair(grid_from_shape(SHAPE, (1., 1., 1.)), fixed, moving, ref, **W)
    OP = Q.make_problem(Q.make_grid(SHAPE, (1., 1., 1.)), fixed, moving, ref, W["lam"], W["mu"], W["nu"], W["kappa"])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return P, OP, dev(base), dev(trial), base, trial


def rel(got, ref):
    return np.linalg.norm(np.asarray(got) - ref) / np.linalg.norm(ref)


def test_energy_and_violations(problem):
    P, OP, bd, td, base, trial = problem
    for dev, host in ((bd, base), (td, trial)):
        terms, bad = P.energy(dev, P.warp(dev)[0])
        ref = Q.energy(OP, host)
        assert bad == 0 and np.all(np.abs(terms - ref) <= TOL * np.abs(ref)), (bad, terms, ref)


def test_differences(problem):
    P, OP, bd, td, base, trial = problem
    wb, wt = P.warp(bd)[0], P.warp(td)[0]
    ob, ot = Q.warp(OP, base)[0], Q.warp(OP, trial)[0]
    dE, dF = Q.differences(OP, base, ob, trial, ot)
    scale = Q.energy(OP, base, ob) + Q.energy(OP, trial, ot)
    _, _, _, bad, one_pass, active = P.trial_energy(bd, wb, td)
    assert bad == 0 and int(active.sum()) == active.numel()
    for got in (P.energy_difference(bd, wb, td, wt), one_pass):
        assert abs(got[0] - dE) <= TOL * scale.sum() and abs(got[1] - dF) <= TOL * (scale[0] + scale[4])


def test_gradients_and_curvature(problem):
    P, OP, bd, td, base, trial = problem
    w, g = P.warp(bd, with_gradient=True)
    ow, og = Q.warp(OP, base, True)
    for term in ("barrier", "outer", "total"):
        assert rel(P.gradient(bd, w, g, term).cpu().numpy(), Q.gradient(OP, base, ow, og, term)) <= TOL, term
    assert rel(P.ggn_diagonal(bd, g).cpu().numpy(), Q.ggn_diagonal(OP, base, og)) <= TOL


def test_node_measure(problem):
    P, OP, bd, td, base, trial = problem
    ref = Q.node_min_jd(OP, base)
    got = P.node_min_jd(bd).cpu().numpy()
    assert np.all(np.abs(got - ref) <= TOL * ref)
    ref, n = Q.node_min_jd(OP, base, .25)
    stats = {}
    got = P.node_min_jd(bd, .25, stats).cpu().numpy()
    assert np.all(got > 0) and np.all(got <= P.node_min_jd(bd).cpu().numpy())


@pytest.mark.parametrize("activation,delta", [(.05, 0.), (.5, .001), (.2, .03)])
def test_barrier_value_has_no_bias(activation, delta):
    """One J in every cell, exactly known: the barrier sum is 27 values per cell of one point's value.  Over 96 J the
    relative errors of a value average out: a point's roundings have a deviation of about 1.7 units of 2^-53, so their
    mean stays below three deviations, 3 * 1.7 / sqrt(96) units."""
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    shape = (5, 5, 6)
    grid = grid_from_shape(shape, (1., 1., 1.))
    zero = np.zeros(shape)
    P = DevicePair(grid, zero, zero, np.zeros(shape + (3,)), **W, activation=activation, delta=delta)
    L = np.longdouble
    errors = []
    for J in np.round(np.linspace(delta + .02 * (activation - delta), activation * .9, 96) * 2. ** 16) / 2. ** 16:
        u = np.zeros(shape + (3,))
        u[..., 0] = (J - 1) * (np.arange(6) - 2.5)
        terms, bad = P.energy(torch.from_numpy(u).cuda(), torch.zeros(shape, dtype=torch.float64, device="cuda"))
        a, d = L(activation), L(delta)
        r = (a - L(J)) / (a - d)
        exact = -27 * grid.n_cells * L(np.float64(W["kappa"]) / 27) * r * r * np.log1p(-r)
        assert bad == 0
        errors.append(float((L(terms[4]) - exact) / exact))
    assert abs(np.mean(errors)) <= 3 * 1.7 / np.sqrt(96) * 2. ** -53
