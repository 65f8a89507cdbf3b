"""A displacement with a value that is not finite.  The cells that touch its node have no J, or an infinite one: the
barrier points whose J is not above delta count as violations, a cell without a J below the activation adds nothing to
the barrier's gradient, and J that are NaN do not enter the node measure; every other cell is as without it.  Checked in
the state that has a mask and in the one whose cells the kernels flag, and for cells of negative J."""
import numpy as np
import pytest
import torch

from oracle import q1 as Q

pytestmark = pytest.mark.gpu
TOL = 1e-12
SHAPE = (8, 9, 11)
W = dict(lam=1e-4, mu=.03, nu=.03, kappa=.002)
NODE = (3, 4, 5)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def problem():
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    rng = np.random.default_rng(6)
    fixed, moving = rng.random(SHAPE), rng.random(SHAPE)
    u = rng.normal(size=SHAPE + (3,)) * .003
    u[..., 0] -= .97 * (np.arange(SHAPE[2]) - 5.)          # J about 0.03 in every cell
    P = DevicePair(grid_from_shape(SHAPE, (1., 1., 1.)), fixed, moving, np.zeros(SHAPE + (3,)), **W)
    OP = Q.make_problem(Q.make_grid(SHAPE, (1., 1., 1.)), fixed, moving, np.zeros(SHAPE + (3,)), *W.values())
    w, g = P.warp(dev(u), with_gradient=True)
    return P, OP, u, w, g


def touched(grid):
    return np.any(Q.cell_nodes(grid) == np.ravel_multi_index(NODE, grid.shape), axis=1)


def barrier_gradient(OP, u, cells):
    op = Q.ops(OP.grid, "closed27_uniform")
    out = np.zeros((3,) + OP.grid.shape)
    _, A, J, _ = Q.geometry(Q.local(u, OP.grid, cells), op)
    slope = Q.barrier_terms(J, OP.delta, OP.barrier_weight, OP.activation)[1]
    Q._scatter(OP.grid, op, Q._flux(A, slope, None), out, cells)
    return Q.restrict(out)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("component", [0, 1, 2])
def test_one_value(problem, value, component):
    P, OP, u, w, g = problem
    broken = u.copy()
    broken[NODE + (component,)] = value
    bd = dev(broken)
    hit = touched(OP.grid)
    with np.errstate(invalid="ignore"):
        J = Q.geometry(Q.local(broken, OP.grid), Q.ops(OP.grid, "closed27_uniform"))[2]
    assert np.isnan(J[hit]).any() and P.energy(bd, w)[1] == (~(J > 0)).sum() >= 8 * 20
    if (J[hit] < OP.activation).any():                       # minus infinity: the gradient has no value there
        return
    ref = barrier_gradient(OP, u, np.flatnonzero(~hit))
    image = P.gradient(dev(u), w, g, "image").cpu().numpy()
    other = np.ones(SHAPE, bool)                             # every node but the broken one, whose u is not finite
    other[NODE] = False
    away = np.ones(SHAPE, bool)                              # nodes of whole cells: gF also reads the soft values
    away.ravel()[Q.cell_nodes(OP.grid)[hit]] = False
    other, away = (np.tile(k[1:-1, 1:-1, 1:-1].ravel(), 3) for k in (other, away))
    for active in (None, dev(np.ones(OP.grid.n_cells, np.uint8))):
        got = P.gradient(bd, w, g, "barrier", active=active).cpu().numpy()
        assert np.linalg.norm((got - ref)[other]) <= TOL * np.linalg.norm(ref)
        gF = P.outer_gradients(bd, w, g, active)[0].cpu().numpy()
        assert np.linalg.norm((gF - image - ref)[away]) <= TOL * np.linalg.norm(gF[away])


def test_node_measure(problem):
    P, OP, u, w, g = problem
    broken = u.copy()
    broken[NODE + (1,)] = np.nan
    hit = touched(OP.grid)
    minima = Q.closed27_cell_minima(Q.geometry(Q.local(u, OP.grid), Q.ops(OP.grid, "closed27_uniform"))[2])
    minima[hit] = np.inf
    node = np.full(int(np.prod(SHAPE)), np.inf)
    for nodes in Q.cell_nodes(OP.grid).T:
        np.minimum.at(node, nodes, minima)
    for extension in (None, .25):
        got = P.node_min_jd(dev(broken), extension).cpu().numpy().ravel()
        assert np.array_equal(np.isinf(got), np.isinf(node)) and np.isinf(node).sum() == 1
        if extension is None:
            known = np.isfinite(node)
            assert np.all(np.abs(got[known] - node[known]) <= TOL * node[known])


def test_zero_weights(problem):
    """With neither soft penalty the soft gradient is zero, also where the field is not finite."""
    from seq_vp_3d_b200.pair import DevicePair
    P, OP, u, w, g = problem
    free = DevicePair(P.grid, np.zeros(SHAPE), np.zeros(SHAPE), np.zeros(SHAPE + (3,)), lam=1e-4, mu=0., nu=0.,
                      kappa=.002)
    broken = u.copy()
    broken[NODE + (0,)] = np.nan
    node = np.ravel_multi_index([i - 1 for i in NODE], [n - 2 for n in SHAPE])      # the broken node's own u enters
    for term in ("jd", "curl"):
        got = free.gradient(dev(broken), w, g, term).cpu().numpy().reshape(3, -1)
        assert not np.delete(got, node, axis=1).any()


def test_folded_cells(problem):
    """Cells of negative J: each point with J <= delta is counted, the others form the barrier sum."""
    P, OP, u, w, g = problem
    rng = np.random.default_rng(9)
    folded = u.copy()
    folded[2:6, 3:7, 4:8] += rng.normal(size=(4, 4, 4, 3)) * .2
    J = Q.geometry(Q.local(folded, OP.grid), Q.ops(OP.grid, "closed27_uniform"))[2]
    bad = J <= 0
    assert bad.any() and np.abs(J).min() > 1e-9
    b = Q.barrier_terms(np.where(bad, 1., J), 0., OP.barrier_weight, OP.activation)[0].sum(dtype=np.longdouble)
    terms, count = P.energy(dev(folded), w)
    assert count == bad.sum()
    assert abs(terms[4] - float(b)) <= TOL * float(b)
    wu = P.warp(dev(u))[0]
    _, _, tterms, tcount, _, active = P.trial_energy(dev(u), wu, dev(folded))
    assert tcount == count and np.array_equal(active.cpu().numpy() != 0, (J < OP.activation).any(axis=1))
