"""Grids large enough that the kernels' inner loops run more than once: a block of the barrier kernels scans several
groups of cells, queues more than it evaluates at a time and carries the rest over; a block of the cell kernels takes
several rounds; a warp of the certificate's first stage writes its list out before it ends; an axis of the DST-I takes
the widest row tiles."""
import numpy as np
import pytest
import torch

from oracle import q1 as Q

pytestmark = pytest.mark.gpu
TOL = 1e-12
W = dict(lam=1e-4, mu=.03, nu=.03, kappa=.002)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rel(got, ref):
    return np.linalg.norm(np.asarray(got) - ref) / np.linalg.norm(ref)


@pytest.fixture(scope="module")
def active_pair():
    """284,000 cells, nearly all of them below the activation."""
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    shape = (63, 67, 70)
    rng = np.random.default_rng(7)
    ident = Q.make_grid(shape, (1., 1., 1.)).identity()
    squeeze = np.array([-.97, 0., 0.]) * (ident - np.array([34.5, 33., 31.]))
    base = squeeze + rng.normal(size=shape + (3,)) * .002
    trial, ref = base + rng.normal(size=shape + (3,)) * .001, rng.normal(size=shape + (3,)) * .003
    fixed, moving = rng.random(shape), rng.random(shape)
    P = DevicePair(grid_from_shape(shape, (1., 1., 1.)), fixed, moving, ref, **W)
    OP = Q.make_problem(Q.make_grid(shape, (1., 1., 1.)), fixed, moving, ref, *W.values())
    return P, OP, base, trial


def test_barrier_of_many_cells(active_pair):
    P, OP, base, trial = active_pair
    op = Q.ops(OP.grid, "closed27_uniform")
    J = Q.geometry(Q.local(trial, OP.grid), op)[2]
    bd, td = dev(base), dev(trial)
    wb = P.warp(bd)[0]
    _, _, terms, count, diff, active = P.trial_energy(bd, wb, td)
    mask = (J < OP.activation).any(axis=1)
    assert mask.mean() > .95 and np.array_equal(active.cpu().numpy() != 0, mask) and count == 0
    b = Q.barrier_terms(J, 0., OP.barrier_weight, OP.activation)[0].sum(dtype=np.longdouble)
    assert abs(terms[4] - float(b)) <= TOL * float(b)
    got, n = P.energy(td, P.warp(td)[0])
    assert n == count and got[4] == terms[4]


def test_energies_of_many_cells(active_pair):
    P, OP, base, trial = active_pair
    ref = Q.energy(OP, base)
    terms, bad = P.energy(dev(base), P.warp(dev(base))[0])
    assert bad == 0 and np.all(np.abs(terms - ref) <= TOL * ref)
    ob, ot = Q.warp(OP, base)[0], Q.warp(OP, trial)[0]
    dE, dF = Q.differences(OP, base, ob, trial, ot)
    got = P.energy_difference(dev(base), dev(ob), dev(trial), dev(ot))
    assert abs(got[0] - dE) <= 2 * TOL * ref.sum() and abs(got[1] - dF) <= 2 * TOL * (ref[0] + ref[4])


def test_derivatives_of_many_cells(active_pair):
    P, OP, base, trial = active_pair
    bd = dev(base)
    w, g = P.warp(bd, with_gradient=True)
    ow, og = Q.warp(OP, base, True)
    for got, term in zip(P.outer_gradients(bd, w, g), ("outer", "image", "total")):
        assert rel(got.cpu().numpy(), Q.gradient(OP, base, ow, og, term)) <= TOL
    assert rel(P.ggn_diagonal(bd, g).cpu().numpy(), Q.ggn_diagonal(OP, base, og)) <= TOL


def test_certificate_of_many_cells():
    """2.9 M cells that nearly all miss the edge hull's proof, a quarter of them also the prescreen's: the fused first
    stage's counts against the per-cell arrays of the separate entry points."""
    from seq_vp_3d_b200 import certificate as cert
    from seq_vp_3d_b200.grid import grid_from_shape
    n = 143
    grid = grid_from_shape((n, n, n), (1., 1., 1.))
    rng = np.random.default_rng(3)
    u = rng.uniform(-.45, .45, (n, n, n, 3))
    u[[0, -1]] = 0.
    u[:, [0, -1]] = 0.
    u[:, :, [0, -1]] = 0.
    ud = dev(u)
    margin = np.asarray(cert.parallel_margins(u, grid, 0.)[0])
    left = np.flatnonzero(~(margin > 0))
    low = np.asarray(cert.prescreen_lower_bounds(u, grid, cert._closed27(grid.spacing), left))
    config = cert.PrescreenCertificateConfig(delta=0., max_depth=48, max_boxes=255, tile_size=65536)
    got = cert.certify_map(ud, grid, config=config, with_hash=False)
    proven = low > 0
    assert left.size > 2.6e6 and (~proven).sum() > 6e5
    assert got.n_fast_cells == margin.size - left.size
    assert got.n_prescreen_cells == proven.sum() and got.n_fallback_cells == (~proven).sum()


# free nodes per axis are the shape less 2: 193, 222 and 254 take four m16 tiles per warp
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [193, 222, 254])
@pytest.mark.parametrize("form,tol", [("plain", 1e-12), ("mixed", 1e-5)])
def test_poisson_apply_widest_tiles(axis, n, form, tol):
    from seq_vp_3d_b200.grid import make_grid_3d
    from seq_vp_3d_b200.pair import DevicePair
    shape = [7, 9, 8]
    shape[axis] = n + 2
    nz, ny, nx = shape
    rng = np.random.default_rng(5)
    grid = make_grid_3d(nx=nx, ny=ny, nz=nz, hx=1.1, hy=0.9, hz=1.0, unit="mm")
    og = Q.make_grid(tuple(shape), (1.1, 0.9, 1.0))
    img = rng.random(shape)
    nf = 3 * int(np.prod(og.interior_shape))
    rhs, scale = rng.normal(size=nf), rng.random(nf) + .5
    P = DevicePair(grid, img, img, np.zeros(tuple(shape) + (3,)), lam=.02, mu=.03, nu=.03, kappa=.002, precision=form)
    got = P.poisson_apply(.02, .03, dev(rhs), scale=dev(scale), sign=-1.).cpu().numpy()
    assert rel(got, -scale * Q.poisson_apply(og, .02, .03, scale * rhs)) < tol
