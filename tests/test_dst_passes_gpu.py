"""The DST-I passes of the Q1 Poisson metric at the edges of their tiles: half axes of 15, 16 and 17 rows (one m16 tile
and the next) and of 31 to 33 (the two row warps), K blocks of 16 that end inside a step, column ranges that end inside
a block and cross components, odd axes with a middle row, axes shorter than a step.  Against the oracle's dense float64
DST-I (oracle/q1.py poisson_apply, scipy's dstn type 1 'ortho' restated)."""
import numpy as np
import pytest

from oracle import q1 as Q

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a).ravel() - np.asarray(b).ravel()) / np.linalg.norm(np.asarray(b).ravel())


# free nodes per axis are the shape less 2: (nz, ny, nx)
@pytest.mark.parametrize("shape", [(31, 33, 32), (32, 34, 35), (36, 31, 66), (64, 65, 35), (67, 36, 68), (5, 6, 131),
                                   (100, 7, 5), (6, 98, 7)])
@pytest.mark.parametrize("form,tol", [("plain", 1e-12), ("mixed", 1e-5)])
def test_poisson_apply(shape, form, tol):
    import torch
    from seq_vp_3d_b200.grid import make_grid_3d
    from seq_vp_3d_b200.pair import DevicePair
    nz, ny, nx = shape
    rng = np.random.default_rng(5)
    grid = make_grid_3d(nx=nx, ny=ny, nz=nz, hx=1.1, hy=0.9, hz=1.0, unit="mm")
    og = Q.make_grid(shape, (1.1, 0.9, 1.0))   # (hx, hy, hz)
    img = rng.random(shape)
    nf = 3 * int(np.prod(og.interior_shape))
    rhs, scale = rng.normal(size=nf), rng.random(nf) + .5
    P = DevicePair(grid, img, img, np.zeros(shape + (3,)), lam=.02, mu=.03, nu=.03, kappa=.002, precision=form)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    got = P.poisson_apply(.02, .03, dev(rhs)).cpu().numpy()
    assert rel(got, Q.poisson_apply(og, .02, .03, rhs)) < tol
    got = P.poisson_apply(.02, .03, dev(rhs), scale=dev(scale), sign=-1.).cpu().numpy()
    assert rel(got, -scale * Q.poisson_apply(og, .02, .03, scale * rhs)) < tol
