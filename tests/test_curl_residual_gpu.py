"""The curl penalty of a state close to its reference.  The curl is linear, so the penalty and its gradient depend on u
- u_ref alone, however large u is against it: on a dyadic lattice, where the difference is exact, they are those of u -
u_ref against a zero reference.  Odd grids, anisotropic voxels.

Tolerance: 1e-14 relative.  The coefficients of the difference round relative to themselves (a few 1e-16 each); the
difference of the two fields' coefficients would round relative to |grad u|, here 1e5 times larger."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing", [((5, 5, 5), (1., 1., 1.)), ((9, 33, 18), (.9, 1.1, 1.3)),
                                           ((12, 7, 66), (1.25, 1., .9))])
def test_small_residual(shape, spacing):
    from seq_vp_3d_b200.grid import grid_from_shape
    from seq_vp_3d_b200.pair import DevicePair
    rng = np.random.default_rng(11)
    lattice = 2. ** -46
    noise = lambda a: np.round(rng.normal(size=shape + (3,)) * a / lattice) * lattice
    ref, d = noise(.1), noise(1e-6)
    grid, zero = grid_from_shape(shape, spacing), np.zeros(shape)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    w = dict(lam=1e-4, mu=0., nu=.03, kappa=.002)
    near = DevicePair(grid, zero, zero, ref, **w)
    alone = DevicePair(grid, zero, zero, np.zeros(shape + (3,)), **w)
    image, image_grad = dev(zero), dev(np.zeros(shape + (3,)))
    got, want = near.energy(dev(ref + d), image)[0][3], alone.energy(dev(d), image)[0][3]
    assert want > 0 and abs(got - want) <= 1e-14 * want
    got, want = (P.gradient(dev(u), image, image_grad, "curl") for P, u in ((near, ref + d), (alone, d)))
    assert float((got - want).norm()) <= 1e-14 * float(want.norm())
    # and the change from one such state to another: the penalty of the second less that of the first
    e = noise(1e-6)
    got = near.energy_difference(dev(ref + d), image, dev(ref + e), image)[0]
    want = alone.energy_difference(dev(d), image, dev(e), image)[0]
    scale = sum(alone.energy(dev(v), image)[0].sum() for v in (d, e))
    assert abs(got - want) <= 1e-14 * scale
