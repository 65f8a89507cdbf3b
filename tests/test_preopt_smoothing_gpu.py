"""One pre-optimizer iteration with every smoothing radius (fused up to 3, separate passes above, none) on grids that
leave remainders in the fused tile, against the same formulas in float64: smoothed gradient, Adam step, capped update,
smoothed field.

Tolerance: 2e-5 of the largest entry.  The gradient and each of some 30 float32 products and sums round at 6e-8; eps
= 0.05 keeps the Adam quotient's derivative below 20 / max |g| of the data's gradients of order 1."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
SHAPES = [(7, 8, 9), (12, 19, 36), (29, 25, 58)]


def smooth(x, sigma):
    """Separable normalised Gaussian of radius ceil(3 sigma), replicate padding, z then y then x."""
    r = int(np.ceil(3 * sigma))
    k = np.exp(-.5 * (np.arange(-r, r + 1) / sigma) ** 2)
    k /= k.sum()
    for axis in (1, 2, 3):
        n = x.shape[axis]
        i = np.clip(np.arange(n)[:, None] + np.arange(-r, r + 1), 0, n - 1)
        x = np.tensordot(np.take(x, i, axis), k, ([axis + 1], [0]))
    return x


@pytest.mark.parametrize("sigma_grad,sigma_field", [(1., 1.), (.3, .6), (.6, 0.), (0., .3), (1.2, 1.), (1., 1.3)])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_one_iteration(shape, sigma_grad, sigma_field):
    from seq_vp_3d_b200 import _lib, preopt
    from seq_vp_3d_b200.device import ptr, stream_ptr
    from seq_vp_3d_b200.grid import grid_from_shape
    rng = np.random.default_rng(5)
    grid = grid_from_shape(shape, (1., 1.1, .9))
    dev = lambda a: torch.from_numpy(a.astype(np.float32)).cuda()
    F, M = dev(rng.random(shape) * 4), dev(rng.random(shape) * 4)
    u = dev(rng.normal(size=(3,) + grid.interior_shape) * .2)
    mu, alpha, kappa, j0, lr, cap, eps = .1, 1e-3, 10., .2, .5, .2, .05
    _, grad = preopt.pre_energy_grad(F, M, grid, u, mu, alpha, kappa, j0)
    g = grad.cpu().double().numpy()
    if sigma_grad:
        g = smooth(g, sigma_grad)
    step = lr * g / (np.abs(g) + eps)            # the first Adam iteration: bias-corrected moments are g and g^2
    largest = np.abs(step).max()
    assert largest > cap
    ref = u.cpu().double().numpy() - step * (cap / largest)
    if sigma_field:
        ref = smooth(ref, sigma_field)
    m, v = torch.zeros_like(u), torch.zeros_like(u)
    prm = _lib.PreParams(mu, alpha, kappa, j0, lr, cap, sigma_grad, sigma_field, .9, .99, eps)
    first, last, hits = (ctypes.c_float * 6)(), (ctypes.c_float * 6)(), ctypes.c_int64()
    _lib.call("svp_pre_level", ptr(F), ptr(M), *shape, *grid.spacing, ctypes.byref(prm), 0, 1, ptr(u), ptr(m), ptr(v),
              first, last, ctypes.byref(hits), stream_ptr())
    assert hits.value == 1 and list(first) == list(last)
    assert np.abs(u.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()
