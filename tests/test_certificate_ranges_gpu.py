"""The certificate's fast forms (edge hull with one finiteness check, prescreen with shared sums) and its fused first
stage against the C oracle, bit for bit, on fields where their range checks decide: zeros and equal magnitudes
(maximum sums that tie), subnormal and huge values, NaN and infinities, flat and folded cells."""
import numpy as np
import pytest

from conftest import same_bits, same_bits_nan
from oracle import cert as oc

pytestmark = pytest.mark.gpu
SHAPES = [((9, 8, 37), (1., 1., 1.)), ((6, 11, 35), (.9, 1.1, 1.3))]
TINY = 4.9406564584124654e-324


def fields(shape, spacing):
    rng = np.random.default_rng(2)
    h, n = np.array(spacing), shape + (3,)
    out = {"smooth": rng.normal(size=n) * 1e-3 * h, "rough": rng.uniform(-.27, .27, n) * h,
           "folding": rng.uniform(-.6, .6, n) * h, "zero": np.zeros(n), "constant": np.full(n, .37),
           "equal magnitudes": rng.integers(-1, 2, n) * .2 * h, "subnormal": rng.integers(-3, 4, n) * TINY,
           "small": rng.normal(size=n) * 10. ** rng.uniform(-320, -290, n),
           "large": rng.normal(size=n) * 10. ** rng.uniform(100, 160, n),
           "overflowing": rng.uniform(-1, 1, n) * 10. ** rng.uniform(290, 308, n)}
    flat = np.zeros(n)
    flat[..., 0] = -np.arange(shape[2]) * h[0]
    out["flat"] = flat
    some = rng.random(n) < .2
    out["some subnormal"] = np.where(some, rng.integers(-2, 3, n) * TINY, out["rough"])
    out["nan"] = np.where(rng.random(n) < .01, np.nan, out["rough"])
    out["infinite"] = np.where(rng.random(n) < .01, np.inf, out["rough"])
    return out


NAMES = sorted(fields((5, 5, 5), (1., 1., 1.)))


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("shape,spacing", SHAPES, ids=["unit", "anisotropic"])
def test_margins_bounds_and_record(shape, spacing, name):
    from seq_vp_3d_b200 import certificate as cert
    from seq_vp_3d_b200.grid import grid_from_shape
    grid = grid_from_shape(shape, spacing)
    u = fields(shape, spacing)[name]
    for delta in (0., .01):
        m, f = cert.parallel_margins(u, grid, delta)
        om, of = oc.edge_hull(u, grid.spacing, delta)
        assert np.array_equal(f, of) and same_bits_nan(m, om)
    if np.isfinite(u).all():
        cells = np.arange(grid.n_cells)
        got = cert.prescreen_lower_bounds(u, grid, cert._closed27(grid.spacing), cells)
        assert same_bits_nan(got, oc.prescreen(u, grid.spacing, cells))
    inside = u.copy()
    inside[[0, -1]] = 0.
    inside[:, [0, -1]] = 0.
    inside[:, :, [0, -1]] = 0.
    for v in (u, inside):
        for tile in (64, 65536):
            config = cert.PrescreenCertificateConfig(delta=0., max_depth=48, max_boxes=255, tile_size=tile)
            got = cert.certify_map(v, grid, config=config, with_hash=False)
            ri, rf = oc.certify_map(v, np.array(spacing), 0., tile_size=tile)
            assert got.status == cert.STATUS[ri[0]] and got.n_boxes == ri[5]
            assert (got.n_uncertain, got.n_infeasible) == (ri[3], ri[4])
            assert (got.n_fast_cells, got.n_fallback_cells, got.n_prescreen_cells) == (ri[8], ri[9], ri[10])
            if got.min_jd_lower_bound is not None:
                assert same_bits(np.array([got.min_jd_lower_bound]), np.array([rf[0]]))
