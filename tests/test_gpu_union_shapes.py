"""Every batch shape of the batch-union iteration kernel at the sizes where the
shape changes: box rows and in-ellipse columns on both sides of each limit,
odd grids with tile remainders, few and many events per pixel.

Tolerances: one iteration within 1e-5 relative L2 of the reference float path
(the bar the path is built to), 3e-5 in the fixed-point mode (one rounding to
2^-22 of an event per batch and pixel, about 1e-5 relative at these event
densities); counters identical.
"""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

PRECISIONS = [capi.PRECISION_FP32, capi.PRECISION_COMPENSATED, capi.PRECISION_FP64_DEN,
              capi.PRECISION_FIXED]
# (n_y, n_z, pixel, sigma_z, sigma_dl, events): box rows 2 int(1.5 sigma_dl / p + 0.5),
# widest row 2 int(2.12 sigma_z / p) + 3 columns
SHAPES = {
    "26 rows x 11 columns": (101, 117, 5.0, 10.0, 42.0, 3001),
    "26 rows x 11 columns, dense": (61, 67, 5.0, 10.0, 42.0, 40000),
    "30 rows x 13 columns": (131, 127, 4.0, 10.0, 41.0, 3001),
    "30 rows x 15 columns": (131, 127, 4.0, 11.5, 41.0, 3001),
    "32 rows x 13 columns": (131, 127, 4.0, 10.0, 42.0, 3001),
    "46 rows x 11 columns": (197, 203, 4.0, 8.0, 62.0, 3001),
    "32 rows x 9 columns, dense": (61, 67, 4.0, 7.0, 44.0, 40000),
    "64 rows x 13 columns": (197, 203, 2.0, 5.3, 42.0, 3001),
    "24 rows x 27 columns": (131, 127, 2.3, 13.2, 18.0, 3001),
    "24 rows x 29 columns": (131, 127, 2.1, 13.2, 16.5, 3001),
    "64 rows x 23 columns": (197, 203, 2.0, 10.0, 42.0, 3001),
    "66 rows x 23 columns": (197, 203, 2.0, 10.0, 44.0, 3001),
    "64 rows x 31 columns": (197, 203, 2.0, 14.0, 42.0, 3001),
    "90 rows x 31 columns": (297, 203, 2.0, 14.0, 60.0, 3001),
    "96 rows x 17 columns": (297, 203, 2.0, 7.0, 64.0, 3001),
    "98 rows x 39 columns": (297, 203, 2.0, 17.0, 65.5, 2001),
}


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _events(n_y, n_z, p, sz, sdl, n):
    hz, hy = min(n_z * p / 2, 480.0), min(n_y * p / 2, 430.0)
    ell = phantom.random_ellipse_phantom(seed=21, half_z=hz, half_y=hy, centre_z=0.6 * hz,
                                         centre_y=0.6 * hy, axes=(10.0, 0.8 * min(hz, hy)))
    return phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=21)


@pytest.mark.parametrize("shape", SHAPES)
def test_every_batch_shape_matches_the_reference_path(shape):
    n_y, n_z, p, sz, sdl, n = SHAPES[shape]
    ev = _events(n_y, n_z, p, sz, sdl, n)
    args = (450.0, 1000.0, n_y, n_z, p, sz, sdl)
    want, st = O.mlem_f(O.Geometry(*args), ev, 1, threads=8)
    for precision in PRECISIONS:
        with capi.StripReconstruction(capi.Geometry(*args), precision=precision) as rec:
            rec.set_events(ev)
            rec.iterate(1)
            got, cnt = rec.rho, rec.counters()
        tol = 3e-5 if precision == capi.PRECISION_FIXED else 1e-5
        assert rel_l2(got, want) < tol, (precision, rel_l2(got, want))
        assert cnt["n_kernel_calls"] == st["n_kernel_calls"]
        assert cnt["n_contributing"] == st["n_contributing"]
