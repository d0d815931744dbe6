"""Windows of the batch-union kernel that are narrow and tall (their rows are padded
in shared memory), or wider than a union row's word can address: every event set
that the other kernels take, it takes, in every accumulation mode.

Tolerance 1e-5 relative L2 against the kernel that evaluates every pixel in the
reference's order, as in the other iteration tests; the fixed-point mode rounds
every contribution to 2^-22 of an event, here of images whose pixels hold a
hundredth of an event and more: 1e-4."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

# (n_y, n_z, pixel width, pixel height, sigma_z, sigma_dl, options)
GRIDS = {
    "16 columns, boxes of 450 rows": (1000, 16, 0.3, 0.3, 3.0, 45.0, {}),
    "5 columns, boxes of 450 rows": (1000, 5, 0.3, 0.3, 3.0, 45.0, {}),
    "tiles of 800 columns": (91, 800, 1.0, 10.0, 8.0, 20.0, dict(tile_w=2000, tile_h=1)),
}
PRECISIONS = [capi.PRECISION_FP32, capi.PRECISION_COMPENSATED, capi.PRECISION_FP64_DEN,
              capi.PRECISION_FIXED]


def _image(g, ev, **opts):
    with capi.StripReconstruction(g, **opts) as r:
        r.set_events(ev)
        r.iterate(1)
        return r.rho.astype(np.float64), r.counters()


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("grid", GRIDS)
def test_window_shapes(grid, precision):
    n_y, n_z, pw, ph, sz, sdl, opts = GRIDS[grid]
    hz, hy = n_z * pw / 2, min(n_y * ph / 2, 430.0)
    ell = phantom.random_ellipse_phantom(seed=9, half_z=hz, half_y=hy, centre_z=0.8 * hz,
                                         centre_y=0.8 * hy, axes=(min(1.0, 0.5 * hz), hz))
    ev = phantom.generate_events(ell, 600, 450.0, 1000.0, sz, sdl, seed=9)
    g = capi.Geometry(450.0, 1000.0, n_y, n_z, pw, sz, sdl, ph)
    want, cnt = _image(g, ev, variant=capi.VARIANT_EXACT)
    got, c = _image(g, ev, precision=precision, **opts)
    assert c["n_kernel_calls"] == cnt["n_kernel_calls"]
    assert c["n_contributing"] == cnt["n_contributing"] > 300
    tol = 1e-4 if precision == capi.PRECISION_FIXED else 1e-5
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
