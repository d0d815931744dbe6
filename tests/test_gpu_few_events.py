"""Sets of few events spread over the SMs in short chunks, and their images are those
of the kernel that evaluates every pixel in the reference's order (1e-5 relative L2
as in the other tests; the fixed-point mode rounds each contribution to 2^-22 of an
event, of images whose pixels hold a thousandth and more: 5e-4)."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

# (n_y, n_z, pixel, sigma_z, sigma_dl)
GRIDS = [(101, 117, 5.0, 10.0, 42.0), (125, 131, 4.0, 7.0, 44.0), (91, 97, 5.0, 20.0, 60.0)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 9, 300, 1000, 5000])
def test_few_events(grid, n):
    n_y, n_z, p, sz, sdl = grid
    g = capi.Geometry(450.0, 1000.0, n_y, n_z, p, sz, sdl)
    ell = phantom.random_ellipse_phantom(seed=3, half_z=n_z * p / 2, half_y=n_y * p / 2,
                                         centre_z=100.0, centre_y=90.0, axes=(10.0, 120.0))
    ev = phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=n)
    out = {}
    for name, opts in dict(exact=dict(variant=capi.VARIANT_EXACT), fp32={},
                           compensated=dict(precision=capi.PRECISION_COMPENSATED),
                           fixed=dict(precision=capi.PRECISION_FIXED)).items():
        with capi.StripReconstruction(g, **opts) as r:
            r.set_events(ev)
            r.iterate(1)
            out[name] = r.rho.astype(np.float64), r.counters()
    want, cnt = out.pop("exact")
    for name, (got, c) in out.items():
        assert c["n_kernel_calls"] == cnt["n_kernel_calls"], name
        assert c["n_contributing"] == cnt["n_contributing"], name
        assert c["n_chunks"] >= min(n, 1000) // 16, name
        tol = 5e-4 if name == "fixed" else 1e-5
        assert np.linalg.norm(got - want) < tol * np.linalg.norm(want), name
