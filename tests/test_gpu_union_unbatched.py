"""Events that no batch of the batch-union kernel takes (rows of more than 40 pixels,
boxes of more than 96 rows) leave it to the large-box kernel where they are many:
rasterised one by one in its windows they took up to four times as long.

Counted in n_exact_path; images within 1e-5 relative L2 of the kernel that
evaluates every pixel in the reference's order, as in the other tests."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

# (pixel width, pixel height, sigma_z, sigma_dl, most events in n_exact_path)
SETS = {
    "rows of 43 pixels": (2.0, 2.0, 20.0, 60.0, 0.1),
    "rows of 40 pixels": (2.0, 2.0, 18.6, 60.0, 0.1),
    "rows of 39 pixels": (2.0, 2.0, 18.0, 60.0, 0.1),
    "boxes of 96 rows": (2.0, 2.0, 8.0, 64.0, 0.1),
    "boxes of 99 rows": (2.0, 2.0, 8.0, 66.0, 0.1),
    "boxes of 105 rows": (2.0, 2.0, 18.0, 70.0, 0.1),
    # the windows of the 64-row shape hold these
    "narrow boxes of 100 rows": (6.0, 1.5, 8.0, 50.0, 1.0),
}


def _image(g, ev, **opts):
    with capi.StripReconstruction(g, **opts) as r:
        r.set_events(ev)
        r.iterate(1)
        return r.rho.astype(np.float64), r.counters()


@pytest.mark.parametrize("events", SETS)
def test_events_beyond_the_batches(events):
    pw, ph, sz, sdl, most = SETS[events]
    g = capi.Geometry(450.0, 1000.0, int(800 / ph), int(800 / pw), pw, sz, sdl, ph)
    ell = phantom.random_ellipse_phantom(seed=7, half_z=400.0, half_y=400.0, centre_z=200.0,
                                         centre_y=200.0, axes=(10.0, 200.0))
    ev = phantom.generate_events(ell, 3000, 450.0, 1000.0, sz, sdl, seed=7)
    want, cnt = _image(g, ev, variant=capi.VARIANT_EXACT)
    got, c = _image(g, ev)
    assert c["n_kernel_calls"] == cnt["n_kernel_calls"]
    assert c["n_contributing"] == cnt["n_contributing"]
    assert c["n_exact_path"] <= most * len(ev)
    assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(want)
