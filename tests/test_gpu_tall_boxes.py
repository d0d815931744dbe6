"""Boxes taller than the batch-union kernel's batches stay in the windows of the other
kernels where those hold them.  Image within 1e-5 relative L2 of the kernel that
evaluates every pixel in the reference's order."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(variant=capi.VARIANT_ROWS, block_threads=256),
                                  dict(variant=capi.VARIANT_WARP)], ids=["rows", "warp"])
def test_boxes_of_105_rows(opts):
    g = capi.Geometry(450.0, 1000.0, 300, 300, 2.0, 8.0, 70.0)
    ell = phantom.random_ellipse_phantom(seed=7, half_z=300.0, half_y=300.0, centre_z=150.0,
                                         centre_y=150.0, axes=(10.0, 150.0))
    ev = phantom.generate_events(ell, 2000, 450.0, 1000.0, 8.0, 70.0, seed=7)
    out = []
    for o in (dict(variant=capi.VARIANT_EXACT), opts):
        with capi.StripReconstruction(g, **o) as r:
            r.set_events(ev)
            r.iterate(1)
            out.append((r.rho.astype(np.float64), r.counters()))
    (want, cnt), (got, c) = out
    assert c["n_oversize"] <= len(ev) // 100
    assert c["n_kernel_calls"] == cnt["n_kernel_calls"]
    assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(want)
