"""Set-up passes of an event set at their edges: tile counts on both sides of the
shared-memory histogram's limit (8192 tiles), chunks of a few events on both
sides of the batch former's groups of four.
Images against the kernel that evaluates every pixel in the
reference's order, within the 1e-5 relative L2 per iteration of the parity
tests; counters equal.
"""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _events(n, half, seed):
    ell = phantom.random_ellipse_phantom(seed, half_z=half, half_y=half, centre_z=0.6 * half,
                                         centre_y=0.6 * half, axes=(10.0, 0.7 * half))
    return phantom.generate_events(ell, n, 450.0, 1000.0, 10.0, 42.0, seed=seed)


def _both(geom, ev, **opts):
    out = []
    for o in ({"variant": capi.VARIANT_EXACT}, opts):
        with capi.StripReconstruction(geom, **o) as rec:
            rec.set_events(ev)
            rec.iterate(1)
            out.append((rec.rho, rec.counters()))
    return out


@pytest.mark.parametrize("n_y,n_z", [(90, 91), (64, 128), (91, 91)])
def test_tiles_on_both_sides_of_the_histogram(n_y, n_z):
    geom = capi.Geometry(450.0, 1000.0, n_y, n_z, 4.0, 10.0, 42.0)
    (want, c0), (got, c1) = _both(geom, _events(20000, 180.0, 7), tile_w=1, tile_h=1)
    assert rel_l2(got, want) < 1e-5
    assert c1["n_kernel_calls"] == c0["n_kernel_calls"]
    assert c1["n_contributing"] == c0["n_contributing"]


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 12, 13, 65])
def test_few_events(n):
    geom = capi.Geometry(450.0, 1000.0, 101, 103, 4.0, 10.0, 42.0)
    (want, c0), (got, c1) = _both(geom, _events(n, 200.0, 8))
    assert rel_l2(got, want) < 1e-5
    assert c1["n_contributing"] == c0["n_contributing"]
