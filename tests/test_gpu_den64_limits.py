"""Double-float denominators (FP64_DEN) at the limits of their range.  A batch's
contribution K rho / sum K rho does not change when rho is scaled by a power of
two: images agree to 1e-6 relative L2 (the order of the window flushes; 24 bits
per addition).  Where the sums overflow the reciprocal is zero: nothing is
added, but the event is still counted, as in the single-precision mode.
"""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

# batches of 64 x 32, 32 x 16, 96 x 40 pixels; 128 threads: 4 events a batch
SHAPES = [(101, 103, 2.0, 10.0, 42.0, 0), (101, 103, 5.0, 10.0, 42.0, 0),
          (151, 103, 2.0, 14.0, 60.0, 0), (101, 103, 2.0, 10.0, 42.0, 128)]


def _run(shape, precision, value):
    n_y, n_z, p, sz, sdl, threads = shape
    half = 0.4 * n_z * p
    ell = phantom.random_ellipse_phantom(seed=9, half_z=half, half_y=half, centre_z=0.6 * half,
                                         centre_y=0.6 * half, axes=(10.0, 0.7 * half))
    ev = phantom.generate_events(ell, 5001, 450.0, 1000.0, sz, sdl, seed=9)
    with capi.StripReconstruction(capi.Geometry(450.0, 1000.0, n_y, n_z, p, sz, sdl),
                                  precision=precision, block_threads=threads) as rec:
        rec.set_events(ev)
        rec.rho = np.full((n_y, n_z), value, np.float32)
        rec.iterate(1)
        return np.asarray(rec.rho, np.float64), rec.counters()["n_contributing"]


@pytest.mark.parametrize("shape", SHAPES)
def test_range_of_the_denominators(shape):
    one, count = _run(shape, capi.PRECISION_FP64_DEN, 1.0)
    for exponent in (-90, 100):
        img, n = _run(shape, capi.PRECISION_FP64_DEN, 2.0 ** exponent)
        assert n == count
        assert np.linalg.norm(img - one) < 1e-6 * np.linalg.norm(one)
    # at 3e38 only an event whose pixels are a few at the image's border stays in range
    (a, na), (b, nb) = (_run(shape, p, 3e38)
                        for p in (capi.PRECISION_FP64_DEN, capi.PRECISION_FP32))
    assert na == nb == count
    assert np.isfinite(a).all() and a.sum() < 0.02 * count
    assert abs(a.sum() - b.sum()) < 1.0
