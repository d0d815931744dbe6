"""Row records of the batch-union kernel when device memory does not hold all of
them: the iteration writes and reads them part by part.

The fixed-point image is a sum of integers, so it does not depend on the order
or the launch in which events are added: equal to the last bit.  The FP32 image
differs by the order of the window flushes, each pixel a sum of positive numbers
with at most one term per chunk (n / 256 chunks at the least): the bar is that
number times 2^-24, at most 7.5e-4, and 1e-5 is expected of random roundings.
"""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

GEOMETRY = capi.Geometry(450.0, 1000.0, 131, 127, 2.0, 10.0, 42.0)


def _iterate(ev, precision):
    with capi.StripReconstruction(GEOMETRY, precision=precision) as rec:
        rec.set_events(ev)
        rec.iterate(2)
        return rec.rho, rec.counters()


@pytest.mark.parametrize("precision", [capi.PRECISION_FIXED, capi.PRECISION_FP32])
def test_parts_match_the_whole(precision):
    torch = pytest.importorskip("torch")
    ell = phantom.random_ellipse_phantom(seed=5, half_z=127.0, half_y=131.0, centre_z=70.0,
                                         centre_y=70.0, axes=(10.0, 100.0))
    ev = phantom.generate_events(ell, 3_000_000, 450.0, 1000.0, 10.0, 42.0, seed=5)
    want, cnt = _iterate(ev, precision)
    # 3 GB of records; the other event arrays take about 1 GB
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - 4 * 2**30, dtype=torch.uint8, device="cuda")
    try:
        got, cnt_parts = _iterate(ev, precision)
    finally:
        del held
        torch.cuda.empty_cache()
    assert cnt_parts == cnt
    if precision == capi.PRECISION_FIXED:
        assert np.array_equal(got, want)
    else:
        scale = np.abs(want).max()
        assert np.abs(got - want).max() < 1e-5 * scale


def test_an_empty_set_after_a_full_one():
    ell = phantom.random_ellipse_phantom(seed=6, half_z=127.0, half_y=131.0, centre_z=70.0,
                                         centre_y=70.0, axes=(10.0, 100.0))
    ev = phantom.generate_events(ell, 2000, 450.0, 1000.0, 10.0, 42.0, seed=6)
    with capi.StripReconstruction(GEOMETRY) as rec:
        rec.set_events(ev)
        rec.iterate(1)
        rec.set_events(ev[:0])
        rec.iterate(1)
        assert not rec.rho.any()
