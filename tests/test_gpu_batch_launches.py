"""Kernels per batched iteration: every instance's clear, its events' kernel and, for
events too large for its windows, the large-box kernel; with too little memory for
all row records, two per part of them."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _events(n, sz, sdl):
    ell = phantom.random_ellipse_phantom(seed=5, half_z=120.0, half_y=120.0, centre_z=60.0,
                                         centre_y=60.0, axes=(10.0, 80.0))
    return phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=5)


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_ROWS])
def test_kernels_of_a_batched_iteration(variant):
    small = capi.Geometry(450.0, 1000.0, 61, 67, 5.0, 10.0, 42.0)
    large = capi.Geometry(450.0, 1000.0, 260, 260, 1.0, 14.0, 60.0)
    with capi.StripBatch([small, small, large], variant=variant) as b:
        b.set_events(0, _events(2000, 10.0, 42.0))
        b.set_events(1, np.zeros((0, 3), np.float32))
        b.set_events(2, _events(2000, 14.0, 60.0))
        assert b.launches_per_iteration() == 0
        b.iterate(2)
        c = b.instance(2).counters()
        assert c["n_oversize"] > 0
        assert b.launches_per_iteration() == 2 + 1 + 2 + (c["n_chunks"] > 0)


def test_kernels_with_records_in_parts():
    g = capi.Geometry(450.0, 1000.0, 131, 127, 2.0, 10.0, 42.0)
    n = 3_000_000  # 3 GB of records; the other event arrays take about 1 GB
    ev = _events(n, 10.0, 42.0)
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - 4 * 2**30, dtype=torch.uint8, device="cuda")
    try:
        with capi.StripBatch([g]) as b:
            b.set_events(0, ev)
            b.iterate(1)
            parts = (b.launches_per_iteration() - 1 - (b.instance(0).counters()["n_oversize"] > 0))
            assert parts >= 4 and parts % 2 == 0  # two parts or more
    finally:
        del held
        torch.cuda.empty_cache()
