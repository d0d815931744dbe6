"""A batch tuned a second time, with events of another count octave in between,
runs the batch shapes that a batch tuned once runs: what the first tuning reports
of its plans is no request to the second.

The shape shows in the counters: events that are too large for its batches are
counted in n_exact_path, those too large for its windows in n_oversize, whatever
tile the tuner picks.  Images within 1e-5 relative L2: one kernel, the same
events, sums in another order."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

# (n_y, n_z, pixel, sigma_z, sigma_dl): boxes of 82 rows x 31 columns (12-warp CTAs),
# of 63 x 23 and of 26 x 11 (4-warp CTAs)
KINDS = [(131, 127, 2.0, 14.0, 55.0), (131, 127, 2.0, 10.0, 42.0), (61, 67, 5.0, 10.0, 42.0)]


def _events(g, n):
    ell = phantom.random_ellipse_phantom(seed=8, half_z=120.0, half_y=120.0, centre_z=60.0,
                                         centre_y=60.0, axes=(10.0, 80.0))
    return phantom.generate_events(ell, n, 450.0, 1000.0, g.sigma_z, g.sigma_dl, seed=n)


@pytest.mark.parametrize("first", [0, 700])  # an instance may also be empty at first
def test_second_tuning_runs_the_shapes_of_a_first_one(first):
    geoms = [capi.Geometry(450.0, 1000.0, *k) for k in KINDS]
    with capi.StripBatch(geoms) as again, capi.StripBatch(geoms) as fresh:
        for i, g in enumerate(geoms):
            again.set_events(i, _events(g, first))
        again.tune()
        for b in (again, fresh):
            for i, g in enumerate(geoms):
                b.set_events(i, _events(g, 20000))
            b.tune()
            b.iterate(1)
        for i in range(len(geoms)):
            a, f = again.instance(i).counters(), fresh.instance(i).counters()
            for key in ("n_oversize", "n_exact_path", "n_kernel_calls", "n_contributing"):
                assert a[key] == f[key], (i, key)
            assert again.plan(i)["block_threads"] == fresh.plan(i)["block_threads"], i
            x, y = again.instance(i).rho.astype(np.float64), fresh.instance(i).rho
            assert np.linalg.norm(x - y) < 1e-5 * np.linalg.norm(y), i
