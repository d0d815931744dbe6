"""Captured batch graphs follow their handles: images and event sets changed
through an instance's own handle between batched iterations, more iteration
counts than graphs kept; and two live handles whose kernels need different
amounts of shared memory.  Tolerance 1e-5: one kernel, the same events, sums in
another order."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _case(n, seed, p=4.0, sz=10.0, sdl=42.0):
    ell = phantom.random_ellipse_phantom(seed, half_z=200.0, half_y=180.0, centre_z=100.0,
                                         centre_y=80.0, axes=(10.0, 120.0))
    ev = phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=seed)
    return capi.Geometry(450.0, 1000.0, 91, 103, p, sz, sdl), ev


def _single(g, ev, n, rho=None):
    with capi.StripReconstruction(g) as r:
        r.set_events(ev)
        if rho is not None:
            r.rho = rho
        r.iterate(n)
        return r.rho


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_ROWS])
def test_graphs_follow_their_handles(variant):
    (g, a), (_, c) = _case(4000, 3), _case(2500, 4)
    with capi.StripBatch([g, g], variant=variant) as b:
        b.set_events(0, a)
        b.set_events(1, c)
        b.iterate(1)
        b.instance(0).iterate(1)  # the handle's buffers swap outside the batch
        b.iterate(1)
        assert rel_l2(b.instance(0).rho, _single(g, a, 3)) < TOL
        assert rel_l2(b.instance(1).rho, _single(g, c, 2)) < TOL
        before = b.instance(0).rho
        b.instance(0).set_events(c)  # another event set through the handle
        b.iterate(1)
        assert rel_l2(b.instance(0).rho, _single(g, c, 1, before)) < TOL
        start = b.instance(1).rho
        for n in range(1, 19):  # more iteration counts than graphs are kept
            b.instance(1).rho = start
            b.iterate(n)
        assert rel_l2(b.instance(1).rho, _single(g, c, 18, start)) < 1e-4


def test_two_live_handles_of_one_kernel_with_different_windows():
    (g, a), (h, c) = _case(3000, 5, p=2.0, sdl=42.0), _case(3000, 6, p=2.0, sz=6.0, sdl=24.0)
    with capi.StripReconstruction(g) as r, capi.StripReconstruction(h) as s:
        r.set_events(a)  # the larger windows first
        s.set_events(c)
        r.iterate(1)
        s.iterate(1)
        assert rel_l2(r.rho, _single(g, a, 1)) < TOL
        assert rel_l2(s.rho, _single(h, c, 1)) < TOL
