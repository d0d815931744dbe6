"""The likelihood of images at the ends of FP32's range: denominators beyond its
largest and below its smallest normal value, and a pixel of infinite activity, are
summed and divided in FP64.

Tolerances: loss 1e-6 as in the other likelihood tests; with an image of 1e-42, a
multiple 714 of the smallest float, each pixel's product is rounded by up to a
part in 1400 and an event's logarithm, of about 93, by less than 1e-5 of itself.
dL/drho 1e-5 relative L2."""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ARGS = (450.0, 1000.0, 91, 97, 2.0, 10.0, 42.0)
N = 300


def _run(rho, variant, sens):
    ell = phantom.random_ellipse_phantom(seed=2, half_z=80.0, half_y=80.0, centre_z=40.0,
                                         centre_y=40.0, axes=(10.0, 40.0))
    ev = phantom.generate_events(ell, N, 450.0, 1000.0, 10.0, 42.0, seed=2)
    with np.errstate(over="ignore"):
        want = O.nll_grad(O.Geometry(*ARGS), ev, rho, s=sens)
    rho_d, sens_d = torch.from_numpy(rho).cuda(), torch.from_numpy(sens).cuda()
    grad = torch.empty_like(rho_d)
    torch.cuda.synchronize()
    with capi.StripReconstruction(capi.Geometry(*ARGS), variant=variant) as rec:
        rec.set_events(ev)
        loss, _, skipped = rec.nll_grad(10.0, 42.0, rho_d.data_ptr(), sens_d.data_ptr(),
                                        grad.data_ptr())
    return loss, skipped, grad.cpu().numpy().astype(np.float64), want


VARIANTS = pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_EXACT])


@VARIANTS
def test_denominators_beyond_the_largest_float(variant):
    rho = np.full((91, 97), 2e36, np.float32)
    loss, skipped, g, want = _run(rho, variant, np.ones((91, 97), np.float32))
    assert skipped == want[3] == 0
    assert abs(loss - want[0]) <= 1e-6 * abs(want[0])
    assert np.array_equal(g, want[1].astype(np.float32))  # 1 less some 1e-37: 1


@VARIANTS
def test_denominators_below_the_smallest_normal_float(variant):
    rho = np.full((91, 97), 1e-42, np.float32)
    loss, skipped, g, want = _run(rho, variant, np.ones((91, 97), np.float32))
    assert skipped == want[3] == 0
    assert abs(loss - want[0]) <= 2e-5 * abs(want[0])
    with np.errstate(over="ignore"):
        expect = want[1].astype(np.float32)
    assert not np.isnan(g).any()
    assert np.isneginf(g[np.isneginf(expect)]).mean() > 0.99  # K / den is no float


@VARIANTS
def test_an_infinite_pixel_takes_its_events_out(variant):
    rho = np.random.default_rng(3).uniform(0.5, 2.0, (91, 97)).astype(np.float32)
    rho[45, 48] = np.inf
    loss, skipped, g, want = _run(rho, variant, np.zeros((91, 97), np.float32))
    assert skipped == want[3] == 0
    assert np.isfinite(want[1]).all() and (want[1] < 0).any()
    assert np.linalg.norm(g - want[1]) < 1e-5 * np.linalg.norm(want[1])


@VARIANTS
def test_negative_denominators_are_skipped(variant):
    rho = np.full((91, 97), -1.0, np.float32)
    _, skipped, g, want = _run(rho, variant, np.ones((91, 97), np.float32))
    assert skipped == want[3] > N // 2
    assert np.array_equal(g, np.ones((91, 97)))
