"""dL/drho where very many events share a pixel: its sum keeps its digits.

The events are one event set repeated, so the exact gradient is a multiple of the
set's own, and only the sum's rounding tells the two apart: both round to float
once (2^-24 relative), and 2^-24 more is left for the additions' order."""
import numpy as np
import pytest

from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_EXACT])
def test_a_set_repeated_multiplies_its_gradient(variant):
    ell = phantom.random_ellipse_phantom(seed=2, half_z=80.0, half_y=80.0, centre_z=40.0,
                                         centre_y=40.0, axes=(10.0, 40.0))
    ev = phantom.generate_events(ell, 100, 450.0, 1000.0, 10.0, 42.0, seed=2)
    times = 8192
    rho = torch.from_numpy(np.random.default_rng(5).uniform(0.5, 2.0, (61, 67))
                           .astype(np.float32)).cuda()
    none = torch.zeros_like(rho)
    out = []
    for e in (ev, np.tile(ev, (times, 1))):
        grad = torch.empty_like(rho)
        torch.cuda.synchronize()
        with capi.StripReconstruction(capi.Geometry(450.0, 1000.0, 61, 67, 5.0, 10.0, 42.0),
                                      variant=variant) as rec:
            rec.set_events(e)
            rec.nll_grad(9.0, 40.0, rho.data_ptr(), none.data_ptr(), grad.data_ptr())
        out.append(grad.cpu().numpy().astype(np.float64))
    seen = out[0] < 0
    assert seen.any() and not out[1][~seen].any()
    assert np.abs(out[1][seen] / (times * out[0][seen]) - 1.0).max() <= 3 * 2.0**-24
