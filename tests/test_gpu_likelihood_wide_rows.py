"""The likelihood kernel on rows of more than 64 pixels (a lane's first two pixels
do not cover them) and of 65 and 33 to 64 pixels, where its pairs are ragged.

Tolerances against the FP64 oracle as in the other likelihood tests: loss 1e-6,
dL/drho 1e-5 relative L2; dL/dsigma, a sum in which the events' terms cancel,
2e-4 of the sum of their magnitudes' order (n / sigma)."""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (n_y, n_z, pixel, sigma_z, sigma_dl, events)
SIZES = {
    "rows of 53 pixels": (61, 97, 1.0, 12.2, 20.0, 65),
    "rows of 67 pixels": (61, 117, 1.0, 15.3, 20.0, 33),
    "rows of 143 pixels": (61, 203, 1.0, 33.3, 20.0, 9),
}


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_EXACT])
@pytest.mark.parametrize("size", SIZES)
def test_likelihood_of_wide_rows(size, variant):
    n_y, n_z, p, sz, sdl, n = SIZES[size]
    hz, hy = min(n_z * p / 2, 480.0), min(n_y * p / 2, 430.0)
    ell = phantom.random_ellipse_phantom(seed=41, half_z=hz, half_y=hy, centre_z=0.5 * hz,
                                         centre_y=0.5 * hy, axes=(0.2 * hy, 0.8 * min(hz, hy)))
    ev = phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=41)
    args = (450.0, 1000.0, n_y, n_z, p, sz, sdl)
    rho = np.random.default_rng(1).uniform(0.2, 2.0, (n_y, n_z)).astype(np.float32)
    kz, kdl = 0.9 * sz, 0.95 * sdl
    want_loss, want_grad, want_gs, want_sk = O.nll_grad(
        O.Geometry(*args[:5], kz, kdl), ev, rho, support_sigma=(sz, sdl))
    rho_d = torch.from_numpy(rho).cuda()
    grad = torch.full_like(rho_d, 7.0)  # what it held before does not matter
    torch.cuda.synchronize()
    with capi.StripReconstruction(capi.Geometry(*args), variant=variant) as rec:
        rec.set_events(ev)
        for g_ptr in (grad.data_ptr(), None):
            loss, gs, skipped = rec.nll_grad(kz, kdl, rho_d.data_ptr(), None, g_ptr)
            assert skipped == want_sk
            assert abs(loss - want_loss) <= 1e-6 * abs(want_loss)
            assert abs(gs[0] - want_gs[0]) <= 2e-4 * max(abs(want_gs[0]), n / kz)
            assert abs(gs[1] - want_gs[1]) <= 2e-4 * max(abs(want_gs[1]), n / kdl)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - want_grad) / np.linalg.norm(want_grad) < 1e-5
