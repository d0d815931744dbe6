"""The likelihood kernels on events of more rows than one block of their set-up holds
(96; 256 where rows may pass 64 pixels), and on either side of that row length.

Tolerances against the FP64 oracle as in the other likelihood tests: loss 1e-6,
dL/drho 1e-5 relative L2; dL/dsigma, a sum in which the events' terms cancel,
2e-4 of the sum of their magnitudes' order (n / sigma)."""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (n_y, n_z, pixel width, pixel height, sigma_z, sigma_dl, events)
SIZES = {
    "97 rows of 11 pixels": (181, 67, 2.0, 1.0, 5.0, 32.5, 40),
    "200 rows of 64 pixels": (301, 181, 1.0, 1.0, 15.0, 68.0, 7),
    "200 rows of 65 pixels": (301, 181, 1.0, 1.0, 15.2, 68.0, 7),
    "258 rows of 85 pixels": (401, 251, 0.5, 0.5, 10.0, 43.0, 9),
    "520 rows of 70 pixels": (701, 131, 1.0, 0.25, 16.3, 43.5, 5),
}


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_EXACT])
@pytest.mark.parametrize("size", SIZES)
def test_likelihood_of_several_blocks(size, variant):
    n_y, n_z, pw, ph, sz, sdl, n = SIZES[size]
    ell = phantom.random_ellipse_phantom(seed=41, half_z=n_z * pw / 2, half_y=n_y * ph / 2,
                                         centre_z=0.3 * n_z * pw, centre_y=0.1 * n_y * ph,
                                         axes=(1.0, 0.3 * n_z * pw))
    ev = phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=41)
    rho = np.random.default_rng(1).uniform(0.2, 2.0, (n_y, n_z)).astype(np.float32)
    kz, kdl = 0.9 * sz, 0.95 * sdl
    want_loss, want_grad, want_gs, want_sk = O.nll_grad(
        O.Geometry(450.0, 1000.0, n_y, n_z, pw, kz, kdl, ph), ev, rho, support_sigma=(sz, sdl))
    rho_d = torch.from_numpy(rho).cuda()
    grad = torch.empty_like(rho_d)
    torch.cuda.synchronize()
    with capi.StripReconstruction(capi.Geometry(450.0, 1000.0, n_y, n_z, pw, sz, sdl, ph),
                                  variant=variant) as rec:
        rec.set_events(ev)
        for g_ptr in (grad.data_ptr(), None):
            loss, gs, skipped = rec.nll_grad(kz, kdl, rho_d.data_ptr(), None, g_ptr)
            assert skipped == want_sk < n
            assert abs(loss - want_loss) <= 1e-6 * abs(want_loss)
            assert abs(gs[0] - want_gs[0]) <= 2e-4 * max(abs(want_gs[0]), n / kz)
            assert abs(gs[1] - want_gs[1]) <= 2e-4 * max(abs(want_gs[1]), n / kdl)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - want_grad) / np.linalg.norm(want_grad) < 1e-5
