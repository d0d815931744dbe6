"""The likelihood kernel's row prefactor far from the event's own row: a scanner of
30 mm radius with events smeared to 2.5 radii, where the prefactor of a row near
the centre is a tenth of that of the event's row.

Tolerance: a kernel value is 2 to the power of an argument of at most about 10 that
is rounded to float, with positions rounded to 2^-24 of 100 mm: 3e-6 of itself at
most, so a pixel's gradient, a quotient of sums of such values, 2e-5; of 99 of
100 pixels, as a pixel on the edge of an event's support may fall to either side in
the oracle's doubles.  The loss 1e-6 as in the other likelihood tests."""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("variant", [capi.VARIANT_FAST, capi.VARIANT_EXACT])
def test_rows_far_from_the_event(variant):
    rng = np.random.default_rng(4)
    n, radius, sz, sdl = 400, 30.0, 10.0, 60.0
    y, z = rng.uniform(60.0, 78.0, n) * rng.choice([-1.0, 1.0], n), rng.uniform(-20.0, 20.0, n)
    t = rng.uniform(-0.4, 0.4, n)
    ev = np.stack([z + (radius - y) * t, z - (radius + y) * t, -2 * y * np.sqrt(1 + t * t)],
                  1).astype(np.float32)
    args = (radius, 200.0, 81, 41, 2.0, sz, sdl)
    rho = rng.uniform(0.2, 2.0, (81, 41)).astype(np.float32)
    none = np.zeros_like(rho)  # no sensitivity: the gradient is the events' sum alone
    want_loss, want, _, want_sk = O.nll_grad(O.Geometry(*args), ev, rho, s=none)
    rho_d, none_d = torch.from_numpy(rho).cuda(), torch.from_numpy(none).cuda()
    grad = torch.empty_like(rho_d)
    torch.cuda.synchronize()
    with capi.StripReconstruction(capi.Geometry(*args), variant=variant) as rec:
        rec.set_events(ev)
        loss, _, skipped = rec.nll_grad(sz, sdl, rho_d.data_ptr(), none_d.data_ptr(),
                                        grad.data_ptr())
    g = grad.cpu().numpy().astype(np.float64)
    assert skipped == want_sk == 0
    assert abs(loss - want_loss) <= 1e-6 * abs(want_loss)
    seen = want < 0  # a corner pixel may lie in no event's support
    assert seen.mean() > 0.95 and np.count_nonzero(g[~seen]) <= 2
    assert np.quantile(np.abs(g[seen] / want[seen] - 1.0), 0.99) < 2e-5
