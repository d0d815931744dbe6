"""The iteration in the reference's operation order (EXACT variant, GPU-reference
mode, large boxes of the other variants, the no-alloc call) at the sizes where it
changes its way: 32 box rows per block, 1024 kept values, boxes of more than 256
columns, rows with no pixel, a single event.

Tolerance: 1e-5 relative L2 of the reference's float path per iteration (the bar
the path is built to); counters identical."""
import numpy as np
import pytest

import oracle as O
from jpet_strip import capi, phantom

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (n_y, n_z, pixel, sigma_z, sigma_dl, events)
SIZES = {
    "one event": (61, 67, 5.0, 10.0, 42.0, 1),
    "26 rows": (61, 67, 5.0, 10.0, 42.0, 777),
    "32 rows": (131, 127, 4.0, 10.0, 42.0, 401),
    "34 rows": (131, 127, 4.0, 10.0, 44.0, 401),
    "82 rows, 1750 pixels": (197, 203, 2.0, 14.0, 55.0, 301),
    "boxes wider than 256 columns": (90, 700, 0.3, 30.0, 4.0, 25),
    "rows of one pixel": (301, 91, 2.0, 0.9, 42.0, 300),
}


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("size", SIZES)
def test_exact_kernel_at_its_limits(size):
    n_y, n_z, p, sz, sdl, n = SIZES[size]
    hz, hy = min(n_z * p / 2, 480.0), min(n_y * p / 2, 430.0)
    ell = phantom.random_ellipse_phantom(seed=31, half_z=hz, half_y=hy, centre_z=0.5 * hz,
                                         centre_y=0.5 * hy, axes=(0.2 * hy, 0.8 * min(hz, hy)))
    ev = phantom.generate_events(ell, n, 450.0, 1000.0, sz, sdl, seed=31)
    args = (450.0, 1000.0, n_y, n_z, p, sz, sdl)
    cg, og = capi.Geometry(*args), O.Geometry(*args)
    want, st = O.mlem_f(og, ev, 1, threads=8)
    for variant in (capi.VARIANT_EXACT, capi.VARIANT_FAST):
        with capi.StripReconstruction(cg, variant=variant) as rec:
            rec.set_events(ev)
            rec.iterate(1)
            got, cnt = rec.rho, rec.counters()
        assert rel_l2(got, want) < 1e-5, variant
        assert cnt["n_kernel_calls"] == st["n_kernel_calls"]
        assert cnt["n_contributing"] == st["n_contributing"]
    with capi.StripReconstruction(cg, mode=capi.MODE_GPU_REFERENCE) as rec:
        rec.set_events(ev)
        rec.iterate(1)
        assert rel_l2(rec.rho, O.mlem_gpuref(og, ev, 1, threads=8)) < 1e-5
    d_ev = torch.from_numpy(ev).cuda()
    rho = torch.ones(n_y, n_z, device="cuda")
    out = torch.empty_like(rho)
    g = cg.c()
    stream = torch.cuda.current_stream().cuda_stream
    capi._check(capi.lib().jpet_strip_iterate_noalloc(capi.C.byref(g), d_ev.data_ptr(), n,
                                                      rho.data_ptr(), out.data_ptr(), stream))
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want) < 1e-5
