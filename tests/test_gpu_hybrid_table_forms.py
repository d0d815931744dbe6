"""The 3D hybrid iteration with the geometry's voxel table in every form of the
denominator loop, with the golden runs' edge responses (ranges one past the LOR's
end, clamped planes): the image of one iteration before and after a call of so many
iterations that the handle makes its table.

Tolerance: both paths lie within 1e-5 relative L2 of the reference's image (the
bar of the other hybrid tests), so within 2e-5 of each other."""
import os

import numpy as np
import pytest

from jpet_strip import hybrid as HY
from jpet_strip import hybrid_workloads as H

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "hybrid_ref.npz")


@pytest.mark.parametrize("tag", ["computed", "given", "multiplane", "sens3d"])
def test_one_iteration_with_and_without_the_table(tag):
    ref = np.load(GOLDEN)
    g = H.from_arrays(ref, tag + "_")
    gi = ref[tag + "_grid"]
    weights = HY.WEIGHTS_GIVEN if gi[4] else HY.WEIGHTS_COMPUTED
    smap = ref[tag + "_sens_in"] if tag + "_sens_in" in ref else None
    sens = (HY.SENSITIVITY_GIVEN_3D if smap is not None
            else HY.SENSITIVITY_ONE if gi[5] else HY.SENSITIVITY_COMPUTED)
    resp, rho = ref[tag + "_responses"], ref[tag + "_rho"][0]
    many = 3_000_000 // len(resp)  # 1.35 ns per event and iteration: 4 ms, the table costs 0.3
    with HY.HybridReconstruction(g, weights, sens, smap) as r:
        r << resp
        r.rho = rho
        r(1)
        want, cnt = r.rho.astype(np.float64), r.statistics()
        r(many)
        r.rho = rho
        r(1)
        got = r.rho.astype(np.float64)
        assert np.linalg.norm(got - want) < 2e-5 * np.linalg.norm(want)
        assert r.statistics() == cnt
        r << resp[:7]  # another set on a handle that holds the table
        r(many)
        r.rho = rho
        r(1)
        few = r.rho.astype(np.float64)
    with HY.HybridReconstruction(g, weights, sens, smap) as r:
        r << resp[:7]
        r.rho = rho
        r(1)
        assert np.linalg.norm(few - r.rho) < 2e-5 * np.linalg.norm(r.rho)
