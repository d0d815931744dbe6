"""3D hybrid iterations with the weights computed per event (few events) and read
from the geometry's voxel table (many): an iteration is linear in the events, so
the images of single events (computed) add up to the image of all of them
(table), in every form of the denominator loop and with the golden runs' edge
responses (ranges one past the LOR's end, clamped planes).

Tolerance: both paths lie within 1e-5 relative L2 of the reference's image
(the bar of the other hybrid tests), so within 2e-5 of each other."""
import os

import numpy as np
import pytest

import oracle as O
from jpet_strip import hybrid as HY
from jpet_strip import hybrid_workloads as H

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "hybrid_ref.npz")


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("tag", ["computed", "given", "multiplane", "sens3d"])
def test_single_events_add_up_to_the_table_image(tag):
    ref = np.load(GOLDEN)
    g = H.from_arrays(ref, tag + "_")
    gi = ref[tag + "_grid"]
    weights = HY.WEIGHTS_GIVEN if gi[4] else HY.WEIGHTS_COMPUTED
    smap = ref[tag + "_sens_in"] if tag + "_sens_in" in ref else None
    sens = (HY.SENSITIVITY_GIVEN_3D if smap is not None
            else HY.SENSITIVITY_ONE if gi[5] else HY.SENSITIVITY_COMPUTED)
    resp, rho = ref[tag + "_responses"], ref[tag + "_rho"][0]
    total = np.zeros(g.n_voxels)
    n = 0
    with HY.HybridReconstruction(g, weights, sens, smap) as one:
        for i in range(len(resp)):
            one << resp[i:i + 1]
            if one.n_events:
                one.rho = rho
                one(1)
                total += one.rho
                n += 1
    with HY.HybridReconstruction(g, weights, sens, smap) as r:
        for _ in range(2):  # the second time on a handle that holds the table
            r << resp
            r.rho = rho
            r(1)
            assert rel_l2(r.rho, total) < 2e-5
            assert r.statistics()["contributing"] == n
        r << resp[:7]  # few events on a handle with a table
        r.rho = rho
        r(1)
        few = r.rho
    with HY.HybridReconstruction(g, weights, sens, smap) as r:
        r << resp[:7]
        r.rho = rho
        r(1)
        assert rel_l2(few, r.rho) < 2e-5


@pytest.mark.parametrize("n_planes", [5, 13])
def test_padded_and_unpadded_planes_against_the_oracle(n_planes):
    g = H.ring_geometry(24, 0.25, 0.02, 24, 0.02, n_planes, 0.015, 0.060, 0.02 * n_planes)
    resp = H.responses(g, 500, seed=3)
    w, s = O.hybrid_setup(g)
    frames = O.hybrid_translate(g, w, resp)
    with HY.HybridReconstruction(g) as r:
        for k in (2, len(resp)):
            f = O.hybrid_translate(g, w, resp[:k])
            want, cnt = O.hybrid_mlem(g, w, s, f, 1, None, threads=4)
            r << resp[:k]
            r.rho = np.ones(g.n_voxels, np.float32)
            r(1)
            assert rel_l2(r.rho, want) < 1e-5
            assert r.statistics()["contributing"] == cnt[3]
    assert len(frames) > 100
