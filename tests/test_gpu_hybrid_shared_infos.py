"""3D hybrid geometries in which two LORs share a range of pixel infos (given weights
allow it): every event's weights are those of its own LOR, however many iterations
run, so that no table by pixel info can stand for them.

Tolerance 1e-5 relative L2 against the oracle, as in the other hybrid tests."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from jpet_strip import hybrid as HY
from jpet_strip import hybrid_workloads as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["ascending", "descending"])
def test_lors_that_share_their_pixel_infos(order):
    g = H.ring_geometry(24, 0.25, 0.02, 24, 0.02, 13, 0.015, 0.060, 0.26)
    resp = H.responses(g, 400, seed=3)
    w, s = O.hybrid_setup(g)
    begin, end = g.info_begin.copy(), g.info_end.copy()
    pairs = 0
    for l in range(1, g.n_lors, 2):
        a, b = (l - 1, l) if order == "ascending" else (l, l - 1)
        if begin[a] < end[a] and begin[b] < end[b]:
            begin[b], end[b] = begin[a], end[a]
            pairs += 1
    assert pairs > 50
    g = dataclasses.replace(g, info_begin=begin, info_end=end, weights=w)
    frames = O.hybrid_translate(g, w, resp)
    assert len(frames) > 100
    want, cnt = O.hybrid_mlem(g, w, s, frames, 1, None, threads=4)
    with HY.HybridReconstruction(g, HY.WEIGHTS_NORMALIZED, HY.SENSITIVITY_GIVEN, s) as r:
        r.set_frame_events(frames)
        for before in (0, 20000):  # iterations that a table would pay for
            r(before)
            r.rho = np.ones(g.n_voxels, np.float32)
            r(1)
            got = r.rho.astype(np.float64)
            assert r.statistics()["contributing"] == cnt[3]
            assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(want), before
